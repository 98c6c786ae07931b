"""
The ring of stages of the FFT passes that re-arm a stage one unit late: when a wait runs out, the block waits for exactly the
copies that it has sent for and not yet seen.
"""
import pytest


@pytest.mark.parametrize('stages', [2, 3, 4])
def test_copies_in_flight_when_a_wait_runs_out(stages):
    from pyrecon_b200 import _lib as L
    pending = L.load().prc_debug_units_in_flight
    for stop in range(5 * stages):
        # the kernels' order: the prologue sends for the first units; unit u waits for its own copy and then, behind the
        # barrier that every thread past unit u - 1 takes, sends for unit u - 1 + stages
        sent, seen = set(range(stages)), set()
        for u in range(stop):
            seen.add(u)
            if u > 0:
                sent.add(u - 1 + stages)
        # the wait of unit `stop` runs out before that unit sends for anything
        assert set(range(stop, stop + pending(stop, stages))) == sent - seen
