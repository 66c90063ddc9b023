"""The pressure solve's shared memory lets two blocks share an SM on every grid: the first tail
levels tried here have 1,375 to 1,500 cells, the most a tail's may have (50 x 29 at 1600 x 900 and
800 x 450, 50 x 30 at 800 x 480, 60 x 25 at 960 x 400, 125 x 12 at 1000 x 96).
"""
import pytest

import sprout_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1600, 900), (800, 450), (800, 480), (960, 400), (1000, 96), (880, 400)])
def test_two_blocks_per_sm(w, h):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = ((w + 15) // 16) * ((h + 15) // 16)
    assert tiles > 2 * sms
    sim = S.FluidSim(w, h, 1024, S.SimParams({"cell_size": 0.002}))
    sim.set_launch(pressure_blocks=tiles, pressure_blocks_mixed=tiles)   # as many as the device holds
    sim.set_precision("mixed")
    got = sim.launch()
    assert got["pressure_blocks"] == 2 * sms and got["pressure_blocks_mixed"] == 2 * sms, got
