"""A batch of more tanks than its pressure solve has blocks: each block then takes several tanks'
tails and sets each up again in every V-cycle. Every tank as it steps alone, bit for bit."""
import pytest

import sprout_gb300 as S
import tanks
from test_gpu_batch import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("blocks", [1, 2, 4])
def test_more_tanks_than_blocks(precision, blocks):
    def mix():   # tails of different sizes, one of a single level after the first
        return [tanks.dam_break(96, 64), tanks.stratified(128, 72), tanks.dam_break(37, 21, width=0.7, height=0.7),
                tanks.dam_break(160, 96), tanks.dam_break(101, 57)]
    alone = [t.engine()[0] for t in mix()]
    batched = [t.engine()[0] for t in mix()]
    for s in alone:
        s.set_precision(precision)
    batch = S.Batch(batched, precision)
    batch.set_launch(pressure_blocks=blocks, pressure_blocks_mixed=blocks)
    n = 4
    for s in alone:
        s.step(n, n / 240.0)
    batch.step(n)
    batch.sync()
    problems = []
    for k, (a, b) in enumerate(zip(alone, batched)):
        problems += compare(a, b, f"tank {k}")
    assert not problems, "\n".join(problems)
