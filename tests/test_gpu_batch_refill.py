"""The one-tile batched kernel where each tile belongs to another entry than the two
before it: a slot's constants are read by ordinary loads until the tile's end and
refilled by bulk copies as soon as it is given up, wide entries following narrow
ones and the other way round, on a few CTAs, against the level kernel bit for bit."""

import pytest
import torch

from test_gpu_batch import _check_against_single, _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 2, 5])
@pytest.mark.parametrize("unit,stages", [(16, 3), (32, 2), (32, 3)])
@pytest.mark.parametrize("widths", [(256, 64), (256, 256, 64, 64), (256, 128, 64), (256,),
                                    (64, 256, 256)])
def test_constants_change_with_every_tile(lib, widths, unit, stages, ctas):
    from mplicits_gb300.batch import BatchEntry
    g = torch.Generator("cuda").manual_seed(3)
    models = [[_model(w, 2 + s % 2, 10 * w + s, "bf16") for s in range(5)] for w in set(widths)]
    models = {m[0].net[0][0].out_features: m for m in models}
    entries = []
    for i in range(90):
        n = 100 + i % 29
        x = torch.rand(n, 3, device="cuda", generator=g) * 2 - 1
        entries.append(BatchEntry(models[widths[i % len(widths)]][i % 5],
                                  torch.full((n,), 5.0, device="cuda"), x=x, n=n))
    _check_against_single(entries, "bf16", 1, unit, stages, ctas)
