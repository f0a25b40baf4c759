"""Selection from rows of few different values: equal ones are taken from the left, positive zeros are above negative ones, and what is
not finite is never taken."""
import numpy as np
import pytest
import torch

from spiraltorch_b200.ops import rank as R

pytestmark = pytest.mark.gpu


def _select(row, k, top):
    bits = row.view(np.uint32)
    order = np.where(bits >> 31, ~bits, bits | np.uint32(0x80000000)).astype(np.int64)      # the values' order as integers
    columns = np.flatnonzero(np.isfinite(row))
    return columns[np.lexsort((columns, -order[columns] if top else order[columns]))][:k]


@pytest.mark.parametrize("rows,cols", [(3, 130), (40, 1063), (300, 4099), (5, 17510), (1, 50000)])
@pytest.mark.parametrize("k", [1, 27, 100])
@pytest.mark.parametrize("kind", ["equal", "zeros", "three", "steps up", "steps down", "masked", "largest"])
def test_selection(rows, cols, k, kind):
    rng = np.random.default_rng(cols + k)
    x = np.ones((rows, cols), np.float32)
    if kind == "zeros":
        x = np.where(rng.random((rows, cols)) < 0.5, np.float32(0.0), np.float32(-0.0))
    elif kind == "three":
        x = rng.integers(-1, 2, (rows, cols)).astype(np.float32)
    elif kind.startswith("steps"):
        x = np.repeat(np.arange(cols // 9 + 1, dtype=np.float32)[None], rows, 0).repeat(9, 1)[:, :cols]
        x = x if kind == "steps up" else x[:, ::-1]
    elif kind == "masked":
        x = rng.standard_normal((rows, cols)).astype(np.float32).round(1)
        u = rng.random((rows, cols))
        x = np.where(u < 0.9, -np.inf, np.where(u < 0.92, np.inf, np.where(u < 0.94, np.nan, x))).astype(np.float32)
    elif kind == "largest":
        big = np.finfo(np.float32).max
        x = rng.choice(np.array([big, -big, np.inf, -np.inf], np.float32), (rows, cols))
    x = np.ascontiguousarray(x)
    for name, top in (("topk", True), ("bottomk", False)):
        values, index = getattr(R, name)(torch.from_numpy(x).cuda(), k)
        values, index = values.cpu().numpy(), index.cpu().numpy()
        for r in range(rows):
            want = _select(x[r], k, top)
            assert (index[r, :len(want)] == want).all()
            assert (values[r, :len(want)].view(np.uint32) == x[r, want].view(np.uint32)).all()
