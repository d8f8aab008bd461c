"""Blocks whose rows are no multiple of 4 items (gathered and scattered item by item), against
the oracle's chunks: several 4096-item slices per block, slices that start inside a row, planes
that start at odd bytes, chunk and array padding, one-dimensional blocks, dense arrays with a
leading dimension of their own."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

GEOMS = [
    ((300, 410), (150, 205), (75, 101)),     # 7575 items: two slices, the second inside a row
    ((130, 97), (130, 97), (65, 97)),        # 6305 items, odd plane starts
    ((97, 1031), (48, 500), (13, 333)),      # 4329 items, ragged edges in both directions
    ((33, 5), (33, 5), (33, 5)),             # less than one quad per row
    ((20001,), (10001,), (4097,)),
]


@pytest.mark.parametrize("geom", GEOMS, ids=lambda g: "x".join(map(str, g[0])))
@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.int64, np.uint32])
def test_odd_blocks(ctx, ia, geom, dtype):
    import torch
    shape, cs, bs = geom
    rng = np.random.default_rng(len(shape) * 100 + shape[-1])
    x = (rng.standard_normal(shape) * 1000).astype(dtype)
    c = ia.Container.from_numpy(ctx, x, cs, bs)
    g, want = O.encode_array(x, cs, bs)
    assert c.chunks() == want
    assert np.array_equal(c.to_numpy(), x)
    if len(shape) == 2:                      # a wider destination keeps its other columns defined
        wide = torch.full((shape[0], shape[1] + 3), 7, dtype=torch.int64 if x.itemsize == 8 else torch.int32, device="cuda")
        torch.cuda.synchronize()
        c.decode_to_device(wide.data_ptr(), shape[1] + 3)
        got = wide[:, :shape[1]].cpu().numpy().view(dtype)
        assert np.array_equal(got, x)
    c.free()
