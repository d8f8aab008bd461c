"""Scattering blocks whose rows are an even number of items but no multiple of 4 (items in pairs) or
an odd one (item by item, four at a time): block sizes of 2 modulo 4, slices that end inside a quad,
array edges and destinations that cut or misalign a pair."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEOMS = [
    ((300, 410), (150, 204), (75, 102)),     # 7650 items (2 modulo 4): two slices
    ((31, 95), (15, 18), (5, 6)),
    ((9, 7), (9, 6), (3, 2)),                # a pair a row
    ((64, 301), (64, 150), (32, 150)),       # 4800 items
    ((50, 45), (25, 9), (25, 3)),            # odd widths, rows shorter than a quad
    ((10, 10003), (5, 5002), (1, 4098)),     # a slice of 2 items
]


@pytest.mark.parametrize("geom", GEOMS, ids=lambda g: "x".join(map(str, g[0])))
@pytest.mark.parametrize("dtype", [np.float64, np.int32])
def test_pairs(ctx, ia, geom, dtype):
    import torch
    shape, cs, bs = geom
    rng = np.random.default_rng(shape[1])
    x = (rng.standard_normal(shape) * 1000).astype(dtype)
    x[::3] = 5                                              # runs beside raw and LZ4 planes
    c = ia.Container.from_numpy(ctx, x, cs, bs)
    assert np.array_equal(c.to_numpy(), x)
    for extra in (0, 1, 2, 3, 4):
        ld = shape[1] + extra
        wide = torch.full((shape[0], ld), 7, dtype=torch.int64 if x.itemsize == 8 else torch.int32, device="cuda")
        torch.cuda.synchronize()
        c.decode_to_device(wide.data_ptr(), ld)
        assert np.array_equal(wide[:, :shape[1]].cpu().numpy().view(dtype), x)
    c.free()
