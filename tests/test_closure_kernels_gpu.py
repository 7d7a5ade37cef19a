"""The persistent convolution and weight-gradient kernels at the edges of their
tiles: one voxel, rows of 126/127/128/129 voxels (where a window of rows stops
holding every dy), tiles that end inside a row, grids of several rounds of the
stage ring and of the accumulators.

Operands are small integers, exact in BF16, and every sum of products stays below
2^24: FP32 results have to be the oracle's exactly, whatever the order. BF16
results are off by one rounding (2^-8 relative) of a product with GELU or its
derivative, which FP32 gives to 2e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1, 1), (2, 3, 5, 7), (1, 2, 3, 126), (1, 2, 3, 127), (2, 1, 2, 128), (1, 2, 2, 129), (1, 3, 1, 300),
          (2, 40, 44, 60), (1, 18, 60, 150)]


def _ints(rng, shape, hi):
    return rng.integers(-hi, hi + 1, shape).astype(np.float64)


def _shifted(t):
    """the same values, one element off a 16-byte boundary"""
    import torch
    flat = torch.zeros(t.numel() + 8, dtype=t.dtype, device=t.device)
    v = flat[1:1 + t.numel()].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize("shape", SHAPES)
def test_conv3d_exact(shape, btlib):
    import torch

    import oracle.closure_oracle as co
    from initializator_gb300 import closure
    nb, nz, ny, nx = shape
    rng = np.random.default_rng(nx)
    x, w, b = _ints(rng, (nb, nz, ny, nx, 16), 2), _ints(rng, (27, 16, 16), 2), _ints(rng, 16, 3)
    z = 0.25 * _ints(rng, (nb, nz, ny, nx, 16), 8)
    lay = closure.PaddedRows(nb, nz, ny, nx)
    xr = lay.pack(x, "cuda")
    wf, wd = closure.pack_weights(torch.tensor(w, dtype=torch.float32, device="cuda"))
    bias = torch.tensor(b, dtype=torch.float32, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    ref, back = co.conv3d(x, w, b), co.conv3d_data_grad(x, w)
    pad = ((0, 0), (1, 1), (1, 1), (1, 1), (0, 0))

    for place in (lambda t: t, _shifted):  # FP32 rows on and off a 16-byte boundary
        rows = lambda: place(torch.full((lay.rows, 16), 7.0, device="cuda"))
        outf, pre, grad = rows(), rows(), rows()
        out, dz = lay.empty("cuda"), lay.empty("cuda")
        zr = place(torch.tensor(np.pad(z, pad).reshape(-1, 16), dtype=torch.float32, device="cuda"))
        closure.conv3d(lay, xr, wf, 0, bias=bias, out=out, pre=pre, status=st)
        closure.conv3d(lay, xr, wf, 1, bias=bias, outf=outf, status=st)
        closure.conv3d(lay, xr, wd, 2, out=dz, pre=zr, status=st)
        closure.conv3d(lay, xr, wd, 3, outf=grad, status=st)
        torch.cuda.synchronize()
        assert int(st.item()) == 0
        full = lambda r: r.float().reshape(nb, nz + 2, ny + 2, nx + 2, 16).cpu().numpy()
        np.testing.assert_array_equal(full(pre), np.pad(ref, pad))
        np.testing.assert_array_equal(full(outf), np.pad(ref, pad))
        np.testing.assert_array_equal(full(grad), np.pad(back, pad))
        for rows16, want, scale in ((out, co.gelu(ref), ref), (dz, back * co.gelu_grad(z), back)):
            assert not rows16[:lay.margin].any() and not rows16[lay.margin + lay.rows:].any()
            err = np.abs(full(rows16[lay.margin:lay.margin + lay.rows]) - np.pad(want, pad))
            assert (err <= np.pad(2.0 ** -8 * np.abs(want) + 2e-6 * np.abs(scale), pad)).all()


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("aligned", [True, False])
def test_weight_grad_exact(shape, aligned, btlib):
    import torch

    import oracle.closure_oracle as co
    from initializator_gb300 import closure
    nb, nz, ny, nx = shape
    rng = np.random.default_rng(nx)
    x, dz = _ints(rng, (nb, nz, ny, nx, 16), 2), _ints(rng, (nb, nz, ny, nx, 16), 2)
    lay = closure.PaddedRows(nb, nz, ny, nx)
    xr, dr = lay.pack(x, "cuda"), lay.pack(dz, "cuda")
    if not aligned:
        xr, dr = _shifted(xr), _shifted(dr)
    gw, gb, _ = closure.weight_grad(lay, xr, dr)
    want_w, want_b = co.conv3d_weight_grad(x, dz)
    np.testing.assert_array_equal(gw.cpu().numpy(), want_w)
    np.testing.assert_array_equal(gb.cpu().numpy(), want_b)


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 3, 5, 7), (1, 2, 3, 127)])
def test_outputs_cover_margins(shape, btlib):
    """BF16 outputs are whole, margins included, in buffers that held something
    else: of the convolution and of FP32 rows turned into padded ones; the grouped
    forms of packing and of the weight gradient give what the single ones give."""
    import ctypes

    import torch
    from initializator_gb300 import closure
    nb, nz, ny, nx = shape
    rng = np.random.default_rng(nx)
    lay = closure.PaddedRows(nb, nz, ny, nx)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    xr = lay.pack(_ints(rng, (nb, nz, ny, nx, 16), 2), "cuda")
    w = torch.tensor(_ints(rng, (3, 27, 16, 16), 2), dtype=torch.float32, device="cuda")
    packed = torch.empty((3, 2, 27 * 512), dtype=torch.uint8, device="cuda")
    assert btlib.bt_conv3d_pack_layers(ptr(w), 3, ptr(packed), stream) == 0
    for i in range(3):
        for k, one in enumerate(closure.pack_weights(w[i])):
            assert torch.equal(packed[i, k], one)

    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    bias = torch.tensor(_ints(rng, 16, 3), dtype=torch.float32, device="cuda")
    clean, dirty = lay.empty("cuda"), torch.full_like(lay.empty("cuda"), 3.0)
    for out in (clean, dirty):
        closure.conv3d(lay, xr, packed[1, 0], 0, bias=bias, out=out, status=st)
    assert torch.equal(clean, dirty) and int(st.item()) == 0

    rows = torch.randn((lay.rows, 16), device="cuda")
    out = torch.full_like(clean, 3.0)
    assert btlib.bt_conv3d_pad_rows(ptr(rows), nb, nx, ny, nz, ptr(out), stream) == 0
    want = lay.empty("cuda")
    want[lay.margin:lay.margin + lay.rows] = rows.to(torch.bfloat16)
    assert torch.equal(out, want)
    assert btlib.bt_conv3d_pad_rows(ctypes.c_void_p(rows.data_ptr() + 4), nb, nx, ny, nz, ptr(out), stream) < 0

    gw, gb, scratch = closure.weight_grad(lay, xr, clean)
    both = torch.full((27 * 256 + 16 + 1,), 5.0, device="cuda")
    assert btlib.bt_conv3d_weight_bias_grad(ptr(xr), ptr(clean), nb, nx, ny, nz, ptr(scratch), ptr(both),
                                            ptr(both[27 * 256:]), stream) == 0
    assert torch.equal(both[:27 * 256], gw.flatten()) and torch.equal(both[27 * 256:-1], gb) and float(both[-1]) == 5.0
