"""bt_step_noalloc's kernel against the handle's list kernels: one voxel, single
rows and planes along each axis, sizes around a CTA of 128 voxels, more voxels
than the launch has threads; with and without flow and precession, an oblique
main field, a trimming box that leaves nothing.

Tolerances as for the entry point's other test: the FP64 field to the last bit,
its sums to 1e-12 of the sum of magnitudes; FP32 to 1e-5."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((1, 1, 1), 1, 1, (0, 0, 0)), ((129, 1, 1), 1, 1, (0, 0, 0)), ((1, 127, 1), 1, 0, (0, 0, 0)),
         ((1, 1, 128), 0, 1, (0, 0, 0)), ((5, 7, 11), 0, 0, (3, 2, 1)), ((6, 8, 10), 1, 1, (5, 4, 3)),
         ((66, 72, 70), 1, 1, (1, 1, 1)), ((64, 100, 63), 0, 1, (0, 3, 0))]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("case", CASES)
def test_single_step_matches_handle(case, precision, btlib):
    import torch

    import initializator_gb300 as bt
    from initializator_gb300 import geometry
    shape, velocity, mult, buffer = case
    rng = np.random.default_rng(shape[2] + velocity)
    mask = (rng.random(shape) < 0.7).astype(np.uint8)
    if mask.size < 8:
        mask[:] = 1
    nz, ny, nx = shape
    vel = [rng.uniform(-1e-3, 1e-3, s) * (rng.random(s) < 0.8) for s in
           ((nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx))] if velocity else None
    st0 = rng.uniform(-1, 1, (3,) + shape) * mask
    prec = bt.BT_F64 if precision == "f64" else bt.BT_F32
    cfg = bt.make_config(shape, precision=prec, dx=1e-6, dy=1.1e-6, dz=0.9e-6,
                         dt=0.5 * geometry.stable_dt(0.9e-6, 2.3e-9), main_field=(0.0, 0.0, 1.0) if mult else (0.2, 0.3, 0.9),
                         grad=(0.02, -0.03, 0.05), d_pore=2.3e-9, t1=0.1, t2=0.05, rho1=3e-5, rho2=5e-5, p_eq=0.5,
                         vector_mult=mult, velocity=velocity, diffusion=1, buffer=buffer)
    with bt.Solver(cfg) as s:
        s.upload_geometry(mask, vel)
        s.set_state(st0)
        ref_mt = s.run(1)[0]
        ref = np.stack(list(s.get_state()))
    dt = torch.float64 if precision == "f64" else torch.float32
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dt)
    mask_d, cur = torch.from_numpy(mask).cuda(), [dev(st0[c]) for c in range(3)]
    vel_d = [dev(v) for v in vel] if velocity else [None] * 3
    out = [torch.full_like(c, 9.0) for c in cur]
    sums = torch.full((3,), float("nan"), dtype=torch.float64, device="cuda")
    rc = btlib.bt_step_noalloc(ctypes.byref(cfg), *[None if t is None else ctypes.c_void_p(t.data_ptr())
                                                    for t in (mask_d, *vel_d, *cur, *out, sums)],
                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    field = np.stack([o.double().cpu().numpy() for o in out])
    if precision == "f64":
        np.testing.assert_array_equal(field, ref)
    else:
        assert np.abs(field - ref).max() <= 1e-5 * max(1e-30, np.abs(ref).max())
    scale = np.abs(ref).sum()
    assert np.abs(sums.cpu().numpy() - ref_mt).max() <= (1e-12 if precision == "f64" else 1e-5) * scale
