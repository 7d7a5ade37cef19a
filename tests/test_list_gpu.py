"""The list kernels (generic: one thread a pore voxel; FP32 fast path: one a group
of four along x) where they can go wrong: FP64 against the oracle, bit for bit (array_equal), over field axes that
take the short relaxation and ones that do not, face velocities at the upwind
switch's edges (zero, tiny, cancelling pairs), gradients along z alone or along
every axis; fields that are not finite; fields that are not zero in solid
voxels (every kernel leaves zero there); sizes around the list's 64 x 8 columns
and 128-thread chunks, grids without a pore voxel among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(shape, seed, axis=(0.0, 0.0, 1.0), grad=(0.0, 0.0, 0.05), porosity=0.6):
    from initializator_gb300 import geometry
    rng = np.random.default_rng(seed)
    mask = (rng.uniform(size=shape) < porosity).astype(np.uint8)
    nz, ny, nx = shape
    vel = [rng.uniform(-1e-3, 1e-3, s) for s in ((nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx))]
    for v in vel:  # the switch's edges: zero, far below 1e-50's reach, just above it, pairs that cancel
        pick = rng.integers(0, 8, v.shape)
        v[pick == 0] = 0.0
        v[pick == 1] = -0.0
        v[pick == 2] *= 1e-45
        v[pick == 3] *= 1e-31
        v[pick == 4] = np.sign(v[pick == 4]) * 1e-3
    dt = 0.5 * geometry.stable_dt(1e-6, 2.3e-9)
    kw = dict(dx=1e-6, dy=1.1e-6, dz=0.9e-6, dt=dt, main_field=axis, grad=grad, d_pore=2.3e-9, t1=0.1, t2=0.05,
              rho1=3e-5, rho2=5e-5, p_eq=0.5, vector_mult=1, velocity=1, diffusion=1, buffer=(1, 0, 2))
    st = rng.uniform(-1, 1, (3,) + shape) * mask
    return mask, vel, st, kw


def _same(a, b):
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("mac", [False, True])
@pytest.mark.parametrize("axis,grad", [((2.5, 0, 0), (0, 0, 0.05)), ((0, 0.3, 0), (0.02, -0.03, 0.05)),
                                       ((0, 0, 1e-3), (0, 0, 0.05)), ((0, 0, -1.0), (0, 0, 0)),
                                       ((0.2, 0.3, 0.9), (0.01, 0, 0.05))])
def test_short_forms_keep_the_bits(axis, grad, mac, btlib, oracle_lib):
    import initializator_gb300 as bt
    import oracle
    shape = (11, 9, 70)
    mask, vel, st, kw = _case(shape, 3, axis, grad)
    ref, ref_mt = oracle.run(oracle.make_params(shape, **kw), mask, st, 12, vel=vel, maccormack=mac)
    scheme = bt.BT_SCHEME_MACCORMACK if mac else bt.BT_SCHEME_REFERENCE
    with bt.Solver(bt.make_config(shape, precision=bt.BT_F64, scheme=scheme, **kw)) as s:
        s.upload_geometry(mask, vel)
        s.set_state(st)
        mt = s.run(12)
        assert _same(s.get_state(), ref)
    assert np.abs(mt - ref_mt).max() <= 1e-12 * np.abs(ref_mt).max()


@pytest.mark.parametrize("diffusion", [0, 1])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_fields_that_are_not_finite(value, diffusion, btlib, oracle_lib):
    """Where the reference's sums are Inf or NaN, so are the kernel's."""
    import initializator_gb300 as bt
    import oracle
    shape = (7, 9, 20)
    mask, vel, st, kw = _case(shape, 5)
    kw["diffusion"] = diffusion
    z, y, x = np.argwhere(mask[3:4, 4:6, 8:12])[0] + (3, 4, 8)
    st[0, z, y, x] = value
    with np.errstate(all="ignore"):
        ref, _ = oracle.run(oracle.make_params(shape, **kw), mask, st, 2, vel=vel)
    with bt.Solver(bt.make_config(shape, precision=bt.BT_F64, **kw)) as s:
        s.upload_geometry(mask, vel)
        s.set_state(st)
        s.run_async(2)
        s.synchronize()
        got = s.get_state()
        with pytest.raises(bt.BtError) as e:
            s.read_mt(2)
        assert e.value.code == -3  # BT_E_NAN
    pore = np.broadcast_to(mask > 0, ref.shape)
    assert _same(got[pore], ref[pore])


@pytest.mark.parametrize("steps", [1, 2, 3, 70])
@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_solid_voxels_of_an_uploaded_field(precision, scheme, steps, btlib):
    """Values in solid voxels act on the first step as they always did (not at
    all but for NaN and Inf: a pore-solid face's diffusivity is 1e-50) and are
    zero after it, in both field buffers."""
    import initializator_gb300 as bt
    shape = (6, 17, 70)
    mask, vel, st, kw = _case(shape, 7, grad=(0, 0, 0))
    for v, dim in zip(vel, (2, 1, 0)):  # closed pore-solid faces
        n = shape[dim]
        open_ = np.take(mask, range(1, n), dim) & np.take(mask, range(n - 1), dim)
        v[tuple(slice(1, n) if d == dim else slice(None) for d in range(3))] *= open_
    kw.update(vector_mult=0)
    dirty = np.random.default_rng(8).uniform(-1, 1, st.shape) * (1 - mask) + st
    out = []
    for start in (st, dirty):
        with bt.Solver(bt.make_config(shape, precision=bt.BT_F32 if precision == "f32" else bt.BT_F64, scheme=scheme,
                                      **kw)) as s:
            s.upload_geometry(mask, vel)
            s.set_state(start)
            if start is dirty and steps > 1:  # as read back before the run
                assert np.abs(s.get_state() - start).max() <= 1e-6
            mt = s.run(steps)
            out.append((s.get_state(), mt))
            mt2 = s.run(1)
            out[-1] += (s.get_state(), mt2)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert not out[1][0][:, mask == 0].any() and not out[1][2][:, mask == 0].any()


@pytest.mark.parametrize("shape,porosity", [((1, 1, 1), 1.0), ((2, 3, 5), 0.0), ((1, 8, 64), 1.0), ((2, 9, 65), 0.3),
                                            ((3, 7, 63), 0.05), ((40, 33, 129), 0.4)])
@pytest.mark.parametrize("scheme", [0, 1])
def test_list_sizes(shape, porosity, scheme, btlib, oracle_lib):
    import initializator_gb300 as bt
    import oracle
    mask, vel, st, kw = _case(shape, 11, grad=(0, 0, 0), porosity=porosity)
    kw.update(buffer=(0, 0, 0), vector_mult=2 * scheme)
    n = 5
    wave = None
    if scheme:
        kw.update(gamma=bt.GAMMA_PROTON)
        wave = np.full((n, 3), 0.05)
    ref, ref_mt = oracle.run(oracle.make_params(shape, **kw), mask, st, n, vel=vel, grad_wave=wave)
    cfg = dict(kw, vector_mult=0)
    with bt.Solver(bt.make_config(shape, precision=bt.BT_F64, scheme=scheme, **cfg)) as s:
        s.upload_geometry(mask, vel)
        if scheme:
            s.set_schedule([], grad_wave=wave)
        s.set_state(st)
        mt = s.run(n)
        got = s.get_state()
    tol = 1e-10 if scheme else 0.0  # KSPACE: phase factors differ in rounding
    assert np.abs(got - ref).max() <= tol
    assert np.abs(mt - ref_mt).max() <= max(tol, 1e-12) * max(np.abs(ref_mt).max(), 1.0)


@pytest.mark.parametrize("shape,porosity", [((1, 1, 1), 1.0), ((3, 2, 5), 0.6), ((2, 9, 64), 1.0), ((17, 8, 65), 0.3),
                                            ((5, 7, 63), 0.05), ((33, 17, 130), 0.5), ((4, 4, 8), 0.0)])
@pytest.mark.parametrize("scheme,axis", [(0, None), (1, None), (1, (0, 0, 1)), (1, (0.3, 0.5, 0.8))])
@pytest.mark.parametrize("batch,flow,trim", [(1, True, False), (1, False, True), (3, True, True)])
def test_quad_list_matches_generic(shape, porosity, scheme, axis, batch, flow, trim, btlib, monkeypatch):
    """The FP32 fast path's quad list against the generic kernel, with a pulse
    step: the same update in another FP32 order, a few ulps a step (1e-5 over
    12 steps); any number of chunks gives the same field, M(t) within 1e-6."""
    import math

    import initializator_gb300 as bt
    mask, vel, st, kw = _case(shape, 17, porosity=porosity, grad=(0, 0, 0))
    kw.update(buffer=tuple(min(1, (n - 1) // 2) if trim else 0 for n in reversed(shape)), velocity=int(flow),
              vector_mult=0)
    wave = None
    if scheme == 1:
        kw.update(gamma=bt.GAMMA_PROTON)
        if axis is not None:
            wave = 0.1 * np.ones((12, batch, 1)) * np.linspace(0, 1, batch)[None, :, None] * np.array(axis)
            wave = wave if batch > 1 else 0.1 * np.ones((12, 1, 1)) * np.array(axis)
    out = []
    for env, chunks in (("1", 0), (None, 0), (None, 1), (None, 7)):
        if env:
            monkeypatch.setenv("BT_NO_TMA", env)
        else:
            monkeypatch.delenv("BT_NO_TMA", raising=False)
        with bt.Solver(bt.make_config(shape, precision=bt.BT_F32, scheme=scheme, batch=batch, **kw)) as s:
            s.upload_geometry(mask, vel if flow else None)
            s.set_schedule([(5, 2, math.pi, (1.0, 0.0, 0.0))], grad_wave=wave)
            s.set_chunks(chunks)
            s.set_state(np.stack([st] * batch))
            mt = s.run(12)
            out.append((s.get_state(), mt))
    top = max(np.abs(out[0][1]).max(), 1e-3 * mask.size)
    assert np.abs(out[1][0] - out[0][0]).max() <= 1e-5
    assert np.abs(out[1][1] - out[0][1]).max() <= 1e-5 * top
    for st2, mt2 in out[2:]:
        assert np.array_equal(st2, out[1][0])
        assert np.abs(mt2 - out[1][1]).max() <= 1e-6 * top


@pytest.mark.parametrize("flow", [False, True])
def test_dense_large_grid_matches_generic(flow, btlib, monkeypatch):
    """A field beyond L2 whose quads nearly all hold a pore voxel takes the TMA
    ring; a shortened wait bound that no wait reaches gives the same bits."""
    import torch

    import initializator_gb300 as bt
    shape = (192, 256, 260)
    rng = np.random.default_rng(3)
    mask = np.ones(shape, np.uint8)
    mask[rng.uniform(size=shape) < 0.02] = 0
    nz, ny, nx = shape
    vel = None
    if flow:
        vel = [rng.uniform(-1e-3, 1e-3, s) for s in ((nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx))]
    kw = dict(dx=1e-6, dt=3e-5, d_pore=2.3e-9, t1=0.1, t2=0.05, rho1=1e-5, rho2=1e-5, p_eq=1.0, velocity=int(flow),
              gamma=bt.GAMMA_PROTON)
    m = torch.rand(shape, device="cuda") * torch.from_numpy(mask).cuda()
    out = []
    for env, polls in (("1", -1), (None, -1), (None, 1 << 19)):
        if env:
            monkeypatch.setenv("BT_NO_TMA", env)
        else:
            monkeypatch.delenv("BT_NO_TMA", raising=False)
        with bt.Solver(bt.make_config(shape, precision=bt.BT_F32, scheme=1, **kw)) as s:
            s.upload_geometry(mask, vel)
            s.set_wait_polls(polls)
            s.set_schedule([], grad_wave=np.full((4, 3), 0.05) * (0, 0, 1))
            s.set_state_device([m, 0.5 * m, m])
            mt = s.run(4)
            out.append(([v.clone() for v in s.field_views()], mt))
    for a, b in zip(out[1][0], out[0][0]):
        assert float((a - b).abs().max()) <= 1e-5
    assert np.abs(out[1][1] - out[0][1]).max() <= 1e-5 * np.abs(out[0][1]).max()
    assert all(torch.equal(a, b) for a, b in zip(out[1][0], out[2][0])) and np.array_equal(out[1][1], out[2][1])


def test_geometry_uploaded_again(btlib):
    """A second geometry under a running field: voxels that became solid are
    zero after the next step, as with a handle that had it from the start."""
    import initializator_gb300 as bt
    shape = (9, 12, 66)
    mask, vel, st, kw = _case(shape, 13, grad=(0, 0, 0))
    mask2, _, _, _ = _case(shape, 14)
    for scheme in (0, 2):
        with bt.Solver(bt.make_config(shape, precision=bt.BT_F64, scheme=scheme, **kw)) as s:
            s.upload_geometry(mask, vel)
            s.set_state(st)
            s.run(3)
            mid = s.get_state()
            s.upload_geometry(mask2, vel)
            mt = s.run(3)
            got = s.get_state()
        with bt.Solver(bt.make_config(shape, precision=bt.BT_F64, scheme=scheme, **kw)) as s:
            s.upload_geometry(mask2, vel)
            s.set_state(mid)
            assert np.array_equal(s.run(3), mt)
            assert np.array_equal(s.get_state(), got)
        assert not got[:, mask2 == 0].any()
