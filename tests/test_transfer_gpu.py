"""Fields across the host boundary, bit for bit: what bt_set_state is given is
what bt_get_state returns (rounded once to FP32 in FP32 handles), for rows shorter
than, equal to and longer than the pitch's unit, single fields and batches, and
the face velocities (rows of nx + 1) as one step sees them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 3), (2, 5, 31), (4, 3, 64), (5, 7, 67), (40, 33, 129)])
def test_state_round_trip(shape, batch, precision, btlib):
    import initializator_gb300 as bt
    rng = np.random.default_rng(shape[2] + batch)
    mask = (rng.random(shape) < 0.6).astype(np.uint8)
    lead = (batch, 3) if batch > 1 else (3,)
    kw = dict(batch=batch, scheme=bt.BT_SCHEME_KSPACE) if batch > 1 else {}
    cfg = bt.make_config(shape, precision=bt.BT_F64 if precision == "f64" else bt.BT_F32, dx=1e-6, dy=1e-6, dz=1e-6,
                         dt=1e-6, main_field=(0.0, 0.0, 1.0), d_pore=2.3e-9, t1=0.1, t2=0.05, p_eq=0.5, diffusion=1, **kw)
    with bt.Solver(cfg) as s:
        s.upload_geometry(mask)
        for _ in range(2):  # the second one while the first one's buffers are in use
            st = rng.uniform(-1, 1, lead + shape) * mask
            s.set_state(st)
            got = s.get_state()
            assert got.shape == st.shape
            np.testing.assert_array_equal(got, st if precision == "f64" else st.astype(np.float32).astype(np.float64))
