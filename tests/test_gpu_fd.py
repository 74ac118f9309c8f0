"""GPU finite-difference operators against the oracle and the reference's
golden outputs: bit-for-bit, FP64 and FP32, host and device arrays."""
import numpy as np
import pytest

from conftest import bits_equal, first_diff

pytestmark = pytest.mark.gpu

GRADS = ("gradf", "gradb", "gradc", "gradfp")
GRADMS = ("gradfm", "gradbm", "gradcm")
ADJS = ("gradf_adj", "gradb_adj", "gradfp_adj")
ADJMS = ("gradfm_adj", "gradbm_adj")


def _z(shape, dt):
    return np.zeros(shape, dtype=dt, order="F")


@pytest.mark.parametrize("dt", ("float64", "float32"))
def test_fd_golden(gpu_ctx, qsm, golden, dt):
    g = golden("fd_ops")
    h = g["h"]
    for si in range(int(g["nshapes"])):
        tag = f"s{si}_{dt}"
        u, x, y, w, G, uw = (g[f"{tag}_{k}"] for k in ("u", "x", "y", "z", "G", "uw"))
        shape = u.shape
        for nm in GRADS + GRADMS:
            r = [_z(shape, dt) for _ in range(3)]
            args = (u, G, h) if nm in GRADMS else (u, h)
            getattr(qsm, nm + "_mex")(*r, *args)
            ref = g[f"{tag}_{nm}"]
            for c in range(3):
                assert bits_equal(r[c], np.asfortranarray(ref[..., c])), f"{nm}{shape}[{c}] {first_diff(r[c], ref[..., c])}"
        for nm in ADJS + ADJMS:
            r = _z(shape, dt)
            args = (x, y, w, G, h) if nm in ADJMS else (x, y, w, h)
            getattr(qsm, nm + "_mex")(r, *args)
            assert bits_equal(r, g[f"{tag}_{nm}"]), f"{nm}{shape} {first_diff(r, g[f'{tag}_{nm}'])}"
        r = _z(shape, dt)
        qsm.lap1_mex(r, u, G, h)
        assert bits_equal(r, g[f"{tag}_lap1"]), f"lap1{shape} {first_diff(r, g[f'{tag}_lap1'])}"
        r = _z(shape, dt)
        qsm.lapw_mex(r, uw, h)
        assert bits_equal(r, g[f"{tag}_lapw"]), f"lapw{shape}"


@pytest.mark.parametrize("shape", [(64, 48, 40), (129, 67, 33), (31, 200, 9)])
@pytest.mark.parametrize("dt", ("float64", "float32"))
def test_fd_vs_oracle_larger(gpu_ctx, qsm, port, shape, dt):
    """Sizes beyond the fixtures (partial tiles, odd extents) against the oracle."""
    rng = np.random.default_rng(hash((shape, dt)) % 2**32)
    u = np.asfortranarray(rng.standard_normal(shape).astype(dt))
    x, y, w = (np.asfortranarray(rng.standard_normal(shape).astype(dt)) for _ in range(3))
    G = np.asfortranarray((rng.random(shape) > 0.2).astype(np.uint8))
    h = [0.8, 1.0, 1.1]
    for nm in GRADS + GRADMS:
        a = [_z(shape, dt) for _ in range(3)]
        b = [_z(shape, dt) for _ in range(3)]
        args = (u, G, h) if nm in GRADMS else (u, h)
        getattr(qsm, nm + "_mex")(*a, *args)
        getattr(port, nm + "_mex")(*b, *args)
        for c in range(3):
            assert bits_equal(a[c], b[c]), f"{nm}[{c}] {first_diff(a[c], b[c])}"
    for nm in ADJS + ADJMS:
        a, b = _z(shape, dt), _z(shape, dt)
        args = (x, y, w, G, h) if nm in ADJMS else (x, y, w, h)
        getattr(qsm, nm + "_mex")(a, *args)
        getattr(port, nm + "_mex")(b, *args)
        assert bits_equal(a, b), f"{nm} {first_diff(a, b)}"
    a, b = _z(shape, dt), _z(shape, dt)
    qsm.lap1_mex(a, u, G, h)
    port.lap1_mex(b, u, G, h)
    assert bits_equal(a, b)
    uw = np.asfortranarray((rng.standard_normal(shape) * 5).astype(dt))
    a, b = _z(shape, dt), _z(shape, dt)
    qsm.lapw_mex(a, uw, h)
    port.lapw_mex(b, uw, h)
    assert bits_equal(a, b)


def test_fd_device_tensors(gpu_ctx, qsm, port):
    """torch CUDA tensors are used in place (C-order (nz,ny,nx) == MATLAB x-fastest)."""
    torch = pytest.importorskip("torch")
    shape = (40, 33, 21)
    rng = np.random.default_rng(5)
    u = np.asfortranarray(rng.standard_normal(shape))
    ut = torch.from_numpy(np.ascontiguousarray(u.transpose(2, 1, 0))).cuda()
    d = [torch.zeros_like(ut) for _ in range(3)]
    qsm.gradc_mex(*d, ut, [1, 1, 1])
    ref = [_z(shape, "float64") for _ in range(3)]
    port.gradc_mex(*ref, u, [1, 1, 1])
    for c in range(3):
        got = d[c].cpu().numpy().transpose(2, 1, 0)
        assert bits_equal(np.asfortranarray(got), ref[c])


def test_masked_leaves_untouched(gpu_ctx, qsm):
    """Masked operators only write where G (the rest keeps the caller's data)."""
    shape = (10, 9, 8)
    u = np.asfortranarray(np.random.default_rng(1).standard_normal(shape))
    G = np.zeros(shape, np.uint8, order="F")
    G[2:7, 2:6, 2:5] = 1
    sentinel = 7.25
    d = [np.full(shape, sentinel, order="F") for _ in range(3)]
    qsm.gradcm_mex(*d, u, G, [1, 1, 1])
    for c in range(3):
        assert np.all(d[c][G == 0] == sentinel)


def test_fd_errors(gpu_ctx, qsm):
    a = np.zeros((1, 4, 4), order="F")
    with pytest.raises(qsm.QsmError, match="DIMS"):
        qsm.gradf_mex(a.copy(order="F"), a.copy(order="F"), a.copy(order="F"), a, [1, 1, 1])
    b = np.zeros((4, 4, 4), np.float32, order="F")
    with pytest.raises(TypeError):
        qsm.gradf_mex(b, b.copy(order="F"), b.copy(order="F"), np.zeros((4, 4, 4), order="F"), [1, 1, 1])


@pytest.mark.parametrize("dt,shape", [("float32", (130, 125, 127)), ("float32", (63, 4, 8001)), ("float32", (3, 700, 960)),
                                      ("float32", (125, 127, 125)), ("float64", (33, 19, 220)), ("float64", (96, 35, 41)),
                                      ("float64", (3, 209, 210)), ("float64", (65, 48, 41))])
def test_lapw_both_forms_vs_oracle(gpu_ctx, qsm, port, dt, shape):
    """The wrapped Laplacian in columns (from 2 M voxels in FP32, 130 k in FP64) and
    one voxel per thread (the fourth and the last case lie just below): tile edges,
    thin volumes, several turns.  Bit-for-bit against the oracle."""
    u = np.asfortranarray((np.random.default_rng(sum(shape)).standard_normal(shape) * 6).astype(dt))
    u[::7] *= 40
    a, b = np.full(shape, 7.0, dt, order="F"), np.full(shape, 7.0, dt, order="F")
    qsm.lapw_mex(a, u, [0.7, 1.0, 1.3])
    port.lapw_mex(b, u, [0.7, 1.0, 1.3])
    assert bits_equal(a, b), first_diff(a, b)


@pytest.mark.parametrize("shape", [(3, 3, 3), (32, 5, 4), (33, 19, 20), (34, 18, 3), (65, 6, 37), (96, 35, 18)])
@pytest.mark.parametrize("dt", ("float64", "float32"))
def test_lapw_tiles_and_wraps_vs_oracle(gpu_ctx, qsm, port, shape, dt):
    """The wrapped Laplacian's tiles (31 voxels per warp, 4 rows and up to 16
    planes per thread) at their edges, with phase differences that are exactly
    pi, one unit beside it, several turns away (the general fmod), and huge.
    Bit-for-bit against the oracle; infinities and NaNs give NaN where it does."""
    rng = np.random.default_rng(sum(shape))
    u = (rng.standard_normal(shape) * 4).astype(dt)
    pi = np.asarray(np.pi, dtype=dt)
    pick = rng.integers(0, 12, shape)
    for q, v in enumerate((0.0, -0.0, pi, -pi, np.nextafter(pi, pi.dtype.type(9)), 3 * pi,
                           -3 * pi, 50.0, -1e6)):
        u[pick == q] = v
    u = np.asfortranarray(u)
    a, b = np.full(shape, 7.0, dt, order="F"), np.full(shape, 7.0, dt, order="F")
    qsm.lapw_mex(a, u, [0.7, 1.0, 1.3])
    port.lapw_mex(b, u, [0.7, 1.0, 1.3])
    assert bits_equal(a, b), first_diff(a, b)
    u[1::2, 0::3, 1::2] = np.inf
    u[0::3, 1::2, 0::2] = np.nan
    qsm.lapw_mex(a, u, [0.7, 1.0, 1.3])
    port.lapw_mex(b, u, [0.7, 1.0, 1.3])
    assert np.array_equal(np.isnan(a), np.isnan(b))
    ok = ~np.isnan(b)
    assert bits_equal(np.asfortranarray(np.where(ok, a, 0)), np.asfortranarray(np.where(ok, b, 0)))
