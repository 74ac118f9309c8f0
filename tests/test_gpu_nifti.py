"""NIfTI on the GPU: the library's device decode (byte order, scaling,
reorientation) and header writer against the numpy restatement
(oracle/nifti.py), bit for bit, and file round trips through loadNii /
saveNii (.nii, .nii.gz, .hdr/.img pairs) with host and device images."""
import numpy as np
import pytest

from test_nifti import CASES, build_header

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nio(port):
    import nifti
    return nifti


@pytest.fixture(scope="module")
def qn(gpu_ctx):
    from qsm_gb300 import nifti
    return nifti


def _payload(nio, dt, n, endian, seed):
    rng = np.random.default_rng(seed)
    t = np.dtype(nio.DT[dt])
    if t.kind == "f":
        a = (rng.standard_normal(n) * 100).astype(t)
    else:
        info = np.iinfo(t)
        a = rng.integers(max(info.min, -(1 << 40)), min(info.max, 1 << 40), n, dtype=t, endpoint=True)
    return a.astype(t.newbyteorder(endian)).tobytes()


@pytest.mark.parametrize("dt", [2, 4, 8, 16, 64, 256, 512, 768, 1024, 1280])
@pytest.mark.parametrize("case", ["identity_sform", "permuted_sform", "qform_rot90_qfac", "four_d", "analyze"])
@pytest.mark.parametrize("endian", ["<", ">"])
def test_decode_bitexact(qn, nio, dt, case, endian):
    kw = dict(CASES[case])
    kw["datatype"] = dt
    if dt in (2, 4, 256, 512) and case == "identity_sform":
        kw.update(slope=0.25, inter=-3.0)  # load_nii scales these to single
    if dt == 64 and case == "permuted_sform":
        kw.update(slope=1.5, inter=2.0)    # a scaled double stays double
    hb = build_header(endian, **kw)
    dim = kw.get("dim", (3, 6, 5, 4, 1, 1, 1, 1))
    n = int(np.prod(dim[1:]))
    pl = _payload(nio, dt, n, endian, dt + len(case))
    ref, rh = nio.load_nii(hb, pl)
    img, h = qn.decode(hb, pl)
    assert img.dtype == ref.dtype and img.shape == ref.shape
    assert np.array_equal(img, ref)
    for odt in (np.float32, np.float64):
        out, _ = qn.decode(hb, pl, out_dtype=odt)
        assert out.dtype == odt and np.array_equal(out, ref.astype(odt))


def test_decode_to_device(qn, nio):
    torch = pytest.importorskip("torch")
    kw = dict(CASES["permuted_sform"], datatype=4, slope=0.5, inter=1.0, dim=(4, 20, 18, 16, 3, 1, 1, 1))
    hb = build_header("<", **kw)
    pl = _payload(nio, 4, 20 * 18 * 16 * 3, "<", 7)
    ref, _ = nio.load_nii(hb, pl)
    d, _ = qn.decode(hb, pl, device=True)
    assert d.is_cuda and d.dtype == torch.float32
    assert np.array_equal(d.cpu().numpy().transpose(3, 2, 1, 0), ref)
    # stored bytes already in HBM
    dp = torch.from_numpy(np.frombuffer(pl, np.uint8).copy()).cuda()
    d2, _ = qn.decode(hb, dp, device=True, out_dtype=np.float64)
    assert np.array_equal(d2.cpu().numpy().transpose(3, 2, 1, 0), ref.astype(np.float64))


@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.int16, np.uint8, np.int32, np.uint16, np.int8,
                                   np.uint32])
def test_header_bitexact(qn, nio, dtype):
    rng = np.random.default_rng(3)
    img = np.asfortranarray((rng.standard_normal((9, 8, 7, 2)) * 60).astype(dtype))
    if np.dtype(dtype).kind == "f":
        img[0, 0, 0, 0] = np.nan  # ignored by max / min
    assert qn.header_bytes(img, (0.9, 1.1, 1.3)) == nio.make_header(img, (0.9, 1.1, 1.3))
    assert qn.header_bytes(img, (1, 1, 1), filetype=1) == nio.make_header(img, (1, 1, 1), filetype=1)


def test_file_round_trips(qn, nio, tmp_path):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    chi = np.asfortranarray(rng.standard_normal((24, 20, 16)))
    for name in ("chi.nii", "sub/chi.nii.gz", "pair/chi.hdr", "pairgz/chi.img.gz"):
        fn = str(tmp_path / name)
        qn.saveNii(fn, chi, [1.0, 0.9, 1.1])  # makes the directory, as saveNii.m does
        nii = qn.load_nii(fn)
        assert nii.img.dtype == np.float64 and np.array_equal(nii.img, chi)
        np.testing.assert_allclose(nii.hdr["pixdim"][1:4], [1.0, 0.9, 1.1], rtol=1e-7)
    raw = open(tmp_path / "chi.nii", "rb").read()
    assert raw == nio.save_bytes(chi, [1.0, 0.9, 1.1])
    ref, _ = nio.load_nii(raw[:352], raw[352:])
    assert np.array_equal(qn.loadNii(str(tmp_path / "chi.nii")).img, ref)
    # a device image saved and read back to the device
    dev = torch.from_numpy(np.ascontiguousarray(chi.astype(np.float32).T)).cuda()
    qn.saveNii(str(tmp_path / "dev.nii.gz"), dev, [1, 1, 1])
    back = qn.loadNii(str(tmp_path / "dev.nii.gz"), device=True)
    assert torch.equal(back.img, dev)
    with pytest.raises(ValueError, match="extension"):
        qn.loadNii(str(tmp_path / "pair" / "chi.hdr"))


def test_misaligned_device_payload_is_rejected(qn, nio):
    """Whole-word loads need an aligned payload: a device buffer at an odd byte
    offset is refused before any launch."""
    torch = pytest.importorskip("torch")
    from qsm_gb300 import _lib
    hb = build_header("<", datatype=4)
    pl = _payload(nio, 4, 6 * 5 * 4, "<", 1)
    buf = torch.zeros(len(pl) + 1, dtype=torch.uint8, device="cuda")
    buf[1:] = torch.from_numpy(np.frombuffer(pl, np.uint8).copy()).cuda()
    with pytest.raises(_lib.QsmError, match="aligned"):
        qn.decode(hb, buf[1:])
    img, _ = qn.decode(hb, buf[1:].clone())
    ref, _ = nio.load_nii(hb, pl)
    assert np.array_equal(img, ref)


def test_fortran_ordered_tensor_saves_in_matlab_order(qn, nio, tmp_path):
    torch = pytest.importorskip("torch")
    chi = np.asfortranarray(np.random.default_rng(8).standard_normal((12, 10, 8)).astype(np.float32))
    f_tensor = torch.from_numpy(np.ascontiguousarray(chi.T)).cuda().permute(2, 1, 0)  # F-contiguous, MATLAB size
    c_tensor = torch.from_numpy(np.ascontiguousarray(chi.T)).cuda()     # C-contiguous, shape reversed
    for t, name in ((f_tensor, "f.nii"), (c_tensor, "c.nii")):
        qn.saveNii(str(tmp_path / name), t, [1, 1, 1])
        assert open(tmp_path / name, "rb").read() == nio.save_bytes(chi, [1, 1, 1])
    with pytest.raises(ValueError, match="contiguous"):
        qn.header_bytes(torch.zeros((6, 6, 6), device="cuda")[:, ::2, :])


@pytest.mark.parametrize("dt", [2, 256, 4, 512, 16])
@pytest.mark.parametrize("slope,inter", [(0.1, 0.0), (0.1, -0.3), (1.0, 0.0), (1.0, 16777216.0), (2.0, 16777217.0), (0.25, -3.0),
                                         (3e-4, 1234.5), (-7.7, 1e-5), (1.0, -100.0), (1e-30, 1.0), (2.0 ** -24, 1.0),
                                         (3 * 2.0 ** -25, 1.0), (1e25, -1e12)])
def test_scaling_in_singles_bitexact(qn, nio, dt, slope, inter):
    """Scaled 8- and 16-bit and single images: every stored value (singles: also
    zeros of both signs, subnormals, huge values, infinities, NaN), with factors
    whose sums are exact, fall midway between two singles, cancel, or leave the
    range the single arithmetic takes.  Bit for bit against load_nii's formula,
    single(slope * double(x) + inter)."""
    t = np.dtype(nio.DT[dt])
    if t.kind == "f":
        rng = np.random.default_rng(3)
        x = (rng.standard_normal(65536) * 10.0 ** rng.uniform(-45, 38, 65536)).astype(t)
        x[:9] = [0.0, -0.0, 1e-45, -1e-38, 3e38, np.inf, -np.inf, np.nan, 1.0]
        x[9:4000] = np.arange(9, 4000)
    else:
        x = np.arange(1 << (8 * t.itemsize)).astype(np.dtype("u%d" % t.itemsize)).view(t)
    n = x.size
    hb = build_header("<", datatype=dt, dim=(3, 32, n // 32, 1, 1, 1, 1, 1), slope=slope, inter=inter)
    s32, i32 = np.float64(np.float32(slope)), np.float64(np.float32(inter))
    with np.errstate(all="ignore"):
        want = (s32 * x.astype(np.float64) + i32).astype(np.float32)
    img, h = qn.decode(hb, x.tobytes())
    if (slope, inter) == (1.0, 0.0):  # load_nii applies no such scaling: the stored class as it is
        assert not h.scaled and img.dtype == t and img.tobytes(order="F") == x.tobytes()
        return
    assert h.scaled and img.dtype == np.float32
    got = img.ravel(order="F")
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))
    wide = qn.decode(hb, x.tobytes(), out_dtype=np.float64)[0].ravel(order="F")
    assert np.array_equal(wide[~nan], want[~nan].astype(np.float64))


@pytest.mark.parametrize("dt", [2, 4, 16])
@pytest.mark.parametrize("nx", [4, 8, 30, 33, 260])
@pytest.mark.parametrize("sx", [1, -1])
@pytest.mark.parametrize("endian", ["<", ">"])
def test_scaling_quads(qn, nio, dt, nx, sx, endian):
    """Rows of four-voxel quads (row length a multiple of four, running along the
    stored rows in either direction) and rows that are none, from aligned device
    buffers and ones that start inside a quad."""
    torch = pytest.importorskip("torch")
    kw = dict(datatype=dt, dim=(4, nx, 5, 3, 2, 1, 1, 1), slope=0.37, inter=-3.1, sform=1,
              srow=[[sx, 0, 0, 0], [0, -1, 0, 0], [0, 0, 1, 0]])
    hb = build_header(endian, **kw)
    pl = _payload(nio, dt, nx * 30, endian, nx)
    ref, _ = nio.load_nii(hb, pl)
    esz = np.dtype(nio.DT[dt]).itemsize
    for shift in (0, esz):
        buf = torch.zeros(len(pl) + 64, dtype=torch.uint8, device="cuda")
        buf[shift:shift + len(pl)] = torch.from_numpy(np.frombuffer(pl, np.uint8).copy()).cuda()
        img, _ = qn.decode(hb, buf[shift:shift + len(pl)], device=True)
        got = img.cpu().numpy().T
        assert got.shape == ref.shape and np.array_equal(got, ref)


@pytest.mark.parametrize("dt,inter,unit", [(2, -0.3, 1.0), (16, -3.0, 1.0), (16, 0.0, 1e-14)])
def test_scaling_time_does_not_depend_on_midway_values(qn, dt, inter, unit):
    """Results midway between two singles are common (8-bit images with a slope of
    0.1: one voxel in 256; singles with 0.25 and -3: half of them) and take about
    the time of an image without any (0.25, and an intercept of 0 for the singles):
    at most twice, where FP64 per voxel takes over four times.  Nor on the unit of
    singles (1e-14)."""
    import time

    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(4)
    n = 224 * 224 * 128 * 2
    raw = rng.integers(0, 256, n, dtype=np.uint8) if dt == 2 else (rng.standard_normal(n) * 500).astype(np.float32).view(np.uint8)
    dev = torch.from_numpy(raw).cuda()
    small = dev if dt == 2 else (dev.view(torch.float32) * unit).view(torch.uint8)

    def best(slope, inter, dev=dev):
        hb = build_header("<", datatype=dt, dim=(4, 224, 224, 128, 2, 1, 1, 1), slope=slope, inter=inter)
        ts = []
        for _ in range(20):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            qn.decode(hb, dev, device=True)
            torch.cuda.synchronize()
            ts.append(time.perf_counter() - t0)
        return min(ts)

    plain = best(0.25, -3.0) if dt == 2 else best(0.25, 0.0)
    ties = best(0.1, inter) if dt == 2 else best(0.25, inter, small)
    assert ties < 2 * plain, (ties, plain)


@pytest.mark.parametrize("slope", [0.1, 1e-30])
def test_large_8_bit_image_to_double(qn, nio, slope):
    """8-bit images of 12 M voxels or more to double go through the table of their
    256 results, as images with factors outside the singles' range do."""
    x = np.random.default_rng(6).integers(0, 256, (240, 220, 230), dtype=np.uint8)
    hb = build_header("<", datatype=2, dim=(3, 240, 220, 230, 1, 1, 1, 1), slope=slope, inter=-0.3)
    want = (np.float64(np.float32(slope)) * x + np.float64(np.float32(-0.3))).astype(np.float32).astype(np.float64)
    img, _ = qn.decode(hb, x.tobytes(order="F"), out_dtype=np.float64)
    assert np.array_equal(img, want)
