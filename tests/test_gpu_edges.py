"""Kernels at the sizes where their splits end: chunk and tile edges, rows
that are not 16-byte aligned, the smallest calls."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _frames_refs(n_img, n_ref, n_pix, seed, mean=2.0):
    rng = np.random.default_rng(seed)
    refs = rng.gamma(2.0, mean / 2, (n_ref, n_pix)).astype(np.float32)
    lam = refs[rng.integers(0, n_ref, n_img)]
    counts = np.minimum(rng.poisson(lam), 65535).astype(np.uint16)
    return counts, refs


@pytest.mark.parametrize("n_img,n_pix", [(1, 16), (1, 127), (5, 128), (3, 130), (2, 132),
                                         (7, 641), (4, 768), (9, 773), (300, 1284), (609, 260),
                                         (700, 66), (1976, 132), (1977, 131)])
def test_rerank_equals_plain_path(n_img, n_pix):
    """The re-ranked indices and distances are the plain path's, bit for bit,
    at whole and ragged chunks and for rows of any alignment."""
    from spinifel_gb300 import matching

    counts, refs = _frames_refs(n_img, 500, n_pix, 7 * n_pix + n_img)
    dev = torch.device("cuda")
    fs = matching.FrameSet.from_counts(torch.as_tensor(counts.view(np.int16), device=dev))
    rs = matching.ReferenceSet(torch.as_tensor(refs, device=dev))
    idx, dist = matching.match_bf16(fs, rs)
    pidx, pdist = matching.argmin_fp32(fs.f32, rs.f32, images_sq=fs.sq, refs_sq=rs.sq)
    assert torch.equal(idx, pidx)
    assert torch.equal(dist, pdist)


@pytest.mark.parametrize("n_pix", [8, 24, 333, 2048, 8200])
@pytest.mark.parametrize("top", [255, 4095, 4096, 65535])
def test_ingest_norms_are_exact_sums(n_pix, top):
    """Squared norms are the exact integer sums rounded once, 4-norms the
    square root of the exact sum within one FP32 rounding of it."""
    from spinifel_gb300 import matching

    rng = np.random.default_rng(n_pix + top)
    c = rng.integers(0, top + 1, (3, n_pix)).astype(np.uint16)
    c[0, :] = top
    dev = torch.device("cuda")
    fs = matching.FrameSet.from_counts(torch.as_tensor(c.view(np.int16), device=dev))
    s2 = [sum(int(v) ** 2 for v in row) for row in c]
    s4 = [sum(int(v) ** 4 for v in row) for row in c]
    assert torch.equal(fs.f32.cpu(), torch.as_tensor(c.astype(np.float32)))
    np.testing.assert_array_equal(fs.sq.cpu().numpy(), np.array(s2, dtype=np.float64)
                                  .astype(np.float32))
    np.testing.assert_allclose(fs.n4.cpu().numpy().astype(np.float64),
                               np.sqrt(np.array(s4, dtype=np.float64)), rtol=2 ** -23)


@pytest.mark.parametrize("n_pix", [1, 3, 32, 1000, 2048, 2049, 2052, 8200, 65537])
@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e-22, 1e15, 1e20])
def test_row_sqnorm_is_the_rounded_sum(n_pix, scale):
    """Within one FP32 rounding of the FP64 sum (2^-24, and 2^-30 for the sum
    itself), also where squares under- or overflow FP32; NaN and infinity stay."""
    from spinifel_gb300 import matching

    rng = np.random.default_rng(n_pix)
    x = (rng.standard_normal((5, n_pix)) * scale).astype(np.float32)
    x[1] = 0.0
    x[2, : n_pix // 2] *= 1e3
    x[3, n_pix // 2] = np.inf
    x[4, n_pix - 1] = np.nan
    got = matching.row_sqnorm(torch.as_tensor(x, device="cuda")).cpu().numpy()
    with np.errstate(over="ignore"):
        want = (x.astype(np.float64) ** 2).sum(axis=1).astype(np.float32)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_allclose(got[:4], want[:4], rtol=2 ** -24 * 1.02 + 2 ** -24,
                               atol=2 ** -149)


@pytest.mark.parametrize("n_pix,step", [(1024, 1), (1001, 32), (8192, 1), (8001, 256)])
def test_row_sqnorm_near_ties(n_pix, step):
    """Rows whose sum lies 2^-52 of itself past the middle between two floats,
    in elements that one thread adds up: as the rounded FP64 sum, which is exact."""
    from spinifel_gb300 import matching

    x = np.zeros((3, n_pix), dtype=np.float32)
    for r, first in enumerate((2.0 ** 12, 2.0 ** 20, 2.0 ** -8)):  # 2^2k + 2^(2k - 24)
        x[r, 0] = first
        x[r, step] = first * 2.0 ** -12
        x[r, 2 * step] = first * 2.0 ** -26
    got = matching.row_sqnorm(torch.as_tensor(x, device="cuda")).cpu().numpy()
    want = (x.astype(np.float64) ** 2).sum(axis=1).astype(np.float32)
    assert (want > x[:, 0].astype(np.float64) ** 2).all()
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n_img,n_ref,n_pix", [(1, 1, 1), (31, 33, 17), (64, 64, 16), (65, 129, 63),
                                               (128, 128, 64), (129, 2000, 100), (700, 1300, 37),
                                               (1500, 1400, 48), (33, 5000, 130)])
def test_distance_tiles(n_img, n_ref, n_pix):
    """Every tile of the distance kernels gives each pair's sequential chain:
    FP32 and FP64 squared differences against an FP64 reference, the fused
    argmin against the smallest of the distances it is defined on."""
    from spinifel_gb300 import matching

    rng = np.random.default_rng(n_img + n_ref)
    x = rng.random((n_img, n_pix)).astype(np.float32)
    r = rng.random((n_ref, n_pix)).astype(np.float32)
    xd, rd = torch.as_tensor(x, device="cuda"), torch.as_tensor(r, device="cuda")
    want = torch.cdist(xd.double(), rd.double(),
                       compute_mode="donot_use_mm_for_euclid_dist").square()
    got = matching.dist_f64(rd.double(), xd.double())
    torch.testing.assert_close(got, want, rtol=(n_pix + 4) * 2.0 ** -52, atol=1e-300)
    k16 = n_pix // 16 * 16
    if k16:
        w16 = (xd.double()[:, None, :k16] - rd.double()[None, :64, :k16]).square().sum(-1)
        g16 = matching.knn_eudist(rd[:64].contiguous(), xd)
        torch.testing.assert_close(g16.double(), w16, rtol=(n_pix + 4) * 2.0 ** -23, atol=1e-30)
    xs, rs = matching.row_sqnorm(xd), matching.row_sqnorm(rd)
    idx, dist = matching.argmin_fp32(xd, rd, xs, rs)
    # acc is a chain of n_pix FMAs: at most n_pix 2^-24 of the sum of |x s|
    err = (n_pix + 4) * 2.0 ** -24 * 2 * (xs.double()[:, None] + rs.double()[None, :])
    best = want.min(dim=1).values
    i = idx.long()
    rows = torch.arange(n_img, device="cuda")
    assert bool((dist.double() - want[rows, i]).abs().le(err[rows, i]).all())
    assert bool((want[rows, i] - best).le(2 * err.max(dim=1).values).all())


def _minima_case(kind, n_img, n_ref, n_pix):
    rng = np.random.default_rng(n_img + n_ref + n_pix)
    r = rng.gamma(2.0, 1.0, (n_ref, n_pix))
    x = rng.poisson(r[rng.integers(0, n_ref, n_img)]).astype(np.float64)
    if kind == "ties":            # every reference several times over
        r = r[rng.integers(0, max(1, n_ref // 5), n_ref)]
    elif kind == "equal":         # no list: all references tie
        r[:] = r[0]
    elif kind == "exact":         # frames that are references
        x = r[rng.integers(0, n_ref, n_img)].copy()
    elif kind == "close":         # apart by less than FP32 resolves
        r = r[:1] * (1 + 1e-12 * rng.standard_normal((n_ref, n_pix)))
    elif kind == "signed":
        x, r = rng.standard_normal((n_img, n_pix)), rng.standard_normal((n_ref, n_pix))
    elif kind == "tiny":
        x, r = x * 1e-25, r * 1e-25
    elif kind == "huge":
        r[::3] *= 1e20
    elif kind == "overflow":
        x, r = x * 1e200, r * 1e200
    elif kind == "zero":
        x[:] = 0.0
        r[0] = 0.0
    elif kind == "nan":
        r[::2, n_pix // 2] = np.nan
        x[0, 0] = np.inf
        if n_img > 1:
            x[1, n_pix - 1] = np.nan
    return x, r


@pytest.mark.parametrize("kind", ["plain", "ties", "equal", "exact", "close", "signed", "tiny",
                                  "huge", "overflow", "zero", "nan"])
@pytest.mark.parametrize("n_img,n_ref,n_pix", [(1, 1, 64), (33, 65, 257), (5, 700, 1025),
                                               (130, 1100, 130), (40, 300, 5000)])
def test_minima_equal_full_fp64_block(kind, n_img, n_ref, n_pix):
    """Picking minima gives the indices and distances of the whole FP64 block,
    bit for bit, in one batch and in several, whatever the values."""
    from spinifel_gb300 import matching

    x, r = _minima_case(kind, n_img, n_ref, n_pix)
    x, r = torch.as_tensor(x, device="cuda"), torch.as_tensor(r, device="cuda")
    for batch in (4096, (n_ref + 2) // 3):
        full = matching.BestTracker64(n_img, x.device)
        for st in range(0, n_ref, batch):
            full.update_block(matching.dist_f64(r[st:st + batch], x), st)
        idx, dist = matching.argmin_fp64(x, r, batch=batch)
        assert torch.equal(idx, full.best_idx)
        assert torch.equal(dist, full.best_dist)


@pytest.mark.parametrize("w,eps", [(3, 1e-2), (5, 1e-4), (7, 1e-6), (8, 1e-7)])
@pytest.mark.parametrize("n,spread", [(1, 3.0), (33, 3.0), (1025, 0.02), (5000, 3.0), (20000, 0.3),
                                      (70001, 3.1), ((1 << 19) - 1, 3.1), ((1 << 19) + 77, 3.1),
                                      (1 << 19, 0.05)])
def test_sorted_spread_equals_per_point_spread(w, eps, n, spread):
    """Bin sort and pencil spreading against one thread per point in the FP64
    plan of the same kernel width (in FP32 that form loses 5e-5 itself where
    2^19 points of one sign add to one cell): the same sums to FP32 rounding,
    for one point, points of one cell, dense clusters and whole grids."""
    from spinifel_gb300.nufft import NufftPlan, NufftPlan64

    rng = np.random.default_rng(n + w)
    P = NufftPlan((19, 24, 31), eps)
    assert P.width == w
    x, y, z = (torch.as_tensor(rng.uniform(-spread, spread, n).astype(np.float32), device="cuda")
               for _ in range(3))
    c = torch.as_tensor(rng.random(n).astype(np.float32), device="cuda")
    P64 = NufftPlan64((19, 24, 31), eps)
    assert P64.width == w
    P64.spread_zero()
    P64.spread(x, y, z, c)
    want = P64.finish(+1, want_imag=True)
    for values in (c, c):  # a second pass over one sort
        P.sort_points(x, y, z)
        P.spread_zero()
        P.spread_sorted(values)
        got = P.finish(+1, want_imag=True)
        # of the complex sums: near the origin the imaginary part alone cancels
        a, b = (torch.complex(re.double(), im.double()) for re, im in (got, want))
        assert float((a - b).norm() / b.norm()) < 1e-5
    from spinifel_gb300 import matching

    matching.check_device_error()


@pytest.mark.parametrize("M,det,n", [(41, (4, 32, 32), 30), (41, (4, 128, 128), 3),
                                     (41, (4, 16, 16), 9), (31, (3, 50, 37), 20),
                                     (61, (1, 7, 33), 40), (21, (2, 8, 16), 50),
                                     (25, (1, 9, 17), 12), (81, (1, 1, 1), 5)])
def test_default_patch_shape_gives_per_point_bits(M, det, n):
    """The patch shape picked by the pixels' spacing slices with the bits of
    the per-point kernel, bf16 copy included, whole and ragged patches alike."""
    from spinifel_gb300 import geom
    from spinifel_gb300.nufft import NufftPlan

    rng = np.random.default_rng(M + n)
    ppr, pdr = geom.flat_detector(*det)
    q = torch.as_tensor(geom.uniform_quaternions(n, rng).astype(np.float32), device="cuda")
    p = torch.as_tensor(ppr.reshape(3, -1).astype(np.float32), device="cuda")
    P = NufftPlan(M, 1e-6)
    P.set_modes(torch.as_tensor(rng.random((M, M, M)).astype(np.float32), device="cuda"))
    mult = np.pi / pdr.max()
    bf = [torch.empty(n, p.shape[1], dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    a = P.slice(q, p, mult, out_bf16=bf[0])
    b = P.slice(q, p, mult, out_bf16=bf[1], det_shape=det)
    assert torch.equal(a, b)
    assert torch.equal(bf[0], bf[1])


@pytest.mark.parametrize("m", [(9, 8, 7), (5, 12, 21), (16, 3, 2)])
@pytest.mark.parametrize("isign", [1, -1])
@pytest.mark.parametrize("eps", [1e-6, 1e-12])
def test_real_transforms_against_direct_sums(m, isign, eps):
    """Both halves of the spectrum, both signs, odd and even mode counts: type
    2 and type 1 against the direct sums at the plan's tolerance (20 eps, and
    1e-5 for what FP32 resolves)."""
    from oracle import nufft as onufft
    from spinifel_gb300.nufft import make_plan

    rng = np.random.default_rng(sum(m) + isign)
    P = make_plan(m, eps)
    dt = np.float32 if eps > 1e-7 else np.float64
    tol = 1e-5 if eps > 1e-7 else 20 * eps
    x, y, z = rng.uniform(-np.pi, np.pi, (3, 300)).astype(dt)
    f, c = rng.standard_normal(m).astype(dt), rng.standard_normal(300).astype(dt)
    t = [torch.as_tensor(v, device="cuda") for v in (x, y, z, c, f)]
    P.set_modes(t[4], isign=isign, want_imag=True)
    re, im = P.interp(*t[:3], want_imag=True)
    got = re.cpu().numpy() + 1j * im.cpu().numpy()
    want = onufft.nudft3d2(x.astype(float), y.astype(float), z.astype(float), f.astype(float),
                           isign)
    assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)
    P.spread_zero()
    P.spread(*t[:4])
    re, im = P.finish(isign, want_imag=True)
    got = re.cpu().numpy() + 1j * im.cpu().numpy()
    want = onufft.nudft3d1(x.astype(float), y.astype(float), z.astype(float), c.astype(float), m,
                           isign)
    assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [1, 31, 257, 1024, 100003])
def test_max_abs_equals_torch(dtype, n):
    """The range check's one-pass maximum is torch's, whichever array and
    sign holds it, and treats NaN and infinity as the maxima of torch do."""
    from spinifel_gb300 import autocorrelation as ac

    rng = np.random.default_rng(n)
    for where in range(3):
        v = [torch.as_tensor(rng.standard_normal(n), device="cuda", dtype=dtype)
             for _ in range(3)]
        v[where][n // 2] = -7.5
        assert ac._max_abs(*v) == 7.5
        for bad in (float("inf"), float("-inf"), float("nan")):
            v[where][n - 1] = bad
            want = max(float(t.abs().max()) for t in v)
            got = ac._max_abs(*v)
            assert got == want or (np.isnan(got) and np.isnan(want))
    assert ac._max_abs(*(torch.zeros(n, device="cuda", dtype=dtype) for _ in range(3))) == 0.0


def test_interp_pairs_equal_single_parts():
    """Both parts from one walk over the footprint: the real part has the bits
    of the walk over the real grid, also after a model without the imaginary
    part was set."""
    from spinifel_gb300.nufft import NufftPlan

    rng = np.random.default_rng(3)
    P = NufftPlan((11, 14, 9), 1e-6)
    x, y, z = (torch.as_tensor(rng.uniform(-3, 3, 501).astype(np.float32), device="cuda")
               for _ in range(3))
    for want_imag in (True, False):
        f = torch.as_tensor(rng.standard_normal((11, 14, 9)).astype(np.float32), device="cuda")
        P.set_modes(f, want_imag=want_imag)
        re, im = P.interp(x, y, z, want_imag=True)
        assert torch.equal(re, P.interp(x, y, z)[0])
        assert bool(torch.isfinite(im).all())


@pytest.mark.parametrize("eps", [1e-2, 1e-5, 1e-9, 1e-11, 1e-12, 1e-13, 1e-14])
@pytest.mark.parametrize("M,det,n", [(21, (4, 16, 16), 6), (13, (2, 9, 21), 5), (41, (1, 4, 8), 3),
                                     (31, (3, 5, 7), 4), (9, (1, 1, 1), 7)])
def test_fp64_slices_by_pairs(eps, M, det, n):
    """FP64 slices from pairs of floats against the direct sums: the plan's
    tolerance (20 eps, and 1e-13 for what the pairs and FP64 resolve), no
    further off than the FP64 kernel by more than a tenth and 1e-14."""
    from oracle import nufft as onufft
    from spinifel_gb300 import geom
    from spinifel_gb300.nufft import NufftPlan64

    rng = np.random.default_rng(M + n)
    ppr, pdr = geom.flat_detector(*det)
    q = geom.uniform_quaternions(n, rng)
    mult = np.pi / pdr.max()
    f = rng.standard_normal((M, M, M))
    P = NufftPlan64(M, eps)
    H, K, L = geom.hkl(q, ppr)
    want = onufft.nudft3d2(H.reshape(-1) * mult, K.reshape(-1) * mult, L.reshape(-1) * mult, f,
                           -1).real.reshape(n, -1)
    for scale in (1.0, 1e-200, 1e200, 3e-30):
        P.set_modes(torch.as_tensor(f * scale, device="cuda"))
        flat = P.slice(q, torch.as_tensor(ppr.reshape(3, -1), device="cuda"), mult)
        pair = P.slice(q, torch.as_tensor(ppr.reshape(3, -1), device="cuda"), mult, det_shape=det)
        e = [np.linalg.norm(v.cpu().numpy() / scale - want) / np.linalg.norm(want)
             for v in (flat, pair)]
        assert e[1] < max(20 * eps, 1e-13)
        assert e[1] <= 1.1 * e[0] + 1e-14


@pytest.mark.parametrize("eps", [1e-6, 1e-9, 1e-12])
def test_fp64_slices_by_pairs_kernel_values(eps):
    """Every pixel of a slice of a flat grid (one mode), which is the product of the
    three axes' sums of kernel values: pairs against the FP64 kernel to 6e-14
    (three axes of 1.1e-14, the largest error of a sum of pair values, and
    2^-46 for the sums over the footprint)."""
    from spinifel_gb300 import geom
    from spinifel_gb300.nufft import NufftPlan64

    rng = np.random.default_rng(21)
    M, det = 21, (4, 64, 64)
    ppr, pdr = geom.flat_detector(*det)
    q = geom.uniform_quaternions(16, rng)
    P = NufftPlan64(M, eps)
    f = np.zeros((M, M, M))
    f[M // 2, M // 2, M // 2] = 1.0
    P.set_modes(torch.as_tensor(f, device="cuda"))
    p = torch.as_tensor(ppr.reshape(3, -1), device="cuda")
    flat = P.slice(q, p, np.pi / pdr.max())
    pair = P.slice(q, p, np.pi / pdr.max(), det_shape=det)
    assert float(((pair - flat) / flat).abs().max()) < 6e-14


@pytest.mark.parametrize("bad", [0.0, 1e-310, float("inf"), float("nan")])
def test_fp64_slices_of_grids_pairs_cannot_hold(bad):
    """Zero, subnormal, infinite and NaN models take the FP64 kernel."""
    from spinifel_gb300 import geom
    from spinifel_gb300.nufft import NufftPlan64

    rng = np.random.default_rng(5)
    ppr, pdr = geom.flat_detector(2, 8, 8)
    q = geom.uniform_quaternions(3, rng)
    P = NufftPlan64(11, 1e-12)
    f = np.zeros((11, 11, 11))
    f[3, 4, 5] = bad
    P.set_modes(torch.as_tensor(f, device="cuda"))
    p = torch.as_tensor(ppr.reshape(3, -1), device="cuda")
    a = P.slice(q, p, np.pi / pdr.max())
    b = P.slice(q, p, np.pi / pdr.max(), det_shape=(2, 8, 8))
    assert torch.equal(torch.nan_to_num(a, nan=7.0), torch.nan_to_num(b, nan=7.0))


@pytest.mark.parametrize("n_img,n_ref,n_pix", [(1, 1, 4096), (5, 7, 2048), (5, 223, 3000),
                                               (3, 225, 4104), (128, 900, 2049),
                                               (129, 3000, 5000), (300, 20000, 2112),
                                               (1, 36000, 2050), (5, 7, 6400), (2, 223, 8200),
                                               (128, 900, 8193), (1, 36000, 8200)])
def test_split_tiles_give_the_same_lists(n_img, n_ref, n_pix):
    """Tiles cut along the pixels (where the rule cuts them) list, per tile and image, the 8 references
    of the undivided tile with the same distances up to FP32 rounding (no more
    than n_pix / 64 partial sums of x.s, so 1e-5 of its size), and the match
    is the plain path's."""
    from spinifel_gb300 import _lib, matching

    size = int(_lib.lib().spf_dist_topk_bf16_work_bytes(n_img, n_ref, n_pix))
    if n_pix > 6000:
        assert size > 0
    counts, refs = _frames_refs(n_img, n_ref, n_pix, n_img + n_ref, mean=1.0)
    fs = matching.FrameSet.from_counts(torch.as_tensor(counts.view(np.int16), device="cuda"))
    rs = matching.ReferenceSet(torch.as_tensor(refs, device="cuda"))
    tiles = int(_lib.lib().spf_dist_topk_bf16_tiles(n_ref))
    got = []
    for work in (None, torch.empty(max(size, 16), dtype=torch.uint8, device="cuda")):
        d = torch.full((tiles, n_img, 8), -1.0, device="cuda")
        i = torch.full((tiles, n_img, 8), -7, dtype=torch.int32, device="cuda")
        _lib.call("spf_dist_topk_bf16_work", _lib.ptr(fs.bf16), n_img, _lib.ptr(rs.bf16), n_ref,
                  n_pix, rs.ld, _lib.ptr(rs.sq), _lib.ptr(d), _lib.ptr(i),
                  _lib.ptr(work) if work is not None else None, size, _lib.stream_handle())
        got.append((d, i))
    (d0, i0), (d1, i1) = got
    tol = 1e-5 * float(rs.sq.max() + 2 * (rs.sq.max() * fs.sq.max()).sqrt())
    fin = torch.isfinite(d0)
    assert torch.equal(fin, torch.isfinite(d1))
    assert float((d0[fin] - d1[fin]).abs().max()) <= tol
    assert torch.equal(i0[~fin], i1[~fin])
    # a listed reference may differ only where its distance ties within rounding
    other = (i0 != i1) & fin
    assert float(other.float().mean()) < 0.01
    idx, dist = matching.match_bf16(fs, rs)
    pidx, pdist = matching.argmin_fp32(fs.f32, rs.f32, images_sq=fs.sq, refs_sq=rs.sq)
    assert torch.equal(idx, pidx)
    assert torch.equal(dist, pdist)
    matching.check_device_error()


def test_automatic_sort_leaves_the_callers_points():
    """Points that a caller sorted on a plan stay its sorted points when an
    automatic choice spreads others there (below 2^21): spread_sorted and the
    direct merge operator give the same sums after as before (to the FP32
    rounding of sums in another order)."""
    from spinifel_gb300 import autocorrelation as ac
    from spinifel_gb300 import geom
    from spinifel_gb300.merge import MergeOperator, antisupport
    from spinifel_gb300.nufft import NufftPlan

    rng = np.random.default_rng(8)
    M, n = 21, 1 << 18
    P = NufftPlan(M, 1e-6)
    mine, other = (tuple(torch.as_tensor(rng.uniform(-3, 3, n).astype(np.float32), device="cuda")
                         for _ in range(3)) for _ in range(2))
    c = torch.as_tensor(rng.random(n).astype(np.float32), device="cuda")
    ppr, pdr = geom.flat_detector(4, 32, 32)
    q = torch.as_tensor(geom.uniform_quaternions(n // 4096, rng).astype(np.float32),
                        device="cuda")
    ppr_t = torch.as_tensor(ppr.reshape(3, -1).astype(np.float32), device="cuda")
    mult = np.pi / pdr.max()
    half = tuple(v[:n // 2].contiguous() for v in other)

    def spread():
        P.spread_zero()
        P.spread_sorted(c)
        return P.finish(+1)[0]

    P.sort_points(*mine)
    want = spread()
    P.spread_zero()
    P.spread_orient(q, ppr_t, mult, c, det_shape=(4, 32, 32))
    got = spread()
    assert float((got - want).norm() / want.norm()) < 1e-5
    a = ac.adjoint(c[:n // 2], *half, M, plan=P)
    b = ac.adjoint(c[:n // 2], *half, M, plan=NufftPlan(M, 1e-6))
    assert float((a - b).norm() / b.norm()) < 1e-4  # per-point sums against sorted ones
    got = spread()
    assert float((got - want).norm() / want.norm()) < 1e-5

    op = MergeOperator(M, 2 * M, 1e-3, 1.0, torch.ones(M, M, M, device="cuda"), antisupport(M, 1))
    op.set_direct(P, q, ppr_t, mult)
    x = torch.as_tensor(rng.random(M ** 3), device="cuda")
    want = op.apply(x, form=op.DIRECT)
    ac.adjoint(c[:n // 2], *half, M, plan=P)
    got = op.apply(x, form=op.DIRECT)
    assert float((got - want).norm() / want.norm()) < 1e-5


def test_automatic_sort_is_not_captured():
    """spread_orient at a size that it sorts by itself is captured unsorted,
    on a plan that never sorted and on one that did; replays give the eager
    sums."""
    from spinifel_gb300 import geom
    from spinifel_gb300.nufft import NufftPlan

    rng = np.random.default_rng(9)
    M, n = 21, 1 << 18
    ppr, pdr = geom.flat_detector(4, 32, 32)
    q = torch.as_tensor(geom.uniform_quaternions(n // 4096, rng).astype(np.float32),
                        device="cuda")
    ppr_t = torch.as_tensor(ppr.reshape(3, -1).astype(np.float32), device="cuda")
    c = torch.as_tensor(rng.random(n).astype(np.float32), device="cuda")
    mult = np.pi / pdr.max()
    P = NufftPlan(M, 1e-6)

    def step():
        P.spread_zero()
        P.spread_orient(q, ppr_t, mult, c, det_shape=(4, 32, 32))
        return P.finish(+1)[0]

    for _ in range(2):
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = step()
        want = step()  # eager: sorted
        g.replay()
        torch.cuda.synchronize()
        assert float((out - want).norm() / want.norm()) < 1e-5


def test_sorts_are_refused_under_capture():
    """A sort called for under graph capture is an error (also where it would
    not have to allocate), and the plan's sorted points stay usable."""
    from spinifel_gb300 import _lib
    from spinifel_gb300.nufft import NufftPlan

    rng = np.random.default_rng(10)
    P = NufftPlan(21, 1e-6)
    pts = tuple(torch.as_tensor(rng.uniform(-3, 3, 3000).astype(np.float32), device="cuda")
                for _ in range(3))

    def spread():
        P.spread_zero()
        P.spread_sorted()
        return P.finish(+1)[0]

    P.sort_points(*pts)
    want = spread()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with pytest.raises(_lib.SpfError, match="capture"):
        with torch.cuda.graph(g):
            P.sort_points(*pts)
    got = spread()
    assert float((got - want).norm() / want.norm()) < 1e-5


def test_sorted_points_are_ordered_across_streams():
    """Sorts and passes over a plan's sorted points run in the order of their
    calls on whatever streams: a pass on another stream than its sort's
    waits for the sort, and the next sort for the pass."""
    from spinifel_gb300 import geom
    from spinifel_gb300.nufft import NufftPlan

    rng = np.random.default_rng(11)
    M, n = 21, 1 << 18
    P = NufftPlan(M, 1e-6)
    ppr, pdr = geom.flat_detector(4, 32, 32)
    ppr_t = torch.as_tensor(ppr.reshape(3, -1).astype(np.float32), device="cuda")
    quats = [torch.as_tensor(geom.uniform_quaternions(n // 4096, rng).astype(np.float32),
                             device="cuda") for _ in range(2)]
    pts = tuple(torch.as_tensor(rng.uniform(-3, 3, n).astype(np.float32), device="cuda")
                for _ in range(3))
    c = torch.as_tensor(rng.random(n).astype(np.float32), device="cuda")
    mult = np.pi / pdr.max()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()

    def sums(a, b):
        """two orientation spreads of one sum, a's stream held up"""
        P.spread_zero()
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            if a is not b:
                torch.cuda._sleep(20_000_000)  # about 10 ms
            P.spread_orient(quats[0], ppr_t, mult, c)
        with torch.cuda.stream(b):
            P.spread_orient(quats[1], ppr_t, mult, c)
        torch.cuda.synchronize()
        return P.finish(+1)[0]

    want = sums(s1, s1)
    for a, b in ((s1, s2), (s2, s1)):
        got = sums(a, b)
        assert float((got - want).norm() / want.norm()) < 1e-5

    def passed(a, b):
        P.spread_zero()
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            if a is not b:
                torch.cuda._sleep(20_000_000)
            P.sort_points(*pts)
        with torch.cuda.stream(b):
            P.spread_sorted(c)
            out = P.finish(+1)[0]
        torch.cuda.synchronize()
        return out

    want = passed(s1, s1)
    P.sort_points(*(v.flip(0) for v in pts))
    got = passed(s1, s2)
    assert float((got - want).norm() / want.norm()) < 1e-5


def _match_operands(n_img, n_ref, n_pix, seed):
    from spinifel_gb300 import matching

    rng = np.random.default_rng(seed)
    refs = rng.gamma(0.5, 1.0, (n_ref, n_pix)).astype(np.float32)
    x = rng.poisson(refs[rng.integers(0, n_ref, n_img)]).astype(np.float32)
    fr = matching.FrameSet(torch.as_tensor(x, device="cuda"))
    return fr, matching.ReferenceSet(torch.as_tensor(refs, device="cuda"))


@pytest.mark.parametrize("n_pix", [1024, 1001])
def test_late_rerank_frames_are_left_open(n_pix):
    """Frames whose re-rank gave up a wait (the test switch: every odd frame)
    are reported and uncertified, and their completion searches all references."""
    from spinifel_gb300 import _lib, matching

    fr, rs = _match_operands(9, 700, n_pix, 12)
    want_i, want_d = matching.argmin_fp32(fr.f32, rs.f32, images_sq=fr.sq, refs_sq=rs.sq)
    _lib.call("spf_tune_set", _lib.SPF_TUNE_STATIC_ABORT_TEST, 1)
    try:
        raw_i, raw_d = matching.match_bf16(fr, rs, exact_fallback=False)
        st = {}
        idx, dist = matching.match_bf16(fr, rs, stats=st)
    finally:
        _lib.call("spf_tune_set", _lib.SPF_TUNE_STATIC_ABORT_TEST, 0)
    with pytest.raises(_lib.SpfError, match="gave up"):
        matching.check_device_error()
    assert bool((raw_i[1::2] == -1).all()) and bool(raw_d[1::2].isnan().all())
    assert st["uncertified"] >= 4
    assert torch.equal(idx.to(want_i.dtype), want_i) and torch.equal(dist, want_d)
    matching.check_device_error()


@pytest.mark.parametrize("n_img,n_ref,n_pix,divided", [
    (9, 1500, 16384, True),    # parts of tiles
    (9, 700, 1000, False),     # whole tiles, one CTA a frame in the re-rank
    (2100, 40000, 64, False),  # several tiles a CTA, four frames a CTA
])
def test_gemm_that_gave_up_leaves_its_frames_open(n_img, n_ref, n_pix, divided):
    """When a wait of the tensor-core GEMM runs out (the test switch: at each
    CTA's last tile) the frames of the tiles left out are uncertified, whatever the
    candidate buffers held before, and their completion is exact."""
    from spinifel_gb300 import _lib, matching

    fr, rs = _match_operands(n_img, n_ref, n_pix, 13)
    size = int(_lib.lib().spf_dist_topk_bf16_work_bytes(n_img, n_ref, n_pix))
    assert (size > 0) == divided
    want_i, want_d = matching.argmin_fp32(fr.f32, rs.f32, images_sq=fr.sq, refs_sq=rs.sq)
    first = {}
    matching.match_bf16(fr, rs, stats=first)  # leaves its candidates in the buffers
    _lib.call("spf_tune_set", _lib.SPF_TUNE_STATIC_ABORT_TEST, 1)
    try:
        st = {}
        idx, dist = matching.match_bf16(fr, rs, stats=st)
    finally:
        _lib.call("spf_tune_set", _lib.SPF_TUNE_STATIC_ABORT_TEST, 0)
    with pytest.raises(_lib.SpfError, match="gave up"):
        matching.check_device_error()
    # as many tiles as CTAs were left out (every one of the small calls)
    tiles = int(_lib.lib().spf_dist_topk_bf16_tiles(n_ref)) * ((n_img + 127) // 128)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert st["uncertified"] == n_img or (tiles > sms and
                                          st["uncertified"] > first["uncertified"])
    assert torch.equal(idx.to(want_i.dtype), want_i) and torch.equal(dist, want_d)
    matching.check_device_error()


@pytest.mark.parametrize("n_ref", [1500, 200])
def test_overlapping_matches_keep_their_scratch_apart(n_ref):
    """match_bf16 calls in flight on several streams, from several threads,
    give each its own answer (products of divided tiles among the scratch)."""
    import threading

    from spinifel_gb300 import matching

    pairs = [_match_operands(n, n_ref, 16384, 20 + n) for n in (3, 5, 8, 13)]
    want = [matching.match_bf16(fr, rs) for fr, rs in pairs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in pairs]
    got = [None] * len(pairs)

    def work(k):
        for _ in range(10):
            got[k] = matching.match_bf16(*pairs[k], stream=streams[k])

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(pairs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for (i, d), (wi, wd) in zip(got, want):
        assert torch.equal(i, wi) and torch.equal(d, wd)
    matching.check_device_error()


def test_argmin_fp64_of_very_many_references():
    """More references than a launch has rows of blocks (65,535 x 512), with a frame
    that is compared with all of them: the FP64 minimum, lowest index on ties."""
    from spinifel_gb300 import _lib, matching

    n_ref = 65535 * 512 + 7
    g = torch.Generator(device="cuda").manual_seed(3)
    refs = torch.rand(n_ref, 1, dtype=torch.float64, device="cuda", generator=g)
    img = torch.tensor([[0.5], [2.0 ** 51]], dtype=torch.float64, device="cuda")
    refs[-1, 0] = 1.5 + 2.0 ** -3  # the large frame's nearest, in the last block
    size = int(_lib.lib().spf_argmin_f64_work_bytes(2, n_ref, 1))
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    t = matching.BestTracker64(2, img.device)
    _lib.call("spf_argmin_f64", _lib.ptr(img), 2, _lib.ptr(refs), n_ref, 1, 0, _lib.ptr(ws), size,
              _lib.ptr(t.best_dist), _lib.ptr(t.best_idx), _lib.stream_handle())
    idx, dist = t.result()
    for i in range(2):
        d = (img[i, 0] - refs[:, 0]) ** 2
        m = d.min()
        assert float(dist[i]) == float(m)
        assert int(idx[i]) == int(torch.nonzero(d == m)[0, 0])


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6, 1e-9])
def test_type1_of_the_smallest_grids(eps):
    """Grids of twice the kernel's width, whose halo wraps onto itself: type 1
    against the direct sums (20 eps, and 1e-5 for FP32)."""
    from oracle import nufft as onufft
    from spinifel_gb300.nufft import make_plan

    rng = np.random.default_rng(31)
    x, y, z = rng.uniform(-3, 3, (3, 500)).astype(np.float32)
    c = rng.random(500).astype(np.float32)
    dev = [torch.as_tensor(v, device="cuda") for v in (x, y, z, c)]
    for m in ((1, 1, 1), (2, 3, 4), (4, 1, 7), (5, 6, 2)):
        P = make_plan(m, eps)
        P.spread_zero()
        P.spread(*dev)
        re, im = P.finish(+1, want_imag=True)
        got = re.cpu().numpy() + 1j * im.cpu().numpy()
        want = onufft.nudft3d1(x, y, z, c, m, +1)
        assert np.linalg.norm(got - want) < max(20 * eps, 1e-5) * np.linalg.norm(want)


def test_plans_do_not_keep_explicit_coordinates():
    """After sort_points the plan has the points itself: the coordinate tensors
    may go, and the passes over the sorted points are as before."""
    import weakref

    from spinifel_gb300.nufft import NufftPlan

    rng = np.random.default_rng(33)
    P = NufftPlan(21, 1e-6)
    pts = [torch.as_tensor(rng.uniform(-3, 3, 5000).astype(np.float32), device="cuda")
           for _ in range(3)]
    P.spread_zero()
    P.spread(*pts, torch.ones(5000, device="cuda"))
    want = P.finish(+1)[0]
    P.sort_points(*pts)
    gone = [weakref.ref(v) for v in pts]
    pts.clear()
    assert all(r() is None for r in gone)
    junk = [torch.full((5000,), 7.0, device="cuda") for _ in range(6)]
    P.spread_zero()
    P.spread_sorted()
    got = P.finish(+1)[0]
    assert float((got - want).norm() / want.norm()) < 1e-5
    del junk


@pytest.mark.parametrize("n_data,n_ref", [(64, 20000), (640, 640), (2000, 8000), (129, 127)])
def test_fp64_distances_where_the_tile_changed(n_data, n_ref):
    """FP64 distance blocks of sizes that take other tiles than FP32 blocks of
    theirs, on reals (to the rounding of seven terms) and on integers (exactly)."""
    from spinifel_gb300 import matching

    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.rand(n_data, 7, dtype=torch.float64, device="cuda", generator=g)
    r = torch.rand(n_ref, 7, dtype=torch.float64, device="cuda", generator=g)
    got = matching.dist_f64(r, x).reshape(n_data, n_ref)
    want = ((x[:, None, :] - r[None, :, :]) ** 2).sum(2)
    assert float((got - want).abs().max()) < 8 * 2 ** -52 * 7
    xi, ri = (x * 100).round(), (r * 100).round()
    got = matching.dist_f64(ri, xi).reshape(n_data, n_ref)
    assert torch.equal(got, ((xi[:, None, :] - ri[None, :, :]) ** 2).sum(2))


@pytest.mark.parametrize("det", [(1, 1, 700), (1, 700, 1), (2, 300, 2), (5, 1, 7)])
@pytest.mark.parametrize("eps", [1e-6, 1e-12])
def test_fp64_slices_of_thin_panels(det, eps):
    """Panels a pixel or two wide: the FP64 kernel's bits where it is the quicker
    one, and never further from them than pairs may be (6e-14 of the largest)."""
    from spinifel_gb300 import geom
    from spinifel_gb300.nufft import NufftPlan64

    rng = np.random.default_rng(41)
    ppr = rng.standard_normal((3,) + det)
    q = geom.uniform_quaternions(4, rng)
    P = NufftPlan64(21, eps)
    P.set_modes(torch.as_tensor(rng.random((21, 21, 21)), device="cuda"))
    p = torch.as_tensor(ppr.reshape(3, -1), device="cuda")
    flat, got = P.slice(q, p, 0.7), P.slice(q, p, 0.7, det_shape=det)
    patches = det[0] * -(-det[1] // 4) * -(-det[2] // 8)
    units = -(-p.shape[1] // 32)
    if (0.12 + 2.3 / P.width) * patches > 0.95 * units:
        assert torch.equal(flat, got)
    assert float((flat - got).abs().max()) <= 6e-14 * float(flat.abs().max())


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6, 1e-7])
def test_slices_by_every_rule_of_the_patch_shape(eps):
    """Detectors and grids on every side of the shape's rule: the bits of the
    thread-per-point kernel, at every width."""
    from spinifel_gb300 import geom
    from spinifel_gb300.nufft import NufftPlan

    rng = np.random.default_rng(43)
    for M in (9, 41, 81):
        P = NufftPlan(M, eps)
        P.set_modes(torch.as_tensor(rng.random((M, M, M)), device="cuda"))
        for det in ((1, 1, 300), (1, 300, 1), (7, 8, 16), (3, 9, 17), (2, 24, 40), (1, 64, 64),
                    (1, 200, 200), (3, 2, 5), (1, 1, 1)):
            ppr = torch.as_tensor(rng.standard_normal((3, int(np.prod(det)))), device="cuda")
            q = torch.as_tensor(geom.uniform_quaternions(3, rng), device="cuda")
            assert torch.equal(P.slice(q, ppr, 0.5, det_shape=det), P.slice(q, ppr, 0.5))


@pytest.mark.parametrize("n_pix", [64, 65])
@pytest.mark.parametrize("per_sm", [4, 10, 13])
def test_rerank_at_the_lines_between_kernels(per_sm, n_pix):
    """One frame fewer, as many and one more than the frames an SM at which
    the re-rank changes kernels: the plain path's answer."""
    from spinifel_gb300 import matching

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    fr, rs = _match_operands(per_sm * sms + 1, 300, n_pix, 50 + per_sm)
    want_i, want_d = matching.argmin_fp32(fr.f32, rs.f32, images_sq=fr.sq, refs_sq=rs.sq)
    for n in (per_sm * sms - 1, per_sm * sms, per_sm * sms + 1):
        part = matching.FrameSet(fr.f32[:n], bf16=fr.bf16[:n], sq=fr.sq[:n], n4=fr.n4[:n])
        idx, dist = matching.match_bf16(part, rs)
        assert torch.equal(idx.to(want_i.dtype), want_i[:n]) and torch.equal(dist, want_d[:n])


@pytest.mark.parametrize("eps", [1e-6, 1e-12])
def test_forward_takes_every_kind_of_array(eps):
    """numpy, host and device tensors of both types: the same values bit for bit where
    the inputs are, single precision's where they are single."""
    from spinifel_gb300 import autocorrelation as ac

    rng = np.random.default_rng(61)
    M, n = 15, 700
    model = rng.random((M, M, M)).astype(np.float32)
    pts = [rng.uniform(-3, 3, n).astype(np.float32) for _ in range(3)]
    want = ac.forward(model, *pts, 1.0, True, n, eps=eps)
    assert isinstance(want, np.ndarray)
    for dt in (np.float32, np.float64):  # the same values in both types
        a = [v.astype(dt) for v in (model, *pts)]
        for dev in (None, "cpu", "cuda"):
            b = a if dev is None else [torch.as_tensor(v, device=dev) for v in a]
            got = ac.forward(*b, 1.0, True, n, eps=eps)
            got = got if dev is None else got.cpu().numpy()
            np.testing.assert_array_equal(got, want)
