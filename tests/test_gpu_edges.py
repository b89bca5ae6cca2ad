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
