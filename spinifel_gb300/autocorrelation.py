"""Forward (type 2) and adjoint (type 1) operators of the autocorrelation
merge, with the reference's signatures (spinifel/autocorrelation.py).

forward(ugrid, H_, K_, L_, support, use_recip_sym, N)      :32-61
adjoint(nuvect, H_, K_, L_, M, use_recip_sym=True, support=None)  :97-128
gen_nonuniform_positions / gen_nonuniform_normalized_positions   :290-323

The NUFFT runs on the GPU (libspinifel_gb300) at tolerance `eps`: FP32
kernels from the default 1e-6 (the GB300 path's specified tolerance) down to
about 1e-7, FP64 kernels below that, down to the 1e-12 in double that the
reference asks finufft for.  Inputs may be numpy arrays (results come back
as numpy) or CUDA tensors (results stay on the device).
"""
from __future__ import annotations

import numpy as np
import torch

from . import _arrays, _lib, geom
from .nufft import FP32_EPS_FLOOR, NufftPlan, make_plan

DEFAULT_EPS = 1e-6
_plans: dict = {}


def plan_for(M, eps=DEFAULT_EPS) -> NufftPlan:
    m = (M, M, M) if np.ndim(M) == 0 else tuple(M)
    key = (m, float(eps), torch.cuda.current_device())
    p = _plans.get(key)
    if p is None:
        p = make_plan(m, eps)
        _plans[key] = p
    return p


def _dtype(eps, *arrs) -> torch.dtype:
    """Device type to bring arrs to for a plan of eps: its own where they are on the
    device (converting to it at once gives what converting through FP64 gives),
    FP64 where they are not (the host converts slower than the copy and the device
    take: 67 / 55 us for 70,000 values, 195 / 152 for 2.1e6)."""
    on_device = all(_arrays.is_torch(a) and a.is_cuda for a in arrs)
    return torch.float32 if on_device and float(eps) >= FP32_EPS_FLOOR else torch.float64


def _numel(a) -> int:
    return a.numel() if _arrays.is_torch(a) else int(np.size(a))


def _max_abs(*arrs) -> float:
    a = arrs[0]
    if len(arrs) == 3 and all(_arrays.is_torch(t) and t.is_cuda and t.is_contiguous()
                              and t.dtype == a.dtype and t.device == a.device
                              and t.numel() == a.numel() for t in arrs) \
            and a.dtype in (torch.float32, torch.float64) \
            and a.device.index == torch.cuda.current_device():
        # one pass over the three arrays and one readback
        out = torch.empty(3, dtype=torch.float64, device=a.device)
        _lib.call("spf_max_abs3", *(_lib.ptr(t) for t in arrs), a.numel(),
                  int(a.dtype == torch.float64), _lib.ptr(out), _lib.stream_handle())
        return max(out.tolist())
    return max(float(a.abs().max()) if _arrays.is_torch(a) else float(np.max(np.abs(a)))
               for a in arrs)


def forward(ugrid, H_, K_, L_, support, use_recip_sym, N, eps=DEFAULT_EPS):
    """Type 2, isign -1: nuvect_j = sum_k (ugrid*support)_k exp(-i k.(H,K,L)_j)."""
    if _numel(H_):
        assert _max_abs(H_, K_, L_) < 3 * np.pi
    if use_recip_sym:
        if _arrays.is_torch(ugrid):
            assert not torch.is_complex(ugrid) or bool((ugrid.imag == 0).all())
        else:
            assert np.all(np.isreal(ugrid))
    g = _arrays.to_dev(ugrid.real if _arrays.is_torch(ugrid) and torch.is_complex(ugrid)
                       else (np.real(ugrid) if not _arrays.is_torch(ugrid) else ugrid),
                       _dtype(eps, ugrid))
    P = plan_for(g.shape, eps)
    P.set_modes(g, support, isign=-1, want_imag=True)
    x, y, z = (_arrays.to_dev(np.asarray(a).reshape(-1) if not _arrays.is_torch(a) else a,
                              _dtype(eps, a)) for a in (H_, K_, L_))
    re, im = P.interp(x, y, z, want_imag=True)
    out = torch.complex(re, im)
    assert out.numel() == N
    return _arrays.like_input(out, ugrid)


# from this many points on, the adjoint bin-sorts them once and spreads with
# the sorted kernel (a pencil's cells summed in registers) instead of one
# thread per point with global atomics.  Whole adjoint, sorted / per point:
# 517 / 530 us at 65,536 points on the 81^3 grid, 489 / 1,015 at 409,600 (41^3),
# 703 / 3,423 at 2,048,000; on grids with few points a bin
# NufftPlan.SORTED_MIN_PER_BIN decides.
SORTED_SPREAD_MIN_POINTS = 1 << 17


def adjoint(nuvect, H_, K_, L_, M, use_recip_sym=True, support=None, eps=DEFAULT_EPS,
            isign=+1, plan=None, sort=None):
    """Type 1 onto M^3 (isign +1), times support, real part, divided by M^3.
    sort: None picks the sorted spreading for large point sets (a smaller one
    never replaces points that the plan's caller sorted: NufftPlan.may_sort);
    True / False forces it on or off."""
    if _numel(H_):
        assert _max_abs(H_, K_, L_) < 3 * np.pi
    P = plan if plan is not None else plan_for(M, eps)
    x, y, z = (_arrays.to_dev(np.asarray(a).reshape(-1) if not _arrays.is_torch(a) else a,
                              P.dtype) for a in (H_, K_, L_))
    c = nuvect if _arrays.is_torch(nuvect) else torch.as_tensor(np.asarray(nuvect))
    c = c.to(_arrays.device()).reshape(-1)
    cre = (c.real if torch.is_complex(c) else c).to(P.dtype).contiguous()
    cim = c.imag.to(P.dtype).contiguous() if torch.is_complex(c) else None
    auto = sort is None and hasattr(P, "may_sort")
    use_sorted = (x.numel() >= SORTED_SPREAD_MIN_POINTS) if sort is None else bool(sort)
    use_sorted = use_sorted and P.supports_sort and (not auto or P.may_sort(x.numel()))
    if use_sorted:
        P.sort_points(x, y, z)
        if auto:
            P.sorted_automatically()

    def spread(values):
        if use_sorted:
            P.spread_sorted(values)
        else:
            P.spread(x, y, z, values)

    P.spread_zero()
    spread(cre)
    fr_re, fr_im = P.finish(isign, want_imag=True)
    re, im = fr_re, fr_im
    if cim is not None and bool((cim != 0).any()):
        P.spread_zero()
        spread(cim)
        fi_re, fi_im = P.finish(isign, want_imag=True)
        re = fr_re - fi_im
        im = fr_im + fi_re
    if support is not None:
        s = _arrays.to_dev(support, P.dtype) if not isinstance(support, (int, float)) else support
        re = re * s
        im = im * s
    out = re if use_recip_sym else torch.complex(re, im)
    out = out / float(M) ** 3
    return _arrays.like_input(out, nuvect)


def gen_nonuniform_positions(orientations, pixel_position_reciprocal):
    if orientations.shape[0] > 0:
        return geom.hkl(orientations, pixel_position_reciprocal)
    print("WARNING: gen_nonuniform_positions got empty orientation - returning h,k,l for "
          "Null rotation")
    return geom.hkl(np.zeros((0, 4)), pixel_position_reciprocal)


def gen_nonuniform_normalized_positions(orientations, pixel_position_reciprocal,
                                        reciprocal_extent, oversampling):
    H, K, L = gen_nonuniform_positions(orientations, pixel_position_reciprocal)
    s = np.pi / reciprocal_extent / oversampling
    return H.flatten() * s, K.flatten() * s, L.flatten() * s
