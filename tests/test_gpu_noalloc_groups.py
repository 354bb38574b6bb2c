"""sph_density_noalloc takes a cell's targets in groups of 32, 16, 8 or 4 by the
particle count: one cloud per group size, half of it in a dense ball (cells of
many groups, windows that fill several times) and half sparse (part-filled
groups, empty cells), against the oracle.  FP64 1e-12, FP32 1e-5 relative, as the
entry point's other tests.
"""
import ctypes as C

import numpy as np
import pytest

from spearhed_b200 import abi

pytestmark = pytest.mark.gpu

TOL = {abi.PREC_FP64: 1e-12, abi.PREC_FP32_COMP: 1e-5}


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_FP32_COMP])
@pytest.mark.parametrize("n,kernel", [(33, abi.KERNEL_CUBIC), (9001, abi.KERNEL_WENDLAND_C2),
                                      (20011, abi.KERNEL_QUINTIC), (40009, abi.KERNEL_CUBIC),
                                      (80021, abi.KERNEL_WENDLAND_C2)])
def test_every_group_size_matches_oracle(oracle, prec, n, kernel):
    import torch
    rng = np.random.default_rng(n)
    s = abi.Species(n)
    s.pos[:] = rng.uniform(0.0, 1.0, (3, n))
    # the ball's density is about eight times the cloud's
    m = n // 2
    d = rng.normal(size=(3, m))
    s.pos[:, :m] = 0.5 + 0.31 * d / np.linalg.norm(d, axis=0) * rng.uniform(0, 1, m) ** (1 / 3)
    sup = 3 if kernel == abi.KERNEL_QUINTIC else 2
    h0 = min((40.0 / n * 3 / (4 * np.pi)) ** (1 / 3) / sup, 0.15)
    s.h[:] = h0 * rng.uniform(0.8, 1.2, n)  # above and below the cull radius' h
    s.mass[:] = rng.uniform(0.5, 1.5, n) / n
    p = abi.default_params(kernel=kernel, precision=prec, h0=h0)
    box = abi.make_box((0, 0, 0), (1, 1, 1), (0, 1, 1))
    cols = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (*s.pos, s.mass, s.h)]
    rho = torch.empty(n, dtype=torch.float64, device="cuda")
    abi.check(abi.lib().sph_density_noalloc(C.byref(p), C.byref(box), n, *[c.data_ptr() for c in cols],
                                            rho.data_ptr(), torch.cuda.current_stream().cuda_stream))
    po = abi.SphParams.from_buffer_copy(p)
    po.precision = abi.PREC_FP64
    orc = oracle.System(po, [box], s.copy(), np.full(n, abi.ROLES_DEFAULT, dtype=np.uint8))
    orc.density(fp32_geometry=prec == abi.PREC_FP32_COMP)
    assert np.max(np.abs(rho.cpu().numpy() / orc.s.density - 1.0)) <= TOL[prec]


@pytest.mark.parametrize("prec,h0", [(abi.PREC_FP32_COMP, 1e-24), (abi.PREC_FP32_COMP, 1.5e-23),
                                     (abi.PREC_FP64, 1e-165), (abi.PREC_FP64, 1.5e-162)])
def test_radius_whose_square_underflows(oracle, prec, h0):
    """R^2 rounds to zero (first of each precision: the density is the self term
    alone) or to a few denormal steps (second: the pairs whose rounded r^2 is
    below it count)."""
    import torch
    n, L = 203, 16 * h0
    rng = np.random.default_rng(3)
    s = abi.Species(n)
    s.pos[:] = rng.uniform(0.0, L, (3, n))
    s.h[:] = rng.uniform(0.8, 1.2, n)
    s.mass[:] = rng.uniform(0.5, 1.5, n)
    p = abi.default_params(kernel=abi.KERNEL_CUBIC, precision=prec, h0=h0)
    box = abi.make_box((0, 0, 0), (L, L, L), (0, 1, 1))
    cols = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (*s.pos, s.mass, s.h)]
    rho = torch.empty(n, dtype=torch.float64, device="cuda")
    abi.check(abi.lib().sph_density_noalloc(C.byref(p), C.byref(box), n, *[c.data_ptr() for c in cols],
                                            rho.data_ptr(), torch.cuda.current_stream().cuda_stream))
    po = abi.SphParams.from_buffer_copy(p)
    po.precision = abi.PREC_FP64
    orc = oracle.System(po, [box], s.copy(), np.full(n, abi.ROLES_DEFAULT, dtype=np.uint8))
    orc.density(fp32_geometry=prec == abi.PREC_FP32_COMP)
    counts, pairs = orc.neighbour_counts(fp32_geometry=prec == abi.PREC_FP32_COMP)
    assert (pairs == 0) == (h0 in (1e-24, 1e-165))
    assert np.max(np.abs(rho.cpu().numpy() / orc.s.density - 1.0)) <= TOL[prec]
