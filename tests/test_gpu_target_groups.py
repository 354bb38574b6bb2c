"""The neighbour build deals a cell's targets to warps in groups of 64, 32, 16, 8
or 4, by the number of particles.  One slab per group size (for either
precision; its full and part-filled chunks, odd counts per cell) against the
oracle: per-particle neighbour counts exact in the precision's geometry, density
within the parity bounds (FP64 1e-12, FP32 1e-5 relative).  nx = 120, 191 and 269
are also sizes whose cell sort scans its digit rows in a launch of their own (more
than 192 tiles); the others let the scatter add them.
"""
import numpy as np
import pytest

from spearhed_b200 import abi, setups

pytestmark = pytest.mark.gpu

TOL = {abi.PREC_FP64: 1e-12, abi.PREC_FP32_COMP: 1e-5}


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_FP32_COMP])
@pytest.mark.parametrize("nx", [31, 97, 120, 137, 191, 269])
def test_every_group_size_matches_oracle(oracle, prec, nx):
    import spearhed_b200 as sb
    w = setups.orszag_tang(nx=nx, nz=4, precision=prec, jitter=0.1, seed=nx)
    s = w.species[abi.SPECIES_DEFAULT].copy()
    orc = oracle.System(w.params, w.boxes, s, np.full(s.n, abi.ROLES_DEFAULT, dtype=np.uint8))
    counts, pairs = orc.neighbour_counts(fp32_geometry=prec == abi.PREC_FP32_COMP)
    orc.density()
    with sb.context_for(w) as ctx:
        ctx.density()
        assert np.array_equal(ctx.neighbour_counts(abi.SPECIES_DEFAULT), counts)
        assert ctx.reduce()["pairs"] == pairs
        rho = ctx.get_species(abi.SPECIES_DEFAULT).density
    assert np.max(np.abs(rho / orc.s.density - 1.0)) <= TOL[prec]


# particle counts above which a cell's targets are not split: 1.25 groups of 64 for
# each of the 148 SMs' resident warps (4 blocks of 4 warps in FP64, 6 in FP32)
FULL_GROUPS = {abi.PREC_FP64: 148 * 4 * 4 * 80, abi.PREC_FP32_COMP: 148 * 6 * 4 * 80}


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_FP32_COMP])
@pytest.mark.parametrize("cull,h_lo,levels", [(abi.CULL_GLOBAL, 1.0, 1), (abi.CULL_PAIR_MAX, 0.7, 1),
                                              (abi.CULL_PAIR_MAX, 0.25, 2)])
def test_dense_cells_in_groups_of_64_match_oracle(oracle, prec, cull, h_lo, levels):
    """A cloud of about ten particles per cell with four balls of 500, each inside
    one cull radius, at a particle count where groups hold 64 targets: the balls'
    cells run many pairs of 32-target chunks and fill several windows per chunk
    pair, so own entries are found and cleared in either chunk and in any window,
    with one and with two cell levels and under both culls."""
    import ctypes as C
    import spearhed_b200 as sb
    n = FULL_GROUPS[prec] + 1013
    rng = np.random.default_rng(17)
    s = abi.Species(n)
    s.pos[:] = rng.uniform(0.0, 1.0, (3, n))
    R = (40.0 / n * 3 / (4 * np.pi)) ** (1 / 3)
    k = 500
    for b in range(4):
        d = rng.normal(size=(3, k))
        d *= 0.4 * h_lo * R * rng.uniform(0.0, 1.0, k) ** (1 / 3) / np.linalg.norm(d, axis=0)
        s.pos[:, b * k:(b + 1) * k] = rng.uniform(0.2, 0.8, (3, 1)) + d
    s.h[:] = 0.5 * R * rng.uniform(h_lo, 1.0, n)
    s.mass[:] = rng.uniform(0.5, 1.5, n) / n
    p = abi.default_params(kernel=abi.KERNEL_CUBIC, precision=prec, cull=cull, h0=0.5 * R)
    boxes = [abi.make_box((0, 0, 0), (1, 1, 1), (0, 1, 1))]
    orc = oracle.System(p, boxes, s.copy(), np.full(n, abi.ROLES_DEFAULT, dtype=np.uint8))
    want, pairs = orc.neighbour_counts(fp32_geometry=prec == abi.PREC_FP32_COMP)
    orc.density(fp32_geometry=prec == abi.PREC_FP32_COMP)
    assert want[:4 * k].min() >= k - 1  # each ball is within every member's reach
    with sb.Context(p, boxes) as ctx:
        ctx.set_species(abi.SPECIES_DEFAULT, s)
        ctx.density()
        grid = (C.c_double * 12)()
        abi.check(abi.lib().sphx_box_grid(ctx._p, 0, grid))
        assert grid[9] == levels
        got = ctx.neighbour_counts(abi.SPECIES_DEFAULT)
        assert np.array_equal(got, want)
        assert ctx.reduce()["pairs"] == pairs
        rho = ctx.get_species(abi.SPECIES_DEFAULT).density
    assert np.max(np.abs(rho / orc.s.density - 1.0)) <= TOL[prec]
