"""The neighbour build deals a cell's targets to warps in groups of 64, 32, 16, 8
or 4, by the number of particles.  One slab per group size (for either
precision; its full and part-filled chunks, odd counts per cell) against the
oracle: per-particle neighbour counts exact in the precision's geometry, density
within the parity bounds (FP64 1e-12, FP32 1e-5 relative).  nx = 120 is also a size whose cell sort scans
its digit rows in a launch of their own; the others let the scatter add them.
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
