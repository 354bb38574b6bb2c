"""The FP32 pair passes of small systems (up to 37,888 particles for the density,
18,944 and 9,472 for the hydro and SPMHD forces) give every target eight lanes, in
kernels of their own for each kernel function and physics variant.
The sums are folded in row order, so the same box must get the same bits alone
(eight lanes) and inside an ensemble above the limits (one lane).
"""
import numpy as np
import pytest

from spearhed_b200 import abi, setups

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "u", "density", "h", "B", "psi", "dvdt", "dudt", "dBdt", "dpsidt", "divB")


def _run(w, steps=3):
    import spearhed_b200 as sb
    with sb.context_for(w) as ctx:
        ctx.step(steps)
        return ctx.get_species(abi.SPECIES_DEFAULT)


# switched off in the ensemble's full SPMHD: each compiled physics variant of the force pass
MHD_EXTRAS = abi.PHYS_DEDNER | abi.PHYS_TENSILE
OFF = {"mhd": 0, "mhd_ideal": MHD_EXTRAS | abi.PHYS_AV, "mhd_av": MHD_EXTRAS,
       "hydro_av": MHD_EXTRAS | abi.PHYS_MHD, "hydro": MHD_EXTRAS | abi.PHYS_MHD | abi.PHYS_AV}


@pytest.mark.parametrize("kernel", [abi.KERNEL_CUBIC, abi.KERNEL_WENDLAND_C2, abi.KERNEL_QUINTIC])
@pytest.mark.parametrize("physics", list(OFF))
def test_a_small_box_gets_the_bits_of_the_large_ensemble(physics, kernel):
    kw = dict(nbox=8, n_lo=4096, n_hi=16384)
    every = setups.brio_wu_ensemble(**kw)
    n = np.bincount(every.species[abi.SPECIES_DEFAULT].box_id)
    assert n.sum() > 37888 and n.min() <= 9472
    every.params.physics &= ~OFF[physics]
    every.params.kernel = kernel
    whole = _run(every)
    of_box = every.species[abi.SPECIES_DEFAULT].box_id
    for b in (int(np.argmin(n)), int(np.argsort(n)[len(n) // 2])):
        alone = setups.brio_wu_ensemble(**kw, boxes=[b])
        alone.params.physics, alone.params.kernel = every.params.physics, kernel
        got = _run(alone)
        for f in FIELDS:
            assert np.array_equal(getattr(got, f), getattr(whole, f)[..., of_box == b]), (b, f)
