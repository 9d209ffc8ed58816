"""The FP64 substep's divisions by known divisors (dx, the RK4 weights, the
dust source's W, D and volume) against the restatement with correctly rounded
e^x: the same bits as IEEE division on grids whose spacing is no power of two,
for ordinary fields, for fields so small that quotients leave the range in which
the remainder is exact (the kernel then divides), and for vanishing ones."""
import numpy as np
import pytest

import oracle
from cosmograph_b200 import ics, state as S
from cosmograph_b200.evolution import BoxConfig, evolve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("amp", [2e-2, 1e-150, 1e-255, 0.0])
@pytest.mark.parametrize("matter,shape,order", [
    (S.DUST, (12, 14, 18), 8),
    (S.DUST, (24, 12, 16), 4),
    (S.SCALAR, (20, 18, 22), 6),
    (S.VACUUM, (13, 17, 19), 2),
])
def test_quotients_bit_exact(matter, shape, order, amp):
    st = ics.perturbed(shape, matter, seed=31, amp=amp)
    ref = oracle.evolve(st, 2, order, lapse="Harmonic", cr=True)
    got = evolve(st, 2, BoxConfig(order=order, lapse="Harmonic"))
    differ = [n for f, n in enumerate(st.names) if not np.array_equal(got.fields[f], ref.fields[f])]
    assert not differ, differ
