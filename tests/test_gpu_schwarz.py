"""The Schwarz bounds order the pair list, by whose positions the processes of
a sharded build (each with a basis of its own) divide the quartets: they have to
come out alike, bit for bit, every time a basis is made."""
import numpy as np
import pytest

import oracle as O
from chronusq_public_b200.basis import BasisSet, Molecule, parse_gbs
from chronusq_public_b200.contraction import DirectTPI

pytestmark = pytest.mark.gpu


def contracted(letter, n):
    return "%s %d 1.00\n" % (letter, n) + "".join("  %g %g\n" % (0.15 * 2.3 ** k, 0.2 + 0.1 * k)
                                                  for k in range(n))


@pytest.mark.parametrize("shells", [(("S", 14), ("P", 9)), (("D", 4), ("P", 1)),
                                    (("S", 3), ("F", 3))])
def test_bounds_are_the_same_in_every_basis(shells):
    gbs = "****\nH 0\n" + "".join(contracted(*s) for s in shells) + "****\n"
    rng = np.random.default_rng(5)
    mol = Molecule.from_angstrom([("H", *x) for x in rng.uniform(-3, 3, (10, 3))])
    bs = BasisSet.build(mol, parse_gbs(gbs))
    Q = [DirectTPI(bs).schwarz() for _ in range(8)]
    for q in Q[1:]:
        assert np.array_equal(q, Q[0])
    ref = O.OracleBasis(bs).schwarz()
    # sums of up to 1e4 primitive terms in another order
    sig = Q[0] > 0
    assert np.abs(Q[0][sig] - ref[sig]).max() < 1e-12 * ref.max()
