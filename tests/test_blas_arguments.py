"""Which moduli the vector calls take does not depend on the calls before (no GPU:
the modulus is looked at before the vectors, which are None here)."""
import numpy as np
import pytest

import benchntt_b200 as bn


def call(q, mu):
    bn.blas(None, "vvadd", None, None, None, q, mu)


@pytest.mark.parametrize("q,mu", [(5.0, 3), (5, 3.0), ("5", 3)])
def test_not_integers_are_refused(q, mu):
    with pytest.raises(TypeError):
        call(q, mu)
    with pytest.raises(AttributeError):   # past the modulus
        call(5, 3)
    with pytest.raises(TypeError):
        call(q, mu)


@pytest.mark.parametrize("q,mu", [(bn.Q_BLAS, bn.MU_BLAS), (bn.Q_BLAS, None), (True, 1),
                                  (np.array(bn.Q_BLAS, dtype=object), np.array(bn.MU_BLAS, dtype=object))])
def test_integers_are_taken(q, mu):
    with pytest.raises(AttributeError):
        call(q, mu)
