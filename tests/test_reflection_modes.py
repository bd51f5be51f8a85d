"""What the marched operator rests on: in sums and differences along the axes the element of an isotropic cube falls apart into
eight blocks of at most 3 x 3. A finest level whose element does not is refused, so no Poisson's ratio that the solver
accepts may come near the host's bound of 1e-12."""
import numpy as np
import pytest

import psfea

CORNERS = np.array([(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)])


def blocks():
    """which of the 24 x 24 mode entries (3 a + c, a = ax + 2 ay + 4 az) belong to one block: the parity of the displacement's own
    axis turns round under its reflection, so modes couple where a xor e_c is the same"""
    parity = np.array([a ^ (1 << c) for a in range(8) for c in range(3)])
    return parity[:, None] == parity[None, :]


@pytest.mark.parametrize("nu", [-0.9999, -0.9, -0.3, 0.0, 0.2, 0.3, 0.45, 0.499, 0.49999, 0.499999])
def test_element_splits_into_the_blocks(nu):
    K, _ = psfea.element_matrix(nu)
    h = np.array([[np.prod([(2 * CORNERS[p, d] - 1) if (a >> d) & 1 else 1 for d in range(3)]) for p in range(8)] for a in range(8)], float)
    T = np.kron(h, np.eye(3))
    B = T @ K @ T.T / 64
    off = np.abs(B[~blocks()]).max() / np.abs(B).max()
    assert off < 1e-14, off
