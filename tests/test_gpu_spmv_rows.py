"""The FP64 panel product on both sides of the line (8,500 nodes) where its loops
change, against the exported matrix."""
import numpy as np
import pytest

import poromec_gb300 as pg
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu


# 7,969 and 12,405 nodes, 4,705 and 8,941, 8,421 and 9,021
@pytest.mark.parametrize("kind,n", [("cube", 12), ("cube", 14), ("tetra", 8), ("tetra", 10),
                                    ("column", 280), ("column", 300)])
def test_product_on_both_sides(kind, n):
    """A row has at most some 700 entries, each product and sum rounded at 2^-53: 1e-13
    of sum |a| |x|."""
    import scipy.sparse as sp
    pb = (meshgen.column_problem(nz=n, lz=n / 4.0) if kind == "column" else
          meshgen.tetra_problem(n=n) if kind == "tetra" else meshgen.cube_problem(n=n))
    m = pg.from_problem(pb)
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    x = np.random.default_rng(n).standard_normal(m.neq)
    ia, ja, ad, al = m.get_csrd()
    L = sp.csr_matrix((al, ja - 1, ia - 1), shape=(m.neq, m.neq))
    y = ad * x + L @ x + L.T @ x
    mag = np.abs(ad * x) + abs(L) @ np.abs(x) + abs(L).T @ np.abs(x)
    assert np.all(np.abs(m.matvec(x) - y) <= 1e-13 * mag)
