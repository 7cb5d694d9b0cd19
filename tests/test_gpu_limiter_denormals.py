"""minmod of a denormal slope and one that is not: the product's sign decides (it underflows to
zero below 2^-1074), as in the oracle."""
import numpy as np
import pytest

from hyperflow_gb300 import mechanism as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left,right", [(2.0 ** -48, 2.0 ** -1068), (2.0 ** -60, 2.0 ** -1023), (2.0 ** -4, 2.0 ** -1071),
                                        (2.0 ** -3, 2.0 ** -1071), (2.0, 2.0 ** -1073), (1.0, 2.0 ** -1022)])
def test_transverse_momentum_at_a_face(gpu, oracle, left, right):
    """Supersonic flow in x, so the flux of the transverse momentum is u times the left state's:
    u (0 + minmod(left, right) / 2)."""
    import torch
    import hyperflow_gb300 as hf
    X = np.zeros(9)
    X[8] = 1.0
    q = M.primitive(300.0, 101325.0, X=X, u=3000.0, v=0.0, ns=9)
    lv = hf.make_level(2, 1, 1e-4, 1e-4, boundary_lo=("transmissive",) * 2, boundary_hi=("transmissive",) * 2)
    a = hf.PatchArray(12, 2, 1)
    g = np.tile(q[:, None, None], (1, 5, 6))
    g[10] = np.array([-left, -left, 0.0, right, right, right])[None]
    g[10, :, 1] = -left
    a.ghosted().copy_(torch.from_numpy(g))
    fx, _ = hf.euler_stage(gpu, lv, a, a.like(), 1e-12, faces=True)
    want = 0.5 * float(oracle.minmod(left, right)[0]) * 3000.0
    got = float(fx[10, 0, 1])
    # the cell values are [-left, 0, right]: face 1 lies right of the cell that holds 0
    if want == 0.0:
        assert got == 0.0
    else:
        # relative rounding of u, and half a unit of 2^-1074 in the slope, 3000 times over
        assert abs(got - want) <= 1e-12 * want + 3000 * 2.0 ** -1074
