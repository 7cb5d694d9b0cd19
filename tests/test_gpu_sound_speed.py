"""Rounding errors of p, a and T against 80-bit or wider arithmetic: what their last
operations leave, and no more."""
import numpy as np
import pytest

from hyperflow_gb300 import mechanism as M

L = np.longdouble


def wide(q, ns):
    """p, a, T of states (n, NV) by Newton in long double from the mechanism's numbers."""
    q = q.astype(L).T
    lo, hi, W = (np.asarray(c, dtype=np.float64).astype(L) for c in (M.NASA_LOW[:ns], M.NASA_HIGH[:ns], M.MW[:ns]))
    R = L(M.GAS_CONSTANT)
    rho = q[:ns].sum(0)
    z = q[:ns] / W[:, None]
    et = (q[ns + 2] - (q[ns] ** 2 + q[ns + 1] ** 2) / (2 * rho)) / R
    T = np.full(q.shape[1], L(1200))
    for _ in range(60):
        m = np.where(T <= 1000, lo.T @ z, hi.T @ z)
        m[0] -= z.sum(0)
        cv = m[0] + T * (m[1] + T * (m[2] + T * (m[3] + T * m[4])))
        e = T * (m[0] + T * (m[1] / 2 + T * (m[2] / 3 + T * (m[3] / 4 + T * m[4] / 5)))) + m[5]
        T = T + (et - e) / cv
    zs = z.sum(0)
    p = R * T * zs
    return p, np.sqrt((cv + zs) / cv * p / rho), T


@pytest.mark.gpu
@pytest.mark.parametrize("ns", [9, 10])
def test_rounding_errors(gpu, ns):
    """One rounding has a relative rms of 2^-53 x 0.577 x 0.72 (mantissas spread evenly) =
    4.6e-17.  a: half of those of R T, p, p/rho (two), zs and the sum under the root
    (6 of them: 5.6e-17), half of T's error, its own last one: 1.0e-16 with T's 1.1e-16; 10% is
    left for the rest.  T and p/T as for the energy equation's terms: 1.5e-16."""
    import torch
    import hyperflow_gb300 as hf
    from hyperflow_gb300 import workloads as W
    assert np.finfo(L).nmant >= 63
    ctx = gpu if ns == 9 else hf.Context("H2_Li+AR")
    q = W.chem_batch(20000, seed=3, diluent="N2" if ns == 9 else "AR")[0]
    p, a, T = (x.cpu().numpy() for x in hf.properties(ctx, torch.from_numpy(q).cuda())[:3])
    pw, aw, Tw = wide(q.T, ns)
    rms = [float(np.sqrt((((x.astype(L) - y) / y) ** 2).mean())) for x, y in ((p, pw), (a, aw), (T, Tw))]
    assert rms[0] < 1.5e-16 and rms[1] < 1.1e-16 and rms[2] < 1.5e-16, rms
