"""The EOS solve, the admissibility test and the limiter at the edges of their fast paths:
temperatures around the bracket's ends and T_mid, densities over 36 decades, states that
must be refused, and slopes whose product underflows."""
import numpy as np
import pytest

import helpers as H
from hyperflow_gb300 import mechanism as M


def edge_states(ns=9):
    """(n, NV): every temperature of the solve's edges at several densities and speeds."""
    rng = np.random.default_rng(7)
    out = []
    for T in (180.0, 249.9, 250.1, 298.0, 999.9, 999.97, 1000.0, 1000.01, 1000.03, 1500.0, 4999.0, 5001.0, 6500.0):
        for scale in (1e-30, 1e-13, 1e-11, 1.0, 1e6):
            for speed in (0.0, 5000.0):
                X = rng.uniform(0.0, 1.0, ns)
                X[rng.uniform(size=ns) < 0.3] = 0.0
                X[1] += 0.1
                th = rng.uniform(0.0, 2 * np.pi)
                q = M.primitive(T, 101325.0, X=X / X.sum(), u=speed * np.cos(th), v=speed * np.sin(th), ns=ns)
                out.append(q * scale)
    return np.array(out)


def refused_states():
    q = H.random_states(14, seed=11)
    q[0, 3] = -1e-30
    q[1, 4] = -5e-324
    q[2, 0] = np.nan
    q[3, 5] = np.inf
    q[4, 9] = np.inf
    q[5, 10] = np.nan
    q[6, 11] = -np.inf
    q[7, :9] = 0.0
    q[8, 11] = -1e12
    q[9, 11] = 0.0
    q[10, 9] = 1e300      # kinetic energy overflows
    q[11, 3] = -0.0       # not negative: admissible
    q[12, 2] = 5e-324     # a denormal partial density: admissible
    return q


def test_heat_capacities_let_newton_contract():
    """cv_k > 0, not decreasing away from where it is small, and within a factor of two of
    its value at T_mid on [250, 5000] K: from T_mid, Newton's steps on a monotone e(T)
    contract (|1 - mean cv / cv(T)| < 1), which is what the FP32 admissibility test assumes."""
    for k in range(10):
        for a, T in ((M.NASA_LOW[k], np.linspace(250.0, 1000.0, 1501)), (M.NASA_HIGH[k], np.linspace(1000.0, 5000.0, 4001))):
            cv = a[0] - 1 + T * (a[1] + T * (a[2] + T * (a[3] + T * a[4])))
            at = cv[-1] if T[-1] == 1000.0 else cv[0]
            assert cv.min() > 0.0 and cv.max() < 2.0 * at and cv.min() > 0.5 * at


@pytest.mark.gpu
def test_properties_at_the_edges(gpu, oracle):
    import torch
    import hyperflow_gb300 as hf
    q = np.vstack([edge_states(), refused_states()])
    p, a, T, st = hf.properties(gpu, torch.from_numpy(q.T.copy()).cuda())
    po, ao, To, sto = oracle.properties(q)
    assert np.array_equal(st.cpu().numpy(), sto)
    ok = sto == 0
    # 5000 m/s at 180 K: the internal energy is 1/100 of the total, so rounding of the energy
    # equation (2^-53 of its terms) stays below 1e-13 of T
    p, a, T = (x.cpu().numpy() for x in (p, a, T))
    # cv jumps at T_mid (the two NASA ranges meet in e, not in cv): a state whose T is T_mid to
    # rounding has the sound speed of one range or of the other
    at_mid = ok & (np.abs(To - 1000.0) < 1e-9)
    assert at_mid.sum() >= 5
    for g, o in ((p[ok], po[ok]), (T[ok], To[ok]), (a[ok & ~at_mid], ao[ok & ~at_mid])):
        assert H.rel_err(g, o) < 1e-12
    for k in np.where(at_mid)[0]:
        z = q[k, :9] / M.MW[:9]
        sides = []
        for c in (M.NASA_LOW[:9], M.NASA_HIGH[:9]):
            cp = float((z * (c[:, 0] + 1e3 * (c[:, 1] + 1e3 * (c[:, 2] + 1e3 * (c[:, 3] + 1e3 * c[:, 4]))))).sum())
            sides.append(np.sqrt(cp / (cp - z.sum()) * po[k] / q[k, :9].sum()))
        assert min(abs(a[k] / s - 1.0) for s in sides) < 1e-12


@pytest.mark.gpu
def test_validate_agrees_with_properties(gpu, oracle):
    """Every state by itself on a one-cell level: the FP32 test must answer as the EOS does."""
    import torch
    import hyperflow_gb300 as hf
    q = np.vstack([edge_states(), refused_states()])
    sto = oracle.properties(q)[3]
    lv = hf.make_level(1, 1, 1e-4, 1e-4)
    pa = hf.PatchArray(12, 1, 1)
    for k in range(len(q)):
        pa.interior().copy_(torch.from_numpy(q[k].reshape(12, 1, 1)))
        try:
            hf.validate(gpu, lv, pa)
            bad = 0
        except hf.DomainError:
            bad = 1
        assert bad == sto[k], (k, q[k])


@pytest.mark.gpu
@pytest.mark.parametrize("tiny", [1e-150, 3e-163, 1e-300, 3e-310])
def test_limiter_where_slopes_underflow(gpu, oracle, tiny):
    """Face fluxes of species whose slopes have a product around 2^-1074: the limiter's sign
    test is the product's, so below it the slope is dropped."""
    import torch
    import hyperflow_gb300 as hf
    nx, ny = 37, 5
    U = H.smooth_field(nx, ny, seed=3)
    rng = np.random.default_rng(5)
    U[:, :, 6] = tiny * rng.uniform(0.5, 1.5, (ny, nx))
    U[:, :, 7] = tiny * (1.0 + np.arange(nx))[None]
    g = oracle.make_grid(nx, ny, 1e-3, 1e-3, periodic=(1, 1), bc_lo=(1, 1), bc_hi=(1, 1), inlet=U[0, 0])
    Ug = oracle.ghosted(U)
    Ug = oracle.fill_ghosts(g, Ug)
    _, fx, fy, st = oracle.euler_stage(g, Ug, 1e-8)
    lv = hf.make_level(nx, ny, 1e-3, 1e-3, periodic=(1, 1))
    a = H.to_patch(gpu, Ug)
    gx, gy = hf.euler_stage(gpu, lv, a, a.like(), 1e-8, faces=True)
    for got, ref in ((gx, fx), (gy, fy)):
        got, ref = got.cpu().numpy()[6:8], ref.transpose(2, 0, 1)[6:8]
        # a few ulp of the flux plus, for denormals, a few units of 2^-1074 per product
        assert np.all(np.abs(got - ref) <= 1e-12 * np.abs(ref).max(axis=(1, 2), keepdims=True) + 1e4 * 5e-324)


@pytest.mark.gpu
def test_trace_species_around_the_cut(gpu, oracle):
    """Partial densities around 2^-110 of the largest, where the solve leaves a species out, in
    lanes next to lanes that hold it: p, a, T as the oracle's (a left-out term is below 2^-98
    of the sums), the same whether a state sits among others like it or not."""
    import torch
    import hyperflow_gb300 as hf
    rng = np.random.default_rng(13)
    q = H.random_states(512, seed=17, speed=300.0, radicals=False)
    top = q[:, :9].max(1)
    for n, k in enumerate((3, 4, 5, 6, 7)):
        e = rng.integers(-130, -90, 512).astype(float)
        q[:, k] = np.where(rng.uniform(size=512) < 0.2, 0.0, np.where(rng.uniform(size=512) < 0.1, 1e-3, 2.0 ** e)) * top
    p, a, T, st = hf.properties(gpu, torch.from_numpy(q.T.copy()).cuda())
    po, ao, To, sto = oracle.properties(q)
    assert np.array_equal(st.cpu().numpy(), sto) and (sto == 0).all()
    for g, o in ((p, po), (a, ao), (T, To)):
        assert H.rel_err(g.cpu().numpy(), o) < 1e-12
    order = rng.permutation(512)
    again = hf.properties(gpu, torch.from_numpy(q[order].T.copy()).cuda())
    for x, y in zip((p, a, T), again):
        assert torch.equal(x[torch.from_numpy(order).cuda()], y)
