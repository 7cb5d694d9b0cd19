"""Cells in groups of 8 lanes (csrc/hf_group.cuh): the drop-in forms of small batches and the
batched form's costly cells, at the edges of the groups, warps and of the rule that picks
them, against the oracle at the chemistry parity bar (T relative 1e-6, Y absolute 1e-8)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def check(oracle, got, U, dt, ns):
    oracle.set_species(ns)
    try:
        ref, bad, _ = oracle.chem_batch(U.T, 0.0, dt_cell=dt)
        assert bad == -1
        got = got.cpu().numpy().T
        Tg, Tr = oracle.properties(got)[2], oracle.properties(ref)[2]
        rho = ref[:, :ns].sum(1)
        assert np.max(np.abs(Tg - Tr) / Tr) < 1e-6
        assert np.max(np.abs(got[:, :ns] - ref[:, :ns]) / rho[:, None]) < 1e-8
    finally:
        oracle.set_species(9)


@pytest.mark.parametrize("ns", [9, 10])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 33])
def test_drop_in_forms_at_group_edges(gpu, oracle, n, ns):
    import hyperflow_gb300 as hf
    from hyperflow_gb300 import workloads as W
    ctx = gpu if ns == 9 else hf.Context("H2_Li+AR")
    U, dt = W.chem_batch(n, seed=40 + n, diluent="N2" if ns == 9 else "AR")
    out = []
    for form in ("plain", "persistent"):
        f = cuda(U)
        hf.ChemistryBatch(ctx, form).advance(f, 0.0, dt_cell=cuda(dt))
        out.append(f)
    assert torch.equal(out[0], out[1])
    check(oracle, out[0], U, dt, ns)


def test_both_sides_of_the_size_rule(gpu, oracle):
    """64 cells per SM go to groups, one more to lanes: the same cells, in both."""
    import hyperflow_gb300 as hf
    from hyperflow_gb300 import workloads as W
    n = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    U, dt = W.chem_batch(48, seed=9, diluent="N2")
    for m in (n, n + 1):
        k = np.arange(m) % 48
        f = cuda(U[:, k])
        hf.ChemistryBatch(gpu, "plain").advance(f, 0.0, dt_cell=cuda(dt[k]))
        # every copy of a cell has the same result, whatever group or lane it was in
        assert torch.equal(f[:, :48], f[:, 48:96]) and torch.equal(f[:, :48], f[:, -(m % 48 or 48) - 48:][:, :48])
        check(oracle, f[:, :48], U, dt, 9)


@pytest.mark.parametrize("form", ["plain", "persistent", "batched"])
def test_a_failing_cell_leaves_the_batch_unchanged(gpu, form):
    """Cells 5 and 2 cannot be taken; the lowest index is reported, nothing is written."""
    import hyperflow_gb300 as hf
    from hyperflow_gb300 import workloads as W
    U, dt = W.chem_batch(11, seed=3, diluent="N2")
    U[3, 5] = -1e-3
    U[11, 2] = np.nan
    f = cuda(U)
    with pytest.raises(RuntimeError) as e:
        hf.ChemistryBatch(gpu, form).advance(f, 0.0, dt_cell=cuda(dt))
    assert e.value.first_failed == 2
    assert np.array_equal(f.cpu().numpy(), U, equal_nan=True)


def test_automatic_groups_of_the_batched_form(gpu, oracle):
    """By default the library picks the cells: after a first call (costs known) the
    costly ones go to groups, with the same results to the parity bar; cold calls use none."""
    import subprocess
    import sys
    import os
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = """
import sys; sys.path[:0] = [%r, %r]
import numpy as np, torch, hyperflow_gb300 as hf, oracle
from hyperflow_gb300 import workloads as W
ctx = hf.Context("H2_Li")
U, dt = W.chem_batch(700, seed=21, diluent="N2")
cb = hf.ChemistryBatch(ctx, "batched")
d = torch.from_numpy(dt).cuda()
f = torch.from_numpy(U).cuda(); cb.advance(f, 0.0, dt_cell=d)
assert ctx.counters()["chem_coop_cells"] == 0
f = torch.from_numpy(U).cuda(); cb.advance(f, 0.0, dt_cell=d)
n = ctx.counters()["chem_coop_cells"]
assert 0 < n <= 700, n
oracle.build(); oracle.set_species(9)
ref, bad, _ = oracle.chem_batch(U.T, 0.0, dt_cell=dt)
got = f.cpu().numpy().T
Tg, Tr = oracle.properties(got)[2], oracle.properties(ref)[2]
rho = ref[:, :9].sum(1)
assert bad == -1 and np.max(np.abs(Tg - Tr) / Tr) < 1e-6
assert np.max(np.abs(got[:, :9] - ref[:, :9]) / rho[:, None]) < 1e-8
""" % (root, os.path.join(root, "oracle"))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=240)
    assert r.returncode == 0, r.stderr[-2000:]
