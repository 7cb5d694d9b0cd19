"""The kernels with one cell per lane of the plain and the persistent form, which take batches
of more than 64 cells per SM: bit-identical to each other, at the chemistry parity bar against
the oracle, all-or-nothing when a cell fails."""
import numpy as np
import pytest
import torch

from test_gpu_group import check, cuda

pytestmark = pytest.mark.gpu
DISTINCT = 48


def batch(ns, n, seed):
    from hyperflow_gb300 import workloads as W
    U, dt = W.chem_batch(DISTINCT, seed=seed, diluent="N2" if ns == 9 else "AR")
    k = np.arange(n) % DISTINCT
    return U, dt, U[:, k], dt[k]


def sizes():
    n = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    return n + 1, 2 * n + 63


@pytest.mark.parametrize("ns", [9, 10])
@pytest.mark.parametrize("which", [0, 1])
def test_plain_and_persistent_agree(gpu, oracle, ns, which):
    import hyperflow_gb300 as hf
    ctx = gpu if ns == 9 else hf.Context("H2_Li+AR")
    n = sizes()[which]
    U, dt, Ub, dtb = batch(ns, n, seed=60 + which)
    out = []
    for form in ("plain", "persistent"):
        f = cuda(Ub)
        hf.ChemistryBatch(ctx, form).advance(f, 0.0, dt_cell=cuda(dtb))
        out.append(f)
    assert torch.equal(out[0], out[1])
    last = n - n % DISTINCT
    assert torch.equal(out[0][:, :n - last], out[0][:, last:])  # a cell's result does not depend on its place
    check(oracle, out[0][:, :DISTINCT], U, dt, ns)


@pytest.mark.parametrize("ns", [9, 10])
@pytest.mark.parametrize("form", ["plain", "persistent"])
def test_a_failing_cell_leaves_a_large_batch_unchanged(gpu, form, ns):
    import hyperflow_gb300 as hf
    ctx = gpu if ns == 9 else hf.Context("H2_Li+AR")
    n = sizes()[0]
    _, _, Ub, dtb = batch(ns, n, seed=62)
    Ub, dtb = Ub.copy(), np.full(n, 1e-9)
    Ub[3, n - 1] = -1e-3
    Ub[ns + 2, 4097] = np.nan
    f = cuda(Ub)
    with pytest.raises(RuntimeError) as e:
        hf.ChemistryBatch(ctx, form).advance(f, 0.0, dt_cell=cuda(dtb))
    assert e.value.first_failed == 4097
    assert np.array_equal(f.cpu().numpy(), Ub, equal_nan=True)
