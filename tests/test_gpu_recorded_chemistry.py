"""The chemistry of a recorded run and the reverse sweep's recomputation of it are one
integration (csrc/hf_group.cuh) at every size: gas that is uniform over a periodic level
stays uniform bit for bit in the flow, so a recorded step of a large level ends in the state
of a small one."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def cells(ns, n, seed):
    from hyperflow_gb300 import workloads as W
    U, dt = W.chem_batch(n, seed=seed, diluent="N2" if ns == 9 else "AR")
    return U, dt


@pytest.mark.parametrize("ns", [9, 10])
def test_a_large_recorded_run_ends_as_a_small_one(gpu, ns):
    import hyperflow_gb300 as hf
    ctx = gpu if ns == 9 else hf.Context("H2_Li+AR")
    big = 64 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    nx = 128
    ny = -(-big // nx)
    U, dt = cells(ns, 4, seed=17)
    for k in range(4):
        end = []
        for mx, my in ((16, 16), (nx, ny)):
            lv = hf.make_level(mx, my, 1.0, 1.0, periodic=(1, 1))
            U0 = torch.from_numpy(U[:, k]).cuda()[:, None, None].expand(-1, my, mx).contiguous()
            fa = hf.FlowAdjoint(ctx, lv, U0, 1, dts=[dt[k]])
            f = fa.final
            assert torch.equal(f, f[:, :1, :1].expand_as(f))
            end.append(f[:, 0, 0].clone())
            fa.close()
        assert not torch.equal(end[0], U0[:, 0, 0])
        assert torch.equal(end[0], end[1])


def test_the_reverse_sweep_integrates_as_the_forward_groups(gpu):
    """One call through the adjoint's kernel (its final temperature) and through the forward
    group kernel: the same bits."""
    import hyperflow_gb300 as hf
    U, _ = cells(9, 64, seed=23)
    U0 = torch.from_numpy(U).cuda()
    J = hf.ChemSensitivity(gpu, 3e-7, 1, objective="final_T").objective(U0)
    f = U0.clone()
    hf.ChemistryBatch(gpu, "plain").advance(f, 3e-7)
    assert torch.equal(J, hf.properties(gpu, f)[2])
