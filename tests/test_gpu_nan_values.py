"""A NaN partial density is not a negative one: the status flags of a step say so whatever the
sign bit that the NaN carries."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
ST_STAGE_BAD, ST_NEGATIVE, ST_FACE_BAD = 1, 2, 8


@pytest.mark.parametrize("flux", ["plain", "fused"])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_flags_of_a_step_with_a_nan_cell(gpu, flux, sign):
    """Gas at rest, 1% of a CFL step, one cell's N2 density a NaN: no density of the step is
    negative.  The state stays as it was."""
    import hyperflow_gb300 as hf
    from hyperflow_gb300 import mechanism as M
    X = np.zeros(9)
    X[0], X[1], X[8] = 0.2, 0.1, 0.7
    nx, ny = 24, 12
    U = np.tile(M.primitive(300.0, 101325.0, X=X, ns=9)[:, None, None], (1, ny, nx))
    U[8, 5, 11] = np.copysign(np.nan, sign)
    lv = hf.make_level(nx, ny, 1e-4, 1e-4, periodic=(1, 1))
    s = hf.Stepper(gpu, lv, torch.from_numpy(U).cuda(), chemistry=False, flux=flux)
    with pytest.raises(hf.DomainError):
        s.step(cfl=0.01)
    flags = s.graph_info()["last_flags"]
    assert flags & ST_FACE_BAD and flags & ST_STAGE_BAD and not flags & ST_NEGATIVE
    assert np.array_equal(s.state().cpu().numpy(), U, equal_nan=True)
    s.close()
