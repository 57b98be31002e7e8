"""gbmd_pair_forces_static at the sizes where its work is cut differently: less than a warp of other
atoms, one atom a warp up to 2,432 (608 blocks of four), two above; against the oracle (1e-12)."""
import numpy as np
import pytest

import oracle
from helpers import LJ_AR, rel_norm_err
from lpmd2_gb300 import inputs as I

pytestmark = pytest.mark.gpu

gbmd = pytest.importorskip("lpmd2_gb300.gbmd")
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 2, 5, 31, 33, 108, 2432, 2433])
def test_static_forces_by_size(n):
    k = 3
    while 4 * k**3 < n:
        k += 1
    pos, L = I.fcc_fast(k, k, k, 5.7)
    pos = I.jitter(pos, 0.3, seed=n)[:n]
    pos[n // 2:] += np.array([1.0, 0.0, -1.0]) * L  # another image: one wrap brings it back
    pos_d = torch.from_numpy(np.ascontiguousarray(pos)).cuda()
    force = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
    out = torch.full((11,), float("nan"), dtype=torch.float64, device="cuda")
    gbmd.pair_forces_static(gbmd.Plugin("lennardjones", LJ_AR), pos_d.data_ptr(), n, L, force.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    f, o = force.cpu().numpy(), out.cpu().numpy()
    if n == 1:
        assert not f.any() and not o.any()
        return
    mass = np.full(n, 0.00964853)  # force factor / mass = 1: accelerations are forces
    ref = oracle.PortSim(pos, L, np.full(n, 18), mass, np.zeros_like(pos))
    ref.set_cell_manager("minimumimage", "cutoff 8.5")
    ref.add_potential("lennardjones", LJ_AR)
    ref.update_forces()
    assert rel_norm_err(f, ref.atoms()[2]) <= 1e-12
    assert abs(o[0] - ref.energy()) <= 1e-12 * abs(ref.energy())
    assert abs(o[1] - ref.virial()) <= 1e-12 * np.abs(o[2:]).max()
    assert np.abs(o[2:] - ref.stress().ravel()).max() <= 1e-12 * np.abs(o[2:]).max()
