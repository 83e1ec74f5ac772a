"""What the library keeps reserved between calls: at most 2 GiB of workspace per
device (include/ebem.h, ebem_release_workspace), also after a call that needed
more."""
import ctypes as C

import pytest

from conftest import cuda_available

pytestmark = pytest.mark.gpu


def test_solve_with_large_blocks():
    if not cuda_available():
        pytest.skip("no CUDA device")
    import elastodynamicebem_b200.core as core
    from elastodynamicebem_b200 import lib, mesh, problem
    prm = problem.ProblemParams(1, 1, 1, 1, 40)
    dm = core.DeviceMesh(mesh.icosphere(3))
    L = core.num_blocks(dm, prm)
    assert 8 * L * (3 * dm.N) ** 2 > 4 << 30
    core.timemarch_sa(dm, prm, 3, problem.DATUM_RADIAL_SIN)
    reserved, used = C.c_ulonglong(), C.c_ulonglong()
    lib.check(lib.load().ebem_workspace_info(0, C.byref(reserved), C.byref(used)))
    assert used.value == 0 and reserved.value <= 2 << 30
