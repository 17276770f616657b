"""Kernel variants chosen by a rule on sizes, at the sizes where the rule or
the variant can go wrong (GPU)."""
import numpy as np
import pytest

import mgcfd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed", "dw"])
@pytest.mark.parametrize("axes", [(3, 3, 3, 3, 3, 3, 4), (8, 8), (5, 8, 3, 16, 4), (9,)])
def test_batch_norms_blocks_within_and_across_meshes(precision, axes):
    """The level-0 norms of a batch, where a block of 128 nodes lies in one
    mesh (8^3 = 4 whole blocks), spans several (27 nodes each) or ends a level,
    against each mesh solved alone.  The states agree to rounding (a few
    1e-16), the residuals are their differences, 1e-7 and more of the state:
    a node's residual agrees to 1e-8 relative, and so do the norms.  A norm that
    missed or double-counted one of at most 4096 nodes is off by 1e-4 or so."""
    meshes = [mgcfd.HostMesh.generate(n, 1, 40 + k) for k, n in enumerate(axes)]
    machs = [0.3 + 0.05 * k for k in range(len(axes))]
    batch = mgcfd.Batch(meshes, machs, [2.0] * len(axes), precision=precision)
    batch.run(3)
    assert batch.synchronize() == 0
    for k, m in enumerate(meshes):
        solo = mgcfd.Solver(m, machs[k], 2.0, precision=precision)
        solo.run(3)
        st, rms, rho = solo.norms()
        bst, brms, brho = batch.mesh_status(k)
        assert (st, bst) == (0, 0)
        np.testing.assert_allclose([brms, brho], [rms, rho], rtol=1e-6, atol=0)
        solo.close()
    batch.close()
