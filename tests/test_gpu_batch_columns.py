"""Several right-hand sides of a batch in FP64: which items of the solve passes
multiply digits goes by the front and the number of columns, so that every
matrix has the bits it has alone."""
import numpy as np
import pytest

from spral_gb300 import batch, matrices as M, ssids

pytestmark = pytest.mark.gpu


# two to sixteen columns: each rule of the passes, and a second pass
@pytest.mark.parametrize("nrhs", [2, 3, 4, 5, 9, 17])
def test_gpu_batch_columns_have_the_bits_of_the_matrix_alone(nrhs):
    rng = np.random.default_rng(nrhs)
    # fronts of one to six pivot blocks that are not small items (separators of
    # up to 324 and 140 columns) among small matrices
    mats = [M.laplacian_3d(18, shift=-0.3), M.laplacian_2d(140, 140, -0.4)]
    orders = [M.nd_order_grid(18, 18, 18), M.nd_order_grid(140, 140)]
    for k in rng.integers(8, 30, 40):
        mats.append(M.laplacian_2d(int(k), int(k), -0.4))
        orders.append(M.nd_order_grid(int(k), int(k)))
    bak = batch.BatchAkeep([m[:2] for m in mats], orders)
    bf = batch.BatchFkeep(bak, [m[2] for m in mats])
    bs = [rng.standard_normal((len(p) - 1, nrhs)) for p, _, _ in mats]
    xs = bf.solve(bs)
    for i in (0, 1, 2, 20):
        p, r, v = mats[i]
        fk = ssids.Fkeep(ssids.analyse(p, r, orders[i]), v)
        assert np.array_equal(fk.solve(bs[i]), xs[i])
        # direct solves: the bound of the reference fixtures
        assert M.scaled_bwd_error(p, r, v, xs[i], bs[i]).max() <= 5e-14
        fk.free()
    bf.free()
