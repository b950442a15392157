"""Precision that the decompositions hold: bounds from the rounding of the stored results, against NumPy in FP64."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24  # unit roundoff of FP32


def _ttr():
    import tensor_train_ring_decompositions_hpc_gpu_b200 as ttr
    return ttr


def _dev(x, dev, dtype=np.float32):
    import torch
    return torch.from_numpy(np.asfortranarray(x, dtype=dtype)).to(dev)


@pytest.mark.parametrize("shape,ranks", [
    ((24, 24, 24, 24), (1, 24, 24, 24, 1)),   # 576 rows, 32 columns: one CholeskyQR launch
    ((256, 64, 48), (1, 16, 20, 1)),          # 24 columns of 256 and of 1024 rows
    ((110, 100, 20, 60), (1, 62, 66, 30, 1)),  # 6200 rows, 74 columns: more than one launch holds
    ((600, 96, 20), (1, 88, 18, 1)),          # 96 columns of 600 rows: rows multiplied by an inverse
])
@pytest.mark.parametrize("power", [0, 1])
def test_fp32_bases_are_orthonormal(gpu, shape, ranks, power):
    """Plain FP32 and fixed ranks.  A basis of m rows whose entries carry independent roundings (its own, those of
    Q and of E: 3 u at most together) has U^T U = I to 2 x 3 u |u_i o u_j| ~ 6 u sqrt(3 / m); 2x that is allowed.  A
    column of Q that is off in length by half an ulp in every row is off by u whatever m is."""
    x = oracle.make_tt_tensor(list(shape), list(ranks), 1e-4, seed=sum(shape))
    res = _ttr().tt_svd(_dev(x, gpu), list(ranks), gemm="fp32", oversample=8, power_iters=power)
    for k, c in enumerate(res.cores[:-1]):
        u = c.double().cpu().numpy().reshape(-1, c.shape[2], order="F")
        if u.shape[0] > 4 * u.shape[1] and u.shape[0] > 130:  # sketched steps
            defect = np.abs(u.T @ u - np.eye(u.shape[1])).max()
            assert defect <= 12 * U32 * np.sqrt(3.0 / u.shape[0]), (k, u.shape, defect)
