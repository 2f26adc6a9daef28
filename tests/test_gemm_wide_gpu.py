"""The 256-column tile variant of the TF32 GEMM where its blocks take several tiles each (more than 148
tiles of 128 x 256): the bits of the 64-column variant, whose sums over K run in the same order."""
import numpy as np
import pytest

import hams_b200

pytestmark = pytest.mark.gpu


# tiles 1, 148, 149, 297 (a third tile for one block) and 450, with remainders of rows, columns and K panels
@pytest.mark.parametrize("m,n,k,alpha,beta,rowmajor", [
    (1, 1, 4, 1.0, 1.0, False),
    (37 * 128, 4 * 256, 32, -1.0, 1.0, False),
    (149 * 128 - 5, 200, 36, -1.0, 1.0, False),
    (27 * 128 - 127, 11 * 256 - 255, 512, 1.0, 0.0, False),
    (25 * 128 - 1, 18 * 256 - 31, 132, 0.5, -2.0, True),
])
def test_several_tiles_per_block(m, n, k, alpha, beta, rowmajor):
    rng = np.random.default_rng(m + n + k)
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = rng.standard_normal((k, n)).astype(np.float32)
    c = rng.standard_normal((m, n)).astype(np.float32)
    want = hams_b200.diag_gemm_tf32(a, b, c, alpha, beta, rowmajor, variant=0)
    for _ in range(2):
        assert np.array_equal(hams_b200.diag_gemm_tf32(a, b, c, alpha, beta, rowmajor, variant=2), want)
