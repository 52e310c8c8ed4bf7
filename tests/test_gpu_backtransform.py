"""
The own eigensolver at the edges of its tiles.  Tridiagonalisation: the first and last columns, where none, one or two
updates are pending, rows of up to 16 warps x 4 and blocks of 256 columns.  Back-transformation: blocks of 16 reflectors
(N - 2 of them), chunks of 64 rows, column tiles of 16 and, from N = 1,311 to 1,900, of 24.  FP32 eigenpairs: residual and
orthogonality within 5e-5 of the norm, as the solver's other tests hold it to.
"""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,batch", [(4, 2), (5, 1), (6, 3), (7, 1), (17, 3), (18, 1), (19, 2), (65, 2), (66, 1), (81, 2), (82, 2), (145, 1), (257, 30), (258, 2), (514, 1), (1310, 1),
                                     (1311, 2), (1321, 1), (1900, 1), (1901, 1)])
def test_eigenpairs(N, batch):
    from fasterlmm_gb300 import _lib, build, fast
    build()
    g = torch.Generator(device="cuda").manual_seed(N)
    Z = torch.randn(batch, N, N + 40, generator=g, device="cuda", dtype=torch.float64)
    K = Z @ Z.transpose(1, 2) / (N + 40)
    U, ev = fast._eigh_batched_f32(_lib.context(0), K)
    U, ev = U.double(), ev.double()
    norm = torch.linalg.matrix_norm(K, 2)
    R = K @ U.transpose(1, 2) - U.transpose(1, 2) * ev[:, None, :]
    assert (R.abs().amax((1, 2)) <= 5e-5 * norm).all()
    O = U @ U.transpose(1, 2) - torch.eye(N, device="cuda", dtype=torch.float64)
    assert O.abs().max() <= 5e-5
