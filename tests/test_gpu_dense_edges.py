"""The dense path at sizes around its tiles of 32 rows, from one state on: all
eigenvalues against numpy's of the oracle's matrix, and the eigenvectors'
residuals and orthonormality, at the solver tests' 1e-10 |H|."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,Sz,k", [
    (4, 3, 6, (0, 0)),   # 1 state
    (4, 3, 4, (1, 0)),   # a handful
    (4, 3, 3, (1, 2)),   # 18: part of a tile
    (4, 4, 5, (0, 0)),   # 35: a tile and a little
    (4, 3, 2, (2, 1)),   # 42
    (4, 3, 1, (0, 0)),   # 66: two tiles and a little
    (4, 4, 4, (1, 3)),   # 112: four tiles
    (4, 4, 3, (2, 0)),   # 273
])
def test_dense_spectrum_at_tile_edges(cuda_device, Lx, Ly, Sz, k):
    from ed_code_gb300 import lattice as L
    from ed_code_gb300 import sector

    model = L.make_model(L.TorusSpec("triangular", Lx, Ly, Jz=0.7, Ch=0.3), Sz, *k, bowties=False)
    ref = O.OracleSector(model)
    H = ref.dense()
    scale = max(1.0, np.abs(H).sum(axis=1).max())
    want = np.linalg.eigvalsh(H)
    for stored in (False, True):
        sec = sector.GpuSector(model)
        if stored:
            assert sec.build_targets()
        eigs, vecs, _ = sec.solve_plain(n_ev=min(3, sec.n_p), want_vectors=True)
        assert len(eigs) == sec.n_p
        assert np.abs(eigs - want).max() <= 1e-10 * scale
        for e, x in zip(eigs, vecs):
            assert np.abs(sec.sHv(x) - e * x).max() <= 1e-10 * scale
        assert np.abs(vecs.conj() @ vecs.T - np.eye(len(vecs))).max() <= 1e-10
