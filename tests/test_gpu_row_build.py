"""Stored rows built by each orbit search, at the edges of their ranges.

The passes that search the targets take 32- or 64-bit states and 4 or 8 packed
row minima by the torus (N <= 32, Ly <= 4; N <= 32; else), the general
row-rotation search for rows longer than 8 sites, and the reference's walk
elsewhere.  Each is compared with the oracle's sHv on a sector of few flipped
spins, at the tolerance of the other FP64 parity tests.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly,Sz,k,J2", [
    (4, 4, 1, (1, 3), 0.0),     # 32-bit states, 4 rows
    (8, 4, 11, (5, 2), 0.0),    # N = 32: the largest 32-bit state, rows of 8
    (4, 8, 11, (1, 6), 0.0),    # 8 rows: the largest packed word
    (6, 5, 10, (2, 3), 0.4),    # 32-bit states, more than 4 rows, two couplings
    (8, 5, -16, (7, 4), 0.0),   # N = 40: 64-bit states
    (9, 4, -14, (4, 1), 0.0),   # rows longer than 8: the general search
])
def test_stored_rows_of_every_search_match_oracle(cuda_device, Lx, Ly, Sz, k, J2):
    from ed_code_gb300 import lattice as L
    from ed_code_gb300 import sector

    model = L.make_model(L.TorusSpec("triangular", Lx, Ly, Jz=0.7, J2=J2, Ch=0.3), Sz, *k, bowties=False)
    ref = O.OracleSector(model)
    sec = sector.GpuSector(model)
    assert sec.n_p == ref.n_p
    v = O.splitmix_vector(sec.n_p, 5)
    w = ref.hv(v)
    assert sec.build_targets()
    assert sec.info["n_targets"] == sec.count_offdiag()
    assert np.abs(sec.sHv(v) - w).max() / max(1.0, np.abs(w).max()) <= 1e-13


@pytest.mark.parametrize("Lx,Ly,Sz,k", [
    (4, 3, 0, (1, 2)),   # 75 rows: a last slice of 11 rows, 8 warps a slice
    (5, 4, 0, (0, 0)),   # 290 slices: 4 warps
    (6, 4, 4, (2, 1)),   # 956 slices: 2 warps
    (6, 4, 2, (3, 0)),   # 2,556 slices: 1 warp
])
def test_row_sums_of_every_split_match_oracle(cuda_device, Lx, Ly, Sz, k):
    """A slice's slots are split among 8, 4, 2 or 1 warps by the sector's size:
    each against the oracle (FP64, and FP32 at the other tests' 2e-5), and the
    block kernel's bits against the single vector's."""
    import torch

    from ed_code_gb300 import lattice as L
    from ed_code_gb300 import sector

    model = L.make_model(L.TorusSpec("triangular", Lx, Ly, Jz=0.7, Ch=0.3), Sz, *k, bowties=False)
    ref = O.OracleSector(model)
    sec = sector.GpuSector(model)
    assert sec.build_targets()
    v = O.splitmix_vector(sec.n_p, 6)
    w = ref.hv(v)
    scale = max(1.0, np.abs(w).max())
    for dt, tol in ((np.complex128, 1e-13), (np.complex64, 2e-5)):
        one = sec.sHv(v.astype(dt), dtype=dt)
        assert np.abs(one - w).max() / scale <= tol
        V = torch.from_numpy(np.stack([v.astype(dt)] * 4, axis=1).copy()).cuda()
        W = torch.empty_like(V)
        sec.hv_block(V, W)
        torch.cuda.synchronize()
        for q in range(4):
            assert np.array_equal(W.cpu().numpy()[:, q], one), (dt, q)


@pytest.mark.parametrize("Lx,Ly,Sz,k,J2,directions", [
    (4, 3, 0, (0, 0), 0.0, False),     # 75 rows at k = 0: many stabilisers, a part of a slice
    (8, 4, 11, (0, 2), 0.0, False),    # 32-bit states, stabilisers beside general targets
    (6, 5, 10, (3, 0), 0.4, True),     # more diagonal parts than are counted
    (8, 5, -16, (4, 0), 0.0, False),   # 64-bit states
    (9, 4, -14, (0, 0), 0.0, False),   # the general row-rotation search
    (6, 4, 0, (3, 2), 0.3, True),      # 112,632 rows, queues of more than one turn
])
def test_matrix_free_of_every_search_matches_oracle(cuda_device, Lx, Ly, Sz, k, J2, directions):
    """The matrix-free H*v and the stored rows against the oracle (FP64 1e-13,
    FP32 2e-5), also with another coupling in every bond direction."""
    from ed_code_gb300 import lattice as L
    from ed_code_gb300 import sector

    model = L.make_model(L.TorusSpec("triangular", Lx, Ly, Jz=0.7, J2=J2, Ch=0.3), Sz, *k, bowties=False)
    if directions:
        for b in model.adj_list:
            d = ((b.y - b.x) % Lx, (b.y // Lx - b.x // Lx) % Ly)
            b.J *= 1.0 + 0.1 * min(d, ((-d[0]) % Lx, (-d[1]) % Ly))[0] + 0.07 * d[1] * (Ly - d[1])
    ref = O.OracleSector(model)
    sec = sector.GpuSector(model)
    v = O.splitmix_vector(sec.n_p, 8)
    w = ref.hv(v)
    scale = max(1.0, np.abs(w).max())
    for stored in (False, True):
        if stored:
            assert sec.build_targets()
        for dt, tol in ((np.complex128, 1e-13), (np.complex64, 2e-5)):
            assert np.abs(sec.sHv(v.astype(dt), dtype=dt) - w).max() / scale <= tol, (stored, dt)


@pytest.mark.parametrize("nv", [2, 4])
def test_block_hv_takes_vectors_between_16_byte_boundaries(cuda_device, nv):
    """FP32 vectors that start 8 bytes past a 16-byte boundary: the same bits as
    aligned ones (the rows' gathers are 16-byte loads), and as one vector alone
    that starts there."""
    import torch

    from ed_code_gb300 import lattice as L
    from ed_code_gb300 import sector

    sec = sector.GpuSector(L.make_model(L.TorusSpec("triangular", 5, 4, Jz=0.7, Ch=0.3), 0, 1, 2, bowties=False))
    assert sec.build_targets()
    V = torch.randn((sec.n_p, nv), dtype=torch.complex64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    W = torch.empty_like(V)
    sec.hv_block(V, W)
    flat, out = (torch.zeros(sec.n_p * nv + 1, dtype=torch.complex64, device="cuda") for _ in range(2))
    odd, wodd = flat[1:].view(sec.n_p, nv), out[1:].view(sec.n_p, nv)
    odd.copy_(V)
    assert odd.data_ptr() % 16 == 8
    sec.hv_block(odd, wodd)
    torch.cuda.synchronize()
    assert torch.equal(W, wodd)
    one, w1 = flat[1: sec.n_p + 1], out[1: sec.n_p + 1]
    one.copy_(V[:, 0])
    sec.hv(one, w1)
    torch.cuda.synchronize()
    assert torch.equal(w1, W[:, 0].contiguous())


@pytest.mark.parametrize("Lx,Ly,Sz,k", [
    (4, 4, 0, (0, 0)), (4, 4, 0, (1, 0)), (4, 4, -2, (2, 2)),  # three halves of the torus
    (6, 3, 0, (2, 0)), (3, 6, 0, (1, 3)),    # orders 2 and 3
    (6, 5, -10, (0, 0)), (6, 5, -10, (3, 1)),  # orders 2, 3 and 5
    (6, 6, -12, (0, 0)), (6, 6, -12, (3, 2)),    # seven shifts, 64-bit states
    (8, 4, -8, (4, 2)), (4, 8, 0, (0, 4)),   # 32 sites, 4 and 8 rows
])
def test_rows_counted_without_a_search_are_complete(cuda_device, Lx, Ly, Sz, k):
    """On a packed torus the rows' lengths come from the anti-aligned pairs and
    the targets with a stabiliser, whose momentum may refuse them: against the
    general search's count, and the rows against the matrix-free H*v (1e-13)."""
    from ed_code_gb300 import lattice as L
    from ed_code_gb300 import sector

    sec = sector.GpuSector(L.make_model(L.TorusSpec("triangular", Lx, Ly, Jz=0.7, Ch=0.3), Sz, *k, bowties=False))
    v = O.splitmix_vector(sec.n_p, 9)
    w, n = sec.sHv(v), sec.count_offdiag()
    assert sec.build_targets()
    assert sec.info["n_targets"] == n
    assert np.abs(sec.sHv(v) - w).max() / max(1.0, np.abs(w).max()) <= 1e-13
