"""The Lanczos reductions (many inner products at once, sums closed on the
device) at the edges of their ranges: vectors shorter than a chunk of 1,024
elements, chunks with remainders, even and odd numbers of chunks, and numbers
of stored vectors that are no multiple of a group of eight or four.  A wrong or
missing product spoils the orthogonality, and with it T: the levels of the
mixed solver (both precisions, every reorthogonalisation) and of the plain one
against the dense path's, at the solver tests' tolerances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spec,k,steps", [
    (("triangular", 4, 3), (1, 2), 61),   # 75 states: a part of one chunk
    (("square", 4, 4), (0, 0), 113),      # 822 states
    (("triangular", 6, 3), (1, 1), 150),  # 2,700 states: three chunks
    (("triangular", 5, 4), (1, 2), 150),  # 9,250 states: ten chunks
])
def test_levels_of_every_reduction_match_dense(cuda_device, spec, k, steps):
    from ed_code_gb300 import lattice as L
    from ed_code_gb300 import sector

    sec = sector.GpuSector(L.make_model(L.TorusSpec(*spec, Jz=0.8), 0, *k, bowties=False))
    assert sec.build_targets()
    if sec.n_p <= 3000:
        e0 = sec.solve_plain()[0][0]
    else:
        e0 = sec.solve_plain(n_ev=1, iterations=steps, ncycles=2, dense_threshold=-1)[0][0]
    for fp64 in (False, True):
        for reorth in (1, 3, -1, 0):
            out = sec.solve_mixed(n_ev=1, iterations=steps, reorth_every=reorth, fp64_vectors=fp64)
            assert abs(out["eigs"][0] - e0) <= 1e-9 * abs(e0), (fp64, reorth, out["eigs"], e0)
    if sec.n_p > 200:  # the plain solver's last cycle keeps every vector orthogonal
        e = sec.solve_plain(n_ev=1, iterations=min(steps, 100), ncycles=3, dense_threshold=-1)[0][0]
        assert abs(e - e0) <= 1e-9 * abs(e0)
