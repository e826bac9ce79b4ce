"""The pair lists at the sizes where their kernel changes shape: bead counts around mask words, more
candidates than one chunk and one warp ballot hold, and both sides of the number of subunits (1,024)
from which candidates come from the cell grid.  Reference: a numpy restatement of update_pairlist
(src/functions.cpp:69-117) over whole subunit blocks, its stale-distance reuse included; lists are
integers and must be identical, in order."""
import numpy as np
import pytest

from souffle_gb300 import gpu, params, state
from test_gpu_energy_kernels import cloud, lattice_state

pytestmark = pytest.mark.gpu


def reference(t, S, d, cl, pos):
    n, L = t.n_beads, d.box
    nl2 = d.nlist_cutoff ** 2
    p = pos.reshape(S, n, 3)
    wrap = lambda x: x - L * np.round(x / L)  # noqa: E731
    ch = np.asarray(t.charge) != 0
    lists = [[] for _ in range(S * n)]
    c = p[:, cl]
    for i in range(S):
        near = np.nonzero((wrap(c[i] - c) ** 2).sum(-1) < 2.25 * nl2)[0]
        for j in near:
            r2 = (wrap(p[i][:, None] - p[j][None]) ** 2).sum(-1)
            seen = (ch[:, None] & ch[None] & ~np.eye(n, dtype=bool)) if i == j else np.ones((n, n), dtype=bool)
            if i == 0 or j == 0:  # entries not recomputed take the last computed distance, row-major
                stale = np.zeros((n, n), dtype=bool)
                if i == 0:
                    stale[cl, :] = True
                if j == 0:
                    stale[:, cl] = True
                fresh = (seen & ~stale).reshape(-1)
                at = np.maximum.accumulate(np.where(fresh, np.arange(n * n), -1))
                first = 0.0 if i == j else r2[cl, cl]
                r2 = np.where(at >= 0, r2.reshape(-1)[np.maximum(at, 0)], first).reshape(n, n)
            for a, b in zip(*np.nonzero(seen & (r2 < nl2))):
                lists[i * n + a].append(j * n + b)
    return lists


@pytest.mark.parametrize("n,S,per_sub,e_cut,cl", [
    (1, 9, 2.5, 3.0, 0),
    (7, 1, 14.0, 5.0, 3),                                             # one subunit: its own block only
    (31, 12, 6.5, 2.0, 30), (32, 12, 6.5, 4.0, 31), (33, 12, 6.6, 4.0, 32), (33, 12, 6.6, 4.0, 0),
    (12, 64, 4.2, 6.0, 5),                                            # dozens of candidates: several chunks and ballots
    (100, 5, 9.5, 4.0, 64), (200, 3, 12.0, 4.0, 199),                 # two rows per thread
    (3, 1024, 3.5, 3.0, 1), (3, 1025, 3.5, 3.0, 1),                   # search in the kernel, cell grid
])
def test_pair_lists_match_reference(n, S, per_sub, e_cut, cl):
    t = cloud(n, seed=n + 1)
    side = per_sub * int(np.ceil(S ** (1 / 3)))
    conc = S * 1000.0 / (side ** 3 * 1e-27 * params.AVOGADRO)
    o = params.CliOptions(C=conc, c=state.salt_for_debye_length(1.0), S=S, E=2.1, e=e_cut, L=0.3, B=10, t=0.001)
    d = params.derive(o, 1e-9, 3.9434e-26, S * n)
    pos = lattice_state(t, S, d.box, 0.3, seed=S + n)
    want = reference(t, S, d, cl, pos)
    s = gpu.GpuSystem(t, [gpu.system_params(o, d, S, cl)], inter_capacity=1500, cand_capacity=1024)
    s.set_state(pos)
    try:
        s.forces(rebuild=True)
    except gpu.SouffleError as e:  # overlapping beads: the forces are out of range, the lists are not
        assert e.code == 4
    counts, ids = s.pairlist(1500)
    for g, w in enumerate(want):
        assert list(ids[g, :counts[g]]) == w, g
