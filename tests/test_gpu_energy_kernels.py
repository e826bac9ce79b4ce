"""The energy kernels at the sizes where they change shape: bead counts around the pair-of-rows and
32-partner boundaries, one to a few subunits, boxes of a few cut-offs, and both sides of the number of
subunits (16,384) from which candidates come from the cell grid.  Reference: FP64 numpy sums over
the pairs a periodic k-d tree finds within the cut-offs (the formulas of src/energies.cpp:24-93).

Tolerance: both sides are FP64 with relative rounding of a few 1e-15 per pair; the reference's
coordinates carry 1.4e-14 at |x| ~ 80, which the steepest pair term (WCA or LJ at r >= 0.9, slope
below 2e3 per unit) turns into at most 3e-11 per pair: 1e-9 per bead covers a hundred such pairs."""
import numpy as np
import pytest

from souffle_gb300 import geometry, gpu, params, state

pytestmark = pytest.mark.gpu


def cloud(n, seed):
    """n beads at least 0.9 apart with mixed charges (some zero), types and diameters; no bonds."""
    rng = np.random.default_rng(seed)
    pts = []
    while len(pts) < n:
        p = rng.uniform(-1, 1, 3) * (0.62 * n ** (1 / 3) + 0.3)
        if all(np.sum((p - q) ** 2) > 0.81 for q in pts):
            pts.append(p)
    types = rng.integers(1, 3, n)
    return geometry.Template(np.array(pts), types, rng.choice([-0.5, 0.0, 0.5, 1.0], n), rng.choice([1.0, 0.8], n),
                             np.ones(n), np.empty((0, 2), dtype=np.int64), np.empty(0, dtype=np.int64), np.empty(0),
                             np.empty((0, 3), dtype=np.int64), [(2, 2), (1, 2)])


def reference(t, S, d, elj, pos):
    from scipy.spatial import cKDTree

    n, L = t.n_beads, d.box
    tree = cKDTree((pos + L / 2) % L, boxsize=L)
    pr = tree.query_pairs(max(d.ecut, d.ecut_el) + 0.01, output_type="ndarray")
    i, j = np.minimum(pr[:, 0], pr[:, 1]), np.maximum(pr[:, 0], pr[:, 1])
    r = pos[i] - pos[j]
    r = np.sqrt(((r - L * np.round(r / L)) ** 2).sum(1))
    li, lj = i % n, j % n
    q, s, ty = np.asarray(t.charge), np.asarray(t.diameter), np.asarray(t.types)
    k = d.kappa
    shc = (s[li] + s[lj]) / 2
    ys = np.exp(k * shc) / ((1 + k * s[li] / 2) * (1 + k * s[lj] / 2))
    ce = ys * q[li] * q[lj] * d.lb * (np.exp(-k * r) / r - np.exp(-k * d.ecut_el) / d.ecut_el)
    ce[(r >= d.ecut_el)] = 0
    att = np.zeros(len(r), dtype=bool)
    for a, b in t.lj_attract:
        att |= (ty[li] == a) & (ty[lj] == b)
    s6 = shc ** 6
    q6, e6 = s6 / r ** 6, s6 / d.ecut ** 6
    ne = np.where(att, np.where(r < d.ecut, 4 * elj * q6 * (q6 - 1) - 4 * elj * e6 * (e6 - 1), 0.0),
                  np.where(r < 1.12246205 * shc, 4 * q6 * (q6 - 1) + 1, 0.0))
    ne[i // n == j // n] = 0
    N = S * n
    return np.bincount(i, ce, N), np.bincount(i, ne, N)


def lattice_state(t, S, box, gap, seed):
    """Subunits on a jittered lattice with random orientations, neighbours about `gap` apart."""
    rng = np.random.default_rng(seed)
    local = t.pos - t.pos.mean(axis=0)
    side = int(np.ceil(S ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:S]
    c = (g + 0.5) * (box / side) - box / 2 + rng.uniform(-gap, gap, (S, 3))
    pos = (np.einsum("sij,bj->sbi", state._random_rotations(rng, S), local) + c[:, None]).reshape(-1, 3)
    pos -= box * np.floor(pos / box + 0.5)
    return np.where(pos >= box / 2, pos - box, pos)


@pytest.mark.parametrize("n,S,per_sub,e_cut", [
    (1, 5, 3.0, 5.0),      # single beads: no pairs inside a subunit
    (2, 3, 4.0, 5.0),      # two rows, one pair
    (7, 1, 14.0, 5.0),     # odd rows, one subunit
    (31, 9, 6.5, 2.0), (32, 9, 6.5, 5.0), (33, 9, 6.6, 5.0),   # around one mask word
    (42, 130, 7.0, 12.0),  # more candidates than one pass of 128, a cut-off of most of the box
    (65, 5, 8.5, 5.0), (200, 4, 12.0, 5.0),                    # several words, one subunit per CTA
])
def test_pair_energies_match_direct_sum(n, S, per_sub, e_cut):
    t = cloud(n, seed=n)
    check(t, S, per_sub, e_cut)


@pytest.mark.parametrize("S", [16384, 16385])
def test_candidate_scan_and_cell_grid_agree_with_direct_sum(S):
    check(cloud(3, seed=3), S, 4.0, 5.0)


def check(t, S, per_sub, e_cut):
    n = t.n_beads
    box_want = per_sub * int(np.ceil(S ** (1 / 3)))
    conc = S * 1000.0 / (box_want ** 3 * 1e-27 * params.AVOGADRO)
    o = params.CliOptions(C=conc, c=state.salt_for_debye_length(1.0), S=S, E=2.1, e=e_cut, L=0.3, B=10, t=0.001)
    d = params.derive(o, 1e-9, 3.9434e-26, S * n)
    pos = lattice_state(t, S, d.box, 0.2, seed=S)
    s = gpu.GpuSystem(t, [gpu.system_params(o, d, S, 0)])
    s.set_state(pos)
    tot, pb = s.energies(per_bead=True)
    ce, ne = reference(t, S, d, o.E, pos)
    for name, want in (("ce", ce), ("ne", ne)):
        got = pb[name]
        close = np.abs(got - want) <= 1e-9 * np.maximum(1.0, np.abs(want))
        assert close.all(), (name, int((~close).sum()), got[~close][:3], want[~close][:3])
    assert tot["electrostatic"] == pytest.approx(pb["ce"].sum(), rel=1e-12, abs=1e-9)
    assert tot["lj"] == pytest.approx(pb["ne"].sum(), rel=1e-12, abs=1e-9)
    again, pb2 = s.energies(per_bead=True)  # the same bits on every call
    assert again == tot and all(np.array_equal(pb[k], pb2[k]) for k in pb)
