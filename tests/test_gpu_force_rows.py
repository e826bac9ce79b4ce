"""Inter-subunit forces over lists of every length class: none, short and full pieces, several pieces, and
lists long enough for a whole warp, by both forms of the force kernel (one item per CTA, CTAs that draw
items) and of the window kernel.  Reference: FP64 numpy sums over the pairs of the kernel's own lists (the
formulas of src/forces.cpp:67-145).

Tolerance, derived: a pair's separation carries 6e-8 of relative rounding, which the steepest term (the
12th power) turns into 1e-6 of its magnitude; reciprocals, roots and exponentials of exponents up to 12
add at most 2e-6: 1e-5 of the sum of the terms' magnitudes, and 1e-7 per pair for the fixed-point
rounding (2^-24 below zero)."""
import numpy as np
import pytest

from souffle_gb300 import gpu, params, state
from test_gpu_energy_kernels import cloud, lattice_state

pytestmark = pytest.mark.gpu


def system(n, S, per_sub, e_cut, **kw):
    t = cloud(n, seed=n + 7)
    side = per_sub * int(np.ceil(S ** (1 / 3)))
    conc = S * 1000.0 / (side ** 3 * 1e-27 * params.AVOGADRO)
    o = params.CliOptions(C=conc, c=state.salt_for_debye_length(1.0), S=S, E=2.1, e=e_cut, L=0.3, B=10, t=0.0001)
    d = params.derive(o, 1e-9, 3.9434e-26, S * n)
    pos = lattice_state(t, S, d.box, 0.2, seed=S + 3 * n)
    s = gpu.GpuSystem(t, [gpu.system_params(o, d, S, 0)], inter_capacity=1500, cand_capacity=1024, **kw)
    s.set_state(pos, np.zeros_like(pos))
    return t, o, d, pos, s


def direct(t, d, elj, pos, i, j):
    n, L = t.n_beads, d.box
    r = pos[i] - pos[j]
    r -= L * np.round(r / L)
    d1 = np.sqrt((r ** 2).sum(1))
    li, lj = i % n, j % n
    q, s, ty = np.asarray(t.charge), np.asarray(t.diameter), np.asarray(t.types)
    k, shc = d.kappa, (s[li] + s[lj]) / 2
    w = q * np.exp(k * s / 2) / (1 + k * s / 2) * np.sqrt(d.lb)
    ce = np.where(d1 < d.ecut_el, w[li] * w[lj] * np.exp(-k * d1) / d1 ** 2 * (k + 1 / d1), 0.0)
    att = np.zeros(len(i), dtype=bool)
    for a, b in t.lj_attract:
        att |= (ty[li] == a) & (ty[lj] == b)
    s6 = (np.where(att, s[li], shc) / d1) ** 6  # attractive pairs take the first bead's diameter
    on = np.where(att, d1 < d.ecut, d1 < 1.12246205 * shc) & (i // n != j // n)
    eps = np.where(att, elj, 1.0)
    c = ce + np.where(on, 48 * eps * s6 * (s6 - 0.5) / d1 ** 2, 0.0)
    mag = np.abs(ce) + np.where(on, 48 * eps * s6 * (s6 + 0.5) / d1 ** 2, 0.0)
    f = np.stack([np.bincount(i, c * r[:, x], len(pos)) for x in range(3)], 1)
    m = np.stack([np.bincount(i, mag * np.abs(r[:, x]), len(pos)) for x in range(3)], 1)
    return f, m, np.bincount(i, minlength=len(pos))


@pytest.mark.parametrize("n,S,per_sub,e_cut,kw", [
    (1, 30, 3.0, 4.0, {}),
    (7, 27, 4.6, 3.0, {}),                          # a few pairs per bead
    (12, 64, 5.0, 6.0, {}),                         # rows of a whole warp
    (33, 12, 7.4, 2.5, {}), (33, 12, 7.4, 6.4, {}), (33, 12, 7.4, 6.4, {"threads_per_cta": 96, "subunits_per_cta": 5}),
    (42, 30, 7.8, 9.0, {}),                         # several rounds of a whole warp
    (42, 400, 7.8, 2.4, {}),                        # the narrow window kernel
    (20, 900, 6.6, 4.0, {"subunits_per_cta": 1}),   # more items than CTAs
])
def test_forces_over_all_row_lengths(n, S, per_sub, e_cut, kw):
    t, o, d, pos, s = system(n, S, per_sub, e_cut, **kw)
    f = s.forces(rebuild=True)
    counts, ids = s.pairlist(1600 if S < 900 else 256)
    i = np.repeat(np.arange(len(pos)), counts)
    j = ids[np.arange(ids.shape[1])[None] < counts[:, None]]
    want, mag, k = direct(t, d, 2.1, s.get_state()[0], i, j)
    assert (np.abs(f - want) <= 1e-5 * mag + 1e-7 * k[:, None]).all(), np.abs(f - want).max()
    # the same forces step by step and in one launch
    one = system(n, S, per_sub, e_cut, **kw)[-1]
    s.md_begin()
    one.md_begin()
    s.md_steps(0, 10)
    for a in range(10):
        one.md_steps(a, 1)
    for x, y in zip((*s.get_state(), s.forces(rebuild=False)), (*one.get_state(), one.forces(rebuild=False))):
        assert np.array_equal(x, y)


BIG = dict(sigma=6.0, charge=-78.0, shc=3.5)


@pytest.mark.parametrize("over,kw,big", [({}, {}, False), ({"D": "b", "d": 100.0}, {}, False),
                                         ({}, {"chain_fp64": True}, False), ({}, {}, True)])
def test_drawn_items_equal_separate_systems(over, kw, big):
    """A batch of more work items than a wave of CTAs (CTAs draw items of several systems, a second
    kernel ends the step) against each system in a handle of its own: bitwise the same."""
    from souffle_gb300 import geometry, workloads
    t = geometry.template_by_name("bilayer_n5")
    ws = [workloads.make(t, S, seed=5 + S, **over) for S in (1501, 700, 302)]
    par = [gpu.system_params(w.opt, w.derived, int(w.opt.S), w.center_local) for w in ws]
    places = workloads.place_big_beads(ws[1], 3, radius=BIG["sigma"] / 2, seed=8)
    batch = gpu.GpuSystem(t, par, **kw)
    batch.set_state(np.concatenate([w.state.pos for w in ws]), np.concatenate([w.state.vel for w in ws]))
    if big:
        batch.set_big_beads(places, system=1, **BIG)
    batch.md_begin()
    batch.md_steps(0, 13)
    pb, vb = batch.get_state()
    fb = batch.forces(rebuild=False)
    off = 0
    for k, (w, p) in enumerate(zip(ws, par)):
        one = gpu.GpuSystem(t, [p], **kw)
        one.set_state(w.state.pos, w.state.vel)
        if big and k == 1:
            one.set_big_beads(places, **BIG)
        one.md_begin()
        one.md_steps(0, 13)
        po, vo = one.get_state()
        n = len(po)
        assert np.array_equal(pb[off:off + n], po) and np.array_equal(vb[off:off + n], vo)
        assert np.array_equal(fb[off:off + n], one.forces(rebuild=False))
        assert np.array_equal(batch.md_scalars(k), one.md_scalars(0))
        off += n
