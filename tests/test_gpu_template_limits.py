"""Templates and CTA shapes at the edge of what shared memory holds: edges by the thousand, more faces than
the energy kernel can keep, and items of as many subunits as are accepted."""
import dataclasses

import numpy as np
import pytest

from conftest import rms_rel
from souffle_gb300 import geometry, gpu, params, state, workloads

pytestmark = pytest.mark.gpu


def force_bytes(t, nbend, subs, threads):
    """What a CTA shape is accepted by: tile, 72 bytes per bead, reductions, the template's tables."""
    n, ne, nf = t.n_beads, len(t.edges), len(t.faces)
    deg = np.bincount(t.edges.reshape(-1), minlength=n).max() + 1
    up = lambda k, m=4: (k + m - 1) // m * m
    return (max(16 * subs * (ne + 4 * nbend), 2048) + 32 * subs * n + threads + 36 * up(subs * n) + 4 * up(subs * n + 1) +
            4 * (n + up(ne + 3 * n + nbend)) + 4 * up(ne + 3 * nf + 6 * nbend + n * (deg + 1 + 2)))


def mesh(n, ne, seed):
    """n uncharged beads of one kind on a 2-sigma lattice, ne springs between random pairs of them."""
    rng = np.random.default_rng(seed)
    pos = 2.0 * np.stack(np.meshgrid(*[np.arange(7)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n].astype(float)
    e = np.stack([np.arange(ne) % n, (np.arange(ne) % n + 1 + rng.integers(0, n - 1, ne)) % n], 1)
    return geometry.Template(pos, np.ones(n, dtype=int), np.zeros(n), np.ones(n), np.ones(n), e, np.zeros(ne, dtype=int),
                             np.linalg.norm(pos[e[:, 0]] - pos[e[:, 1]], axis=1) * 1.01, np.empty((0, 3), dtype=int), [])


def test_a_template_just_below_the_limit():
    n = 256
    ne = max(k for k in range(2000, 9000, 16) if force_bytes(mesh(n, k, 3), 0, 1, 256) <= 200 * 1024)
    t = mesh(n, ne, 3)
    opt = params.CliOptions(C=1.0, c=state.salt_for_debye_length(1.0), S=2, E=2.0, e=2.5, L=0.3, B=10, t=1e-4)
    d = params.derive(opt, 1e-9, 3.9434e-26, 2 * n)
    c = t.pos.mean(axis=0)
    pos = np.concatenate([t.pos - c - 15, t.pos - c + 15])
    s = gpu.GpuSystem(t, [gpu.system_params(opt, d, 2, 0)])
    s.set_state(pos, np.zeros_like(pos))
    _, sf, _ = s.forces(rebuild=True, parts=True)
    e, l0 = t.edges, t.edge_len0
    r = t.pos[e[:, 0]] - t.pos[e[:, 1]]
    l = np.linalg.norm(r, axis=1)
    f = r * ((l0 - l) * opt.s / l)[:, None]
    want = np.zeros((n, 3))
    np.add.at(want, e[:, 0], f)
    np.add.at(want, e[:, 1], -f)
    # FP32 separations (6e-8) against length changes of 1 %: 1e-5 per edge, 50 edges of either sign per bead
    assert rms_rel(sf, np.concatenate([want, want])) < 1e-4
    tot = s.energies()
    assert tot["stretching"] == pytest.approx(2 * 0.5 * opt.s * ((l0 - l) ** 2).sum(), rel=1e-9)


def test_more_faces_than_shared_memory_holds():
    """Faces behind those of the bending edges change nothing: bitwise the energies and forces without them."""
    w = workloads.make(geometry.bilayer_n5(), 4, seed=3)
    t = w.template
    rng = np.random.default_rng(1)
    # triangles that share no edge with the template: triples of mutually unbonded beads
    bonded = {tuple(sorted(e)) for e in t.edges.tolist()}
    free = [(a, b, c) for a in range(t.n_beads) for b in range(a) for c in range(b)
            if not {(b, a), (c, a), (c, b)} & bonded]
    extra = np.array(free)[rng.integers(0, len(free), 9000)]
    many = dataclasses.replace(t, faces=np.concatenate([np.asarray(t.faces), extra]))
    out = []
    for tpl in (t, many):
        s = gpu.GpuSystem(tpl, [gpu.system_params(w.opt, w.derived, 4, w.center_local)], subunits_per_cta=1)
        s.set_state(w.state.pos, w.state.vel)
        tot, per = s.energies(per_bead=True)
        out.append([s.forces(), *[per[k] for k in sorted(per)], np.array(list(tot.values()))])
    assert abs(out[0][1]).max() > 0  # (bending)
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n,subs", [(168, 16), (10, 16)])
def test_items_of_as_many_subunits_as_are_accepted(n, subs):
    t = mesh(n, 1, 5)
    assert force_bytes(t, 0, subs, 256) <= 200 * 1024
    S = 2 * subs
    opt = params.CliOptions(C=20.0, c=state.salt_for_debye_length(1.0), S=S, E=2.0, e=2.5, L=0.3, B=10, t=1e-3)
    d = params.derive(opt, 1e-9, 3.9434e-26, S * n)
    st = state.random_state(t, S, d.box, temperature=1.0, seed=4)
    out = []
    for kw in ({}, {"subunits_per_cta": subs}):
        p = gpu.system_params(opt, d, S, 0)
        s = gpu.GpuSystem(t, [p, p], **kw)  # (a batch: its items are as long as asked for)
        s.set_state(np.concatenate([st.pos, st.pos]), np.concatenate([st.vel, st.vel]))
        f = s.forces()
        s.md_begin()
        s.md_steps(0, 10)
        out.append([f, *s.get_state()])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
