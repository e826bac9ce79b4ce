"""Templates at the edge of what shared memory holds: more faces than the energy kernel can keep."""
import dataclasses

import numpy as np
import pytest

from souffle_gb300 import geometry, gpu, workloads

pytestmark = pytest.mark.gpu


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
