"""Windows of steps in one launch (every work item resident at once) against the same steps taken one
launch pair at a time: bitwise the same state, forces and scalars, for window lengths around the
rebuild period, CTA shapes, batches, and both integrators."""
import numpy as np
import pytest

from souffle_gb300 import geometry, gpu, workloads

pytestmark = pytest.mark.gpu


def handle(ws, **kw):
    s = gpu.GpuSystem(ws[0].template, [gpu.system_params(w.opt, w.derived, int(w.opt.S), w.center_local) for w in ws], **kw)
    s.set_state(np.concatenate([w.state.pos for w in ws]), np.concatenate([w.state.vel for w in ws]))
    s.md_begin()
    return s


def result(s, n_sys):
    p, v = s.get_state()
    f = s.forces(rebuild=False)
    return [p, v, f] + [np.array(s.md_scalars(k)) for k in range(n_sys)]


@pytest.mark.parametrize("template,subs,over,kw", [
    ("patch_n3", [1], {}, {}),
    ("patch_n3", [20], {}, {}),
    ("bilayer_n5", [3], {}, {"subunits_per_cta": 2, "threads_per_cta": 96}),   # an item of one, a partial warp half
    ("bilayer_n5", [64], {}, {}),
    ("bilayer_n5", [64], {}, {"subunits_per_cta": 8, "threads_per_cta": 256}),  # more beads than threads
    ("bilayer_n5", [400], {"D": "b", "d": 100.0}, {}), ("bilayer_n5", [600], {}, {}),   # 512, 320, 256 threads
    ("bilayer_n5", [800], {}, {}), ("bilayer_n5", [1700], {}, {}),              # dealt subunits: items of one and two, two and three
    ("bilayer_n5", [5, 17, 2], {}, {}),                                         # systems of a batch, one grid barrier
    ("bilayer_n5", [33], {"D": "b", "d": 100.0}, {}),
    ("bilayer_n5", [9, 30], {"D": "b", "d": 100.0}, {}),
    ("bilayer_n5", [40], {"q": 1}, {}), ("bilayer_n5", [40], {"q": 3}, {}),     # chain lengths
])
def test_windows_equal_single_steps(template, subs, over, kw):
    t = geometry.template_by_name(template)
    ws = [workloads.make(t, S, seed=70 + S, **over) for S in subs]
    one, win = handle(ws, **kw), handle(ws, **kw)
    a = 0
    for n in (10, 20, 3, 17, 10):  # whole windows, and steps outside them
        win.md_steps(a, n)
        for k in range(n):
            one.md_steps(a + k, 1)
        a += n
        for x, y in zip(result(one, len(ws)), result(win, len(ws))):
            assert np.array_equal(x, y), (a, np.abs(x - y).max())
