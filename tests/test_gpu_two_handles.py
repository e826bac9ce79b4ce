"""Handles alive at the same time: what one of them plans (shared memory of its launches) leaves the
launches of the others as they were.  Bitwise against the same handle by itself."""
import numpy as np
import pytest

from souffle_gb300 import geometry, gpu, workloads

pytestmark = pytest.mark.gpu


def handle(template, S, **kw):
    w = workloads.make(geometry.template_by_name(template), S, seed=90 + S)
    s = gpu.GpuSystem(w.template, [gpu.system_params(w.opt, w.derived, S, w.center_local)], **kw)
    s.set_state(w.state.pos, w.state.vel)
    return s


def run(s):
    f = s.forces(rebuild=True, parts=True)
    s.md_begin()
    s.md_steps(0, 23)  # windows and single steps
    tot, per = s.energies(per_bead=True)
    return list(f) + list(s.get_state()) + [np.array(s.md_scalars())] + [per[k] for k in sorted(per)] + [np.array(list(tot.values()))]


@pytest.mark.parametrize("template,S,kw", [
    ("bilayer_n5", 64, {}),                                                       # the window kernel's wide form
    ("bilayer_n5", 800, {}),                                                      # dealt subunits
    ("bilayer_n5", 40, {"subunits_per_cta": 16, "threads_per_cta": 256}),         # above 48 KB
])
def test_an_older_handle_runs_beside_newer_ones(template, S, kw):
    alone = handle(template, S, **kw)
    want = run(alone)
    alone.close()
    first = handle(template, S, **kw)
    others = [handle("bilayer_n5", 600), handle("bilayer_n5", 2000), handle("patch_n3", 20), handle("patch_n3", 1)]
    got = run(first)
    for x, y in zip(want, got):
        assert np.array_equal(x, y)
    for o in others:
        run(o)
