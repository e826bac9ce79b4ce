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


@pytest.mark.parametrize("template,S,over", [("patch_n3", 20, {}), ("bilayer_n5", 800, {}), ("bilayer_n5", 33, {"D": "b", "d": 100.0})])
def test_a_wait_that_runs_out_is_reported_and_the_state_has_to_be_set_again(template, S, over):
    w = workloads.make(geometry.template_by_name(template), S, seed=12, **over)
    good = handle([w])
    good.md_steps(0, 30)
    want = result(good, 1)
    s = handle([w])
    polls = s.lib.souffle_gpu_window_polls
    polls.argtypes, polls.restype = [gpu.C.c_void_p, gpu.C.c_uint32], gpu.C.c_int32
    assert polls(s.h, 0) > 0  # every wait gives up at its first look
    s.md_enqueue(0, 30)       # the windows behind the failing one leave at once
    with pytest.raises(gpu.SouffleError) as e:
        s.synchronize()
    assert e.value.code == 2 and "wait ran out" in str(e.value)
    for call in (lambda: s.md_steps(30, 10), s.md_begin, s.get_state, s.energies, lambda: s.forces(rebuild=False)):
        with pytest.raises(gpu.SouffleError) as e:
            call()
        assert e.value.code == 6  # no state
    polls(s.h, 1 << 22)
    s.set_state(w.state.pos, w.state.vel)
    s.md_begin()
    s.md_steps(0, 30)
    for x, y in zip(want, result(s, 1)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("template,subs,over", [
    ("patch_n3", [20], {}), ("bilayer_n5", [64], {}), ("bilayer_n5", [1700], {}), ("bilayer_n5", [5, 17, 2], {}),
    ("bilayer_n5", [33], {"D": "b", "d": 100.0}), ("bilayer_n5", [3000], {})])
@pytest.mark.parametrize("begun", [False, True])
def test_autotune_keeps_the_windows_and_the_state(template, subs, over, begun):
    """The shape is chosen by the steps that the handle takes: one that cannot take windows never wins over
    one that can, and the steps timed leave no trace."""
    ws = [workloads.make(geometry.template_by_name(template), S, seed=40 + S, **over) for S in subs]
    a, b = handle(ws), handle(ws)
    if begun:
        a.md_steps(0, 10)
        b.md_steps(0, 10)
    else:
        for s in (a, b):
            s.set_state(np.concatenate([w.state.pos for w in ws]), np.concatenate([w.state.vel for w in ws]))
    polls = b.lib.souffle_gpu_window_polls
    polls.argtypes, polls.restype = [gpu.C.c_void_p, gpu.C.c_uint32], gpu.C.c_int32
    had = polls(b.h, 1 << 22)
    t = b.autotune(trials=20)
    print(t, had, polls(b.h, 1 << 22))
    assert t["candidates"] >= 3 and 0 < t["forces_us"] <= t["default_forces_us"]
    assert (polls(b.h, 1 << 22) > 0) == (had > 0)
    if not begun:
        a.md_begin()
        b.md_begin()
    a.md_steps(10, 20)
    b.md_steps(10, 20)
    for x, y in zip(result(a, len(ws)), result(b, len(ws))):
        assert np.array_equal(x, y)
