"""The search over schedules times launches, not names: classes that differ in mode, waves or
N-tile alone run alike, and the plan over all classes is the fastest block shape, B form and order."""
import pytest

from dtc_b200 import costmodel as cm

pytestmark = pytest.mark.gpu


def _matrix():
    import torch
    from dtc_b200 import gen, metcf
    A = gen.zipf(20000, seed=4)
    rp, col = torch.from_numpy(A.rowptr).cuda(), torch.from_numpy(A.col).cuda()
    return rp, col, metcf.convert(rp, col, A.M, values=torch.from_numpy(A.val).cuda())


def test_plan_over_all_classes_times_each_launch_once(cuda, monkeypatch):
    rp, col, m = _matrix()
    timed = []
    run = cm.tune.run

    def count(mm, planes, fmt, N, prec, sched, **kw):
        timed.append((mm.H, mm.W, fmt, id(mm)))
        return run(mm, planes, fmt, N, prec, sched, **kw)
    monkeypatch.setattr(cm.tune, "run", count)
    s = cm.Scheduler()
    plan = s.plan(rp, col, m, 128, reps=2, verify_top=cm.K)
    # twelve launches: two orders, three block shapes, two forms (one run and two timed ones each)
    assert len(set(timed)) == 12 and len(timed) == 12 * 3
    assert plan.source == "model+verify" and (plan.H, plan.W) in cm.SHAPES


def test_autotune_gives_equal_launches_one_time(cuda):
    import torch
    from dtc_b200 import tune
    _, _, m = _matrix()
    B = torch.randn(m.M, 512, device="cuda")
    scheds, best = tune.autotune(m, [B], tune.FORMS["tf32"][0], 512, tune.FORMS["tf32"][1], reps=2)
    assert len(scheds) == len(tune.candidates(512)) and len({s.ms for s in scheds}) == 1
    outs = [tune.run(m, [B], tune.FORMS["tf32"][0], 512, tune.FORMS["tf32"][1], s) for s in
            (best, scheds[-1])]
    assert torch.equal(*outs)
