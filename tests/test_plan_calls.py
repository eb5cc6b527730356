"""Call numbers of a plan (no GPU: the library is a fake that records what it is asked to launch)."""
import pytest

from tileccl_b200.ops import _plan


class _FakeLib:
    def __init__(self):
        self.numbers, self.rc = [], 0

    def tcl_gemm_plan_run(self, handle, number, stream):
        self.numbers.append(number)
        return self.rc

    def tcl_gemm_plan_run_on(self, handle, a, b, number, stream):
        return self.tcl_gemm_plan_run(handle, number, stream)

    def tcl_gemm_plan_destroy(self, handle):
        pass


@pytest.mark.parametrize("call", [lambda p: p.run(), lambda p: p.run_on(16, 32)], ids=["run", "run_on"])
def test_a_refused_launch_does_not_use_up_a_call_number(monkeypatch, call):
    """Peers compare their counters with call number x producers: a rank whose operand was refused must make its
    next call under the number that its peers expect."""
    monkeypatch.setattr(_plan, "raw_stream", lambda stream=None: 0)
    fake = _FakeLib()
    plan = _plan.Plan.__new__(_plan.Plan)
    plan.lib, plan.handle, plan.epoch_dev, plan._host_epoch, plan.launches = fake, 1, None, 0, 0
    call(plan)
    fake.rc = 716
    with pytest.raises(RuntimeError):
        call(plan)
    fake.rc = 0
    call(plan)
    assert fake.numbers == [1, 2, 2]
    assert plan.epoch == 2 and plan.launches == 2
