"""The word in which kernels say that a bounded wait gave up is looked at wherever such kernels ran: also where a graph was replayed and
where decode steps run ahead of the host.  The word is set from the host; no wait has to run out for that."""
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.fixture
def engine(tmp_path):
    """An engine whose graphs go when the test ends: the errors that it expects keep frames alive, and a graph that is collected while another is
    captured spoils that capture."""
    made = []

    def make(dtype, n):
        made.append(_engine(tmp_path, dtype, n))
        return made[0]

    yield make
    made[0].runner._graphs.clear()


def _engine(tmp_path, dtype, n, max_new=12):
    from return_b200.engine.config import EngineConfig
    from return_b200.engine.engine import Engine
    from return_b200.engine.request import Request
    d = helpers.make_model_dir(tmp_path, "B")
    eng = Engine(d, EngineConfig(max_token=1024, max_reside=n, page_size=8, prefill_chunk=64, dtype=dtype, use_cuda_graph=True))
    for i in range(n):
        eng.add_request(Request(f"r{i}", helpers.random_ids(384, 3 + i, i), max_new_tokens=max_new, temperature=0.0))
    return eng


def _raise_word():
    from return_b200.ext import ops
    ops.tc5_status(DEV).fill_(1)


# a step of 12 tokens in bfloat16 runs the rows' products, one of 3 in float32 the split ones
@pytest.mark.parametrize("dtype,n", [("bfloat16", 12), ("float32", 3)])
def test_replayed_step(engine, dtype, n):
    from return_b200.ext import ops
    eng = engine(dtype, n)
    while not eng._can_run_ahead():
        eng.step()
    eng.step()                                                # captures
    eng.step()
    ops.check_status(DEV)
    _raise_word()
    with pytest.raises(ops.KernelError, match="bounded wait"):
        eng.step()
    assert int(ops.tc5_status(DEV)) == 0                      # read and put back


@pytest.mark.parametrize("dtype,n", [("bfloat16", 12), ("float32", 3)])
def test_steps_that_run_ahead(engine, monkeypatch, dtype, n):
    from return_b200.ext import ops
    eng = engine(dtype, n)
    while not eng._can_run_ahead():
        eng.step()
    calls, step = [], eng.runner.step

    def third_goes_wrong(*args):
        logits = step(*args)
        calls.append(1)
        if len(calls) == 3:
            _raise_word()
        return logits

    monkeypatch.setattr(eng.runner, "step", third_goes_wrong)
    before = {r.id: len(r.output) for r in eng.scheduler.running}
    with pytest.raises(ops.KernelError, match="bounded wait"):
        eng.run()
    assert all(len(r.output) - before[r.id] <= 2 for r in eng.scheduler.running)       # nothing of the third step was given out


def test_a_graph_without_such_kernels_asks_for_nothing(engine):
    from return_b200.ext import ops
    eng = engine("bfloat16", 3)                    # weight streaming and decode attention: no wait
    while not eng._can_run_ahead():
        eng.step()
    eng.step()
    ops.check_status(DEV)
    eng.step()
    assert DEV not in ops._tc5_launched


def test_every_launch_with_bounded_waits_is_known():
    from return_b200.ext import ops
    x, w = torch.randn(16, 128, device=DEV).bfloat16(), torch.randn(64, 128, device=DEV).bfloat16()
    out, wide = torch.empty(16, 64, device=DEV, dtype=torch.bfloat16), torch.empty(16, 128, device=DEV)
    for launch in (lambda: ops.gemm_tc5(x, w, out, simple_bn=64), lambda: ops.gemm_rows(x, w, out), lambda: ops.gemm_stream(x, w, out),
                   lambda: ops.gemm_tc5_bmn(x, torch.randn(128, 128, device=DEV).bfloat16(), wide),
                   lambda: ops.gemm_f32(x.float(), w.float(), wide[:, :64])):
        ops.check_status(DEV)
        assert DEV not in ops._tc5_launched
        launch()
        assert DEV in ops._tc5_launched
    ops.check_status(DEV)
