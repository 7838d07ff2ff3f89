"""bench.py's reference arm: kernels that cannot be loaded are reported in one line, a failure of the
run itself is raised (no GPU needed)."""
import json
import types

import pytest

import bench
from oracle import oracle as O

ARGS = types.SimpleNamespace(steps=1, warmup=3, sessions=64)


@pytest.mark.parametrize("error,text", [(RuntimeError("not built\nsecond line"), "not built"),
                                        (OSError(), "OSError()"), (RuntimeError(""), "RuntimeError('')")])
def test_kernels_that_cannot_be_loaded_are_reported(monkeypatch, capsys, error, text):
    def ref():
        raise error
    monkeypatch.setattr(O, "ref", ref)
    assert bench.run_reference(ARGS, 0, 1) == 0
    assert json.loads(capsys.readouterr().out) == {"impl": "reference", "unavailable": text}


@pytest.mark.parametrize("error", [RuntimeError("a stage failed"), OSError("no frames")])
def test_a_failing_run_is_raised(monkeypatch, error):
    def run(args, **kw):
        raise error
    monkeypatch.setattr(O, "ref", lambda: object())
    monkeypatch.setattr(bench, "cpu_baseline", run)
    with pytest.raises(type(error)):
        bench.run_reference(ARGS, 0, 1)
