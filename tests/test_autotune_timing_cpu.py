"""The autotuner's timed passes come after the one that an engine captures."""
import importlib
import sys
from types import SimpleNamespace

from conftest import load_package

DIRECT_PASSES = 4  # launched kernel by kernel before an engine captures (csrc/search.cuh)


def test_nothing_is_captured_while_timing(pst):
    load_package()
    autotune = importlib.import_module(sys.modules["pst_b200"].__name__ + ".autotune")
    log = []
    engine = SimpleNamespace(run=lambda *a, sync, **k: log.append("waiting" if sync else "pass"))
    event = lambda **k: SimpleNamespace(record=lambda s: log.append("event"), synchronize=lambda: None,  # noqa: E731
                                        elapsed_time=lambda other: 1.0)
    fake = SimpleNamespace(cuda=SimpleNamespace(Event=event, current_stream=lambda: None, synchronize=lambda: None))
    autotune._time(engine, None, None, None, "ids", 5, fake)
    start, end = [i for i, x in enumerate(log) if x == "event"]
    assert log[start + 1:end] == ["pass"] * 5
    assert log[:start].count("pass") > DIRECT_PASSES  # (waiting passes may take another path)
