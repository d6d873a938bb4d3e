"""Entry points that hold a context's lock call none that takes it: the lock is
a plain mutex, and an error path that freed a batch through prrtc_batch_free
while it was held never returned.  Read from the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "prrtc_gb300" / "csrc"
FUNCTION = re.compile(r"^(?:extern \"C\" )?(?:static )?[\w:]+(?: \*?|\*)(prrtc_\w+)\([^;{]*\)\n\{\n(.*?)^\}", re.S | re.M)


def functions():
    out = {}
    for f in CSRC.glob("*.cu"):
        out |= {name: body for name, body in FUNCTION.findall(f.read_text())}
    return out


def offending(bodies):
    locking = {n for n, b in bodies.items() if re.search(r"lock_guard<std::mutex> \w+\(c->mu\)", b)}
    bad = []
    for name in locking:
        held = bodies[name].split("lock_guard", 1)[1]
        bad += [(name, callee) for callee in re.findall(r"\b(prrtc_\w+)\(", held) if callee in locking]
    return locking, bad


def test_no_locking_entry_point_is_called_with_the_lock_held():
    locking, bad = offending(functions())
    assert {"prrtc_batch_create", "prrtc_batch_free", "prrtc_env_upload", "prrtc_solve"} <= locking
    assert bad == []


@pytest.mark.parametrize("call", ["prrtc_batch_free(ctx, b);"])
def test_the_reading_sees_such_a_call(call):
    bodies = functions()
    bodies["prrtc_batch_create"] += call
    assert ("prrtc_batch_create", "prrtc_batch_free") in offending(bodies)[1]
