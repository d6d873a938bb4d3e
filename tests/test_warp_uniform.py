"""The batched planner's search for work (batch_kernel.cuh) runs as one warp:
its whole-warp instructions (`..._sync(FULL, ...)`) may not depend on a value
that each lane reads from memory for itself, since other warps change that
memory meanwhile and lanes that read different values would part at the
instruction.  Read from the source: in the search, no branch on a value that
is read or derived per lane holds a whole-warp instruction."""
import re
from pathlib import Path

SRC = Path(__file__).resolve().parents[1] / "prrtc_gb300" / "csrc" / "batch_kernel.cuh"
WHOLE_WARP = re.compile(r"_sync\(FULL")


def search_block() -> str:
    text = re.sub(r"//[^\n]*", "", SRC.read_text().split("// ---- find work", 1)[1].split("// ---- one round of", 1)[0])
    return text


def balanced(text: str, at: int, pair: str) -> int:
    """Index behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced")


def branches(text: str):
    """(condition, controlled statement) of every if, for and while."""
    for m in re.finditer(r"\b(?:if|for|while)\s*\(", text):
        end = balanced(text, m.end() - 1, "()")
        rest = text[end:]
        pad = len(rest) - len(rest.lstrip())
        at = end + pad
        if text[at] == "{":
            body = text[at:balanced(text, at, "{}")]
        else:
            body = text[at:text.index(";", at) + 1]
        yield text[m.end():end - 1], body


def per_lane(text: str) -> set:
    """Names that hold a value read, or derived from one read, per lane."""
    outside = text
    for cond, body in branches(text):          # lane 0's own work is shared by a shuffle
        if re.fullmatch(r"\s*lane == 0.*", cond, re.S):
            outside = outside.replace(body, ";", 1)
    names = {"lane"}
    assigned = re.findall(r"\b(\w+) = ([^;]*);", outside)
    while True:
        more = {n for n, v in assigned if not re.match(r"\s*__\w+_sync\(FULL", v) and
                ("vload(" in v or "volatile" in v or names & set(re.findall(r"\w+", v)))}
        if more <= names:
            return names
        names |= more


def offending(text: str) -> list:
    names = per_lane(text)
    return [c for c, body in branches(text) if WHOLE_WARP.search(body) and names & set(re.findall(r"\w+", c))]


def test_search_branches_on_whole_warp_values():
    text = search_block()
    assert WHOLE_WARP.search(text) and {"st", "run", "w"} <= per_lane(text)   # the reading sees the search
    assert offending(text) == []


def test_the_reading_sees_a_per_lane_condition():
    """A queue position that every lane reads for itself is found."""
    text = re.sub(r"int pending = 0;\s*if \(lane == 0\) pending = ([^;]*);\s*pending = __shfl_sync\(FULL, pending, 0\);",
                  r"const bool pending = \1;", search_block())
    assert any("pending" in c for c in offending(text))
