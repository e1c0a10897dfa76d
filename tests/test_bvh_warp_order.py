"""The warp-built subtrees of the device BVH build (k_small, bvh_build.cu)
exchange primitives in a permutation that every lane of the warp reads.  No
lane may write it while another can still be about to read it, so a warp-wide
barrier stands between the last reads and each write, and between each write
and the next reads.  Whether the lanes happen to run together decides what a
missing barrier does, so its order is read from the source."""
import re
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "zigtrace_b200" / "csrc" / "bvh_build.cu"


def _body(name):
    text = re.sub(r"/\*.*?\*/", " ", SRC.read_text(), flags=re.S)
    at = text.index("{", text.index(f" {name}("))
    depth, end = 0, at
    for end in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        if depth == 0:
            break
    return text[at:end]


def _steps(body):
    """'r' reads of idx, 'w' writes of it, 'b' warp-wide barriers, in order."""
    pat = re.compile(r"(?P<b>__(?:syncwarp|shfl_sync|ballot_sync)\()|(?P<i>\bidx\[[^\]]*\])(?P<eq>\s*=(?!=))?")
    return [(("b" if m["b"] else "w" if m["eq"] else "r"), m.start()) for m in pat.finditer(body)]


def test_a_barrier_separates_reads_and_writes_of_the_permutation():
    body = _body("k_small")
    steps = _steps(body)
    assert {"r", "w", "b"} <= {k for k, _ in steps}
    for (a, at), (b, _) in zip(steps, steps[1:]):
        assert (a, b) not in (("r", "w"), ("w", "r")), body[max(0, at - 120):at + 200]


def test_every_turn_of_the_loop_ends_with_a_barrier():
    """The next turn reads what this one wrote."""
    body = _body("k_small")
    turns = re.findall(r"__syncwarp\(\);\s*continue;", body)
    assert len(turns) == len(re.findall(r"\bcontinue;", body)) - len(re.findall(r"!= \(uint32_t\)lane\) continue;", body))
    assert re.search(r"__syncwarp\(\);\s*\}\s*if \(lane == 0\) st\.internal", body)
