"""Memory order of the ray queues' warp cursor (kernel sources, read as text).

A source that keeps a cursor per warp in shared memory has it written by one
refill's leader lane and read by the next one's.  Only __syncwarp() orders the
two (shuffles and votes do not), and no run on a GPU can show that it is
missing: so every refill claims through claim_slots, which synchronises between
the claim and the shuffles that publish it, for each such source."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "renderbox2_b200" / "csrc"
KERNELS = {p.name: p.read_text() for p in sorted(CSRC.glob("*.cu*"))}


def test_refills_claim_in_order():
    claims = [(name, m.start()) for name, s in KERNELS.items() for m in re.finditer(r"\bsrc\.claim\(", s)]
    assert [name for name, _ in claims] == ["rb2_traverse.cuh"]
    body = KERNELS["rb2_traverse.cuh"][claims[0][1]:]
    assert re.match(r"src\.claim\([^;]*;\s*if constexpr \(Source::kWarpCursor\) __syncwarp\(\);\s*b1 = __shfl_sync", body)
    assert KERNELS["rb2_traverse.cuh"].count("claim_slots(src,") == 1
    assert KERNELS["rb2_traverse_cw8.cuh"].count("claim_slots(src,") == 1


def test_every_source_with_a_cursor_says_so():
    sources = {}
    for s in KERNELS.values():
        for m in re.finditer(r"^struct (\w+Source) \{(.*?)^\};", s, re.M | re.S):
            sources[m[1]] = m[2]
    assert {"JobSource", "AoSource", "QueueSource", "IsectSource"} <= set(sources)
    for name, body in sources.items():
        claim = body[body.index("void claim("):body.index("fetch(")]
        flag = re.search(r"kWarpCursor = (true|false)", body)
        assert flag, name
        assert (flag[1] == "true") == ("rem" in claim), name
