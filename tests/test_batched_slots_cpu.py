"""The partial-sum slots of the grid-wide batched PCG, checked on its source:
its CTAs write their sums to global slots (publish), read everyone's (total)
and meet at grid barriers (sync_grid), so a slot that is both read and written
between two barriers is a race between a CTA ahead and one behind."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _phases():
    """[(slots written, slots read)] of the intervals between the barriers of
    one pass, with the first pass's extra ones, in program order."""
    src = open(os.path.join(ROOT, "simit_gb300", "csrc", "sg_batched.cu")).read()
    names = dict((k, int(v)) for k, v in re.findall(r"\b(DS_\w+) = (\d+)", src))
    body = src[src.index("k_batched_grid(GridArgs g) {"):]
    body = body[body.index("for (int64_t pass"):body.index("// Lanes per row, threads per CTA")]
    for k in sorted(names, key=len, reverse=True):
        body = re.sub(r"\b%s\b" % k, str(names[k]), body)
    out = [(set(), set())]
    for call in re.findall(r"publish\([^;]*\);|total\([^;]*?\)(?=[,; ])|sync_grid\(\)", body):
        if call.startswith("sync_grid"):
            out.append((set(), set()))
            continue
        inner = call[call.index("(") + 1:call.rindex(")")]
        args = inner.rsplit(", ", 1)
        if call.startswith("publish"):  # slots [first, last); either may be "c ? a : b"
            lo, hi = [[eval(t) for t in a.split("?")[-1].split(":")] for a in args]
            out[-1][0].update(range(min(lo), max(hi)))
        else:
            out[-1][1].add(int(args[1]))
    return out


def test_no_slot_is_read_and_written_between_two_barriers():
    phases = _phases()
    assert len(phases) == 4  # three barriers a pass
    first, last = phases[0], phases[-1]
    phases = [(first[0] | last[0], first[1] | last[1])] + phases[1:-1]
    assert sum(len(w) for w, _ in phases) >= 3 and sum(len(r) for _, r in phases) >= 3
    for written, read in phases:
        assert not written & read, "slots %s" % sorted(written & read)
    assert set().union(*(r for _, r in phases)) <= set().union(*(w for w, _ in phases))
