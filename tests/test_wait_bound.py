"""How long a kernel waits on an mbarrier that never completes: the poll limit of every mbar_wait times the time of a poll."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nanovllm_jax_b200", "csrc")
# measured on a B200 for mbarrier.try_wait with the hint of mbar_wait: 1000 polls of a barrier that nothing completes, 3.995 ms
POLL_NS = 3995


def _value(text, consts):
    text = re.sub(r"\b(\d+)u\b", r"\1", text)
    for name, value in consts.items():
        text = text.replace(name, str(value))
    return int(eval(text, {"__builtins__": {}, "polls_of_ms": lambda ms: ms * 1000000 // consts.get("kPollNanoseconds", 1)}))


def test_no_wait_takes_longer_than_six_seconds():
    with open(os.path.join(CSRC, "common.cuh")) as f:
        header = f.read()
    consts = {m[1]: int(m[2]) for m in re.finditer(r"constexpr uint32_t (\w+) = (\d+);", header)}
    limits = [re.search(r"bool mbar_wait\([^;{]*?limit = ([^{;]+)\) \{", header)[1]]
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name), errors="ignore") if name.endswith((".cu", ".cuh")) else open(os.devnull) as f:
            limits += re.findall(r"mbar_wait\([^;]*?, (polls_of_ms\(\d+\)|[0-9u<() ]+)\);", f.read())
    assert len(limits) >= 2, "the default and the one that lets loads land"
    assert abs(consts.get("kPollNanoseconds", POLL_NS) - POLL_NS) < 100
    for limit in limits:
        assert _value(limit, consts) * POLL_NS < 6e9, f"a wait of {_value(limit, consts) * POLL_NS * 1e-9:.1f} s ({limit})"
