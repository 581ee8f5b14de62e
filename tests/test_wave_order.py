"""The launch order inside a wave, read from the source: a kernel that starts
before its predecessor has completed ("beside") takes over the visibility of
what it reads through a mark before it reads anything, the kernel that heads
such a chain releases that mark after its own wait, and no kernel of a wave
reads a count or a queue, which change while it may already be resident,
through the read-only path."""
import re
from pathlib import Path

import pytest

SRC = (Path(__file__).resolve().parents[1] / "slr_gb300" / "csrc" / "render.cu").read_text()


def _kernels():
    """name -> (parameter list, body) of the kernels launched in wave order."""
    launched = set(re.findall(r"launchWaveKernel\((k\w+)", SRC))
    found = {}
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(k\w+)\(", SRC):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(SRC[i], 0)
            i += 1
        params, start, depth = SRC[m.end():i - 1], SRC.index("{", i), 0
        for j in range(start, len(SRC)):
            depth += {"{": 1, "}": -1}.get(SRC[j], 0)
            if depth == 0:
                break
        found[m.group(1)] = (params, SRC[start + 1:j])
    assert launched <= set(found)
    return {k: found[k] for k in sorted(launched)}


KERNELS = _kernels()


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_no_count_or_queue_through_the_read_only_path(name):
    params, body = KERNELS[name]
    assert not re.search(r"const uint32_t\s*\*\s*__restrict__", params + body)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_the_wait_or_the_mark_comes_before_the_first_read(name):
    params, body = KERNELS[name]
    begin = re.search(r"waveBegin(After|Beside)?\(([^;]*)\);", body)
    assert begin
    before = body[:begin.start()]
    # nothing but shared-memory declarations and the choice of the parameter block
    before = re.sub(r"__shared__[^;]*;|const WaveParams &wp = wpDev \? \*wpDev : wpArg;|if \(!MULTI\)|//[^\n]*", "", before)
    assert before.strip() == ""
    if "waveEnd" in body:     # it may start before its predecessor has completed
        assert begin.group(1) != "After" and "mark" in begin.group(2)
        assert re.search(r"uint32_t\* mark", params)


def test_marks_are_released_after_the_wait_and_acquired():
    after = re.search(r"void waveBeginAfter\(.*?\n}", SRC, re.S).group(0)
    assert after.index("waveWait()") < after.index("st.release.gpu") < after.index("waveTrigger()")
    beside = re.search(r"void waveBeginBeside\(.*?\n}", SRC, re.S).group(0)
    assert beside.index("ld.acquire.gpu") < beside.index("__syncthreads_and") < beside.index("waveWait()")


def test_every_chain_of_beside_kernels_has_a_head_that_marks():
    for head, mark, users in (("kExtendSort", "kCtrExtMark", ["kShadow"]), ("kExtend", "kCtrExtMark", ["kShadowVol"]),
                              ("kVolInteract", "kCtrVolMark", ["kShadowVolMedium"])):
        assert mark in re.search(r"waveBeginAfter\(([^;]*)\);", KERNELS[head][1]).group(1)
        for user in users:
            calls = re.findall(rf"launchWaveKernel\({user}(?:<\w+>)?,[^;]*;", SRC)
            assert calls and all(mark in c for c in calls)
    # the shading kernels share one mark: the first stores it, the others load it
    for name in ("kShadeMiss", "kShadeSurf", "kShadeVol"):
        assert re.search(r"waveBegin\(mark, beside\);", KERNELS[name][1])
        calls = re.findall(rf"launchWaveKernel\({name}<[^;]*beside\)", SRC)
        assert calls and all("ctr + kCtrShadeMark, beside" in c for c in calls)
