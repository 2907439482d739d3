"""What the kernels hand over through mbarriers, read from their source.  A warp whose lanes have written data says so with one lane's arrival; that
lane's release covers the other lanes' writes only behind a warp barrier (a shuffle or a vote orders no memory), and a wrong order would show on the
GPU now and then or never."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "vllm-backend-public_b200" / "csrc"
KERNELS = sorted(p.name for p in CSRC.glob("*_tc5.cu"))
# arrivals that carry only the arriving lane's own work, or none
OWN = {
    ("delta_tc5.cu", "out(u)"): "its own bulk stores have been read",
    ("delta_tc5.cu", "stored"): "its own bulk stores have been read",
    ("latent_tc5.cu", "full"): "the other warp's boxes fill the stage",
    ("prompt_turns_tc5.cu", "bar(L::BAR_P + lane)"): "TMEM is free at the start",
}


def _code(name):
    return [re.sub(r"//.*", "", line) for line in (CSRC / name).read_text().splitlines()]


@pytest.mark.parametrize("name", KERNELS)
def test_one_lane_arrives_behind_a_warp_barrier(name):
    lines = _code(name)
    loose = []
    for i, line in enumerate(lines):
        for m in re.finditer(r"b2::mbar_arrive\((.*?)\);", line):
            before = [s.strip() for s in lines[max(0, i - 5):i + 1] if s.strip()]
            # back from the arrival: its guard and writes of the arriving lane itself, then the barrier
            ok = False
            for s in reversed(before):
                if "__syncwarp();" in s:
                    ok = True
                    break
                if not (s == before[-1] or re.match(r"(if|\} else if|for) \(|[\w.\->\[\]]+ = [^;]*;$", s)):
                    break
            if not ok and (name, m.group(1)) not in OWN:
                loose.append((i + 1, line.strip()))
    assert not loose, loose


# kernels whose waits may give up, and the barriers that their boxes or MMAs complete
IN_FLIGHT = [
    ("prompt_turns_tc5.cu", "prompt_turns_kernel", ["L::BAR_Q)", "L::BAR_Q + 1)", "L::BAR_V : L::BAR_K"]),
    ("prompt_tc5.cu", "prompt_tc5_kernel", ["L::BAR_V : L::BAR_K"]),
    ("latent_tc5.cu", "latent_tc5_kernel", ["FULL"]),
    ("moe_tc5.cu", "moe_tc5_kernel", ["full(", "s_end"]),
    ("delta_tc5.cu", "chain_kernel", ["here(", "done"]),
    ("delta_tc5.cu", "read_kernel", ["s_here", "s_done"]),
]


@pytest.mark.parametrize("name,kernel,bars", IN_FLIGHT)
def test_what_is_in_flight_is_waited_for_when_a_wait_gave_up(name, kernel, bars):
    """A wait of any role may give up last, when those that copy have left their loops: what is under way is waited for behind a barrier of the
    whole CTA, not where a copying warp's own wait failed."""
    text = "\n".join(_code(name))
    body = text[text.index(kernel + "("):]
    body = body[:body.index("\n}\n")]
    at_end = body[body.rindex("__syncthreads();"):]
    drained = re.findall(r"drain\((.*)", at_end)
    assert re.search(r"if \([^{]*failed", at_end)
    for bar in bars:
        assert any(bar in d for d in drained), (bar, drained)
