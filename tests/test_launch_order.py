"""Reads behind a kernel's wait for the kernel in front, by the sources: a kernel that works before ``pdl_wait()`` passes every
``__restrict__`` pointer to memory that earlier kernels write through ``pdl_fresh`` behind it.  The compiler takes such memory for
unchanging while the kernel runs, so that it may move its loads above the wait; what that yields depends on the timing of two kernels
and cannot be provoked."""
import re
from pathlib import Path

import pytest

SOURCES = sorted((Path(__file__).resolve().parent.parent / "airframe_b200" / "csrc").glob("*.cu"))

# Memory that no kernel of a step writes: the step's inputs and the model's weights.
FIXED = {"positions", "seq_of_token", "seq_starts", "seq_first_chunk", "chunk_starts", "tiles", "slots", "lens", "len_after", "page_table",
         "inv_freq", "bias", "q_weight", "k_weight", "sinks", "slopes", "w", "w0", "w1", "w2t", "w_post", "w_next", "b_post", "b_next", "a_bias",
         "ls", "mu", "mix", "out_w", "in_next", "ba", "bi", "rate", "bx", "by", "bz", "cw", "cb"}
FIXED_IN = {("expert_plan_kernel", "table")}                       # (the experts of every token id)
WRITTEN_IN = {("chunk_cumulate_kernel", "w")}                      # (a projection's decays)


def kernels():
    for path in SOURCES:
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            at = text.find("{", m.end())
            head = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)|__cluster_dims__\s*\([^()]*\)", "", text[m.end():at])
            if ";" in head:
                continue                                           # (a declaration)
            depth, end = 0, at
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
                if depth == 0:
                    break
            yield path.name, re.search(r"(\w+)\s*\(", head).group(1), head[head.find("("):], text[at:end]


def loads(code):
    """Whether code in front of the wait reads memory through a pointer (declarations of arrays are no reads)."""
    code = re.sub(r"__shared__[^;]*;", "", code)
    return re.search(r"=[^=;]*\w\[[^\]]*\]|->|__ldg|\(const \w+4? ?\*\)|qk_cache_rows|reinterpret_cast<const", code) is not None


CASES = [pytest.param(*k, id=k[1]) for k in kernels() if "pdl_wait()" in k[3] and loads(k[3].split("pdl_wait()")[0])]


def test_kernels_were_found():
    assert len(CASES) > 30


@pytest.mark.parametrize("file, name, head, body", CASES)
def test_what_earlier_kernels_write_is_read_behind_the_wait(file, name, head, body):
    behind = body.split("pdl_wait()", 1)[1]
    fresh = set(re.findall(r"pdl_fresh\((\w+)\)", body))
    # (a row's pointer that is made from the parameter before the wait and re-derived behind it)
    fresh |= {m.group(2) for m in re.finditer(r"(\w+) = (\w+) \+[^;]*;", body) if m.group(1) in fresh}
    stale = []
    for const, p in re.findall(r"(const )?\w+\*\s*__restrict__ (\w+)", head):
        if p in fresh or not re.search(rf"\b{p}\b", behind):
            continue
        if const:
            read = (name, p) not in FIXED_IN and (p not in FIXED or (name, p) in WRITTEN_IN)
        else:
            read = p in ("x", "state", "prev", "local") or re.search(rf"\b{p}\[[^;=]*\] [-+*]=", behind) is not None
        if read:
            stale.append(p)
    assert not stale, f"{file}: {name} reads {stale} behind pdl_wait() as it was passed"
