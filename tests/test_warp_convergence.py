"""Warps are converged where the tensor-core kernels need them to be.

tcgen05.ld.sync.aligned and the named barriers are instructions of a whole
converged warp.  A lane that polls an mbarrier leaves its loop on its own, so

  - mbar_wait_bounded may be called by a single thread only: inside a branch or
    a conditional expression that picks one thread (every lane of a warp waits
    through mbar_wait_warp, whose vote brings the lanes together);
  - the wrappers of those instructions start with __syncwarp().

Read from the source: running the contrary is not an option."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "hairmsnn_gb300" / "csrc"
ONE = r"(?:leader|tid == 0|lane == 0|threadIdx\.x == 0)"


def code(path):
    text = re.sub(r"/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m.group()), path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), text)


def body(text, signature):
    at = text.index("{", text.index(signature))
    depth = 0
    for k in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[at + 1:k]
    raise AssertionError(signature)


def unguarded(text):
    """Lines of mbar_wait_bounded calls outside every one-thread branch."""
    bad, heads, stmt = [], [], 0
    for k, c in enumerate(text):
        if c == "{":
            heads.append(text[stmt:k])
            stmt = k + 1
        elif c == "}":
            if heads:
                heads.pop()
            stmt = k + 1
        elif c == ";" and text.count("(", stmt, k) == text.count(")", stmt, k):
            stmt = k + 1
        elif text.startswith("mbar_wait_bounded(", k):
            picks = any(re.search(r"\bif \([^{]*\b" + ONE + r"[^{]*\)\s*$", h) for h in heads)
            picks = picks or re.search(r"\b" + ONE + r"\s*\?", text[stmt:k]) is not None
            if not picks:
                bad.append(text[text.rfind("\n", 0, k) + 1:text.index("\n", k)].strip())
    return bad


@pytest.mark.parametrize("name", ["hm_mlp_tc.cu", "hm_mlp_x3.cu"])
def test_only_single_threads_wait_without_a_vote(name):
    assert unguarded(code(CSRC / name)) == []


def test_guard_is_recognised():
    assert unguarded("if (leader) { ok = mbar_wait_bounded(b, 0); }\n") == []
    assert unguarded("const bool ok = tid == 0 ? mbar_wait_bounded(b, 0) : true;\n") == []
    bare = "for (;;) { ok = ok && mbar_wait_bounded(b, 0); }"
    assert unguarded(bare + "\n") == [bare]


@pytest.mark.parametrize("signature", ["void tmem_ld16(", "void group_sync(", "bool group_sync_or("])
def test_warp_instructions_start_converged(signature):
    text = body(code(CSRC / "hm_tc.cuh"), signature)
    assert "__syncwarp();" in text[:text.index("asm volatile")]


def test_vote_follows_the_wait():
    assert "__all_sync(0xffffffffu, mbar_wait_bounded(" in body(code(CSRC / "hm_tc.cuh"), "bool mbar_wait_warp(")
