"""The hand-over between the proposal windows of a slice, explored on the CPU.

In a round every warp posts its candidate, waits at the block barrier and reads
all posts; with a candidate there the warps meet at a second barrier and go
round again, without one they go to the next window.  All interleavings of the
warps are walked, each post going to the word that the kernel's own header
(csrc/z2_window.h) gives it: no warp may read a post of another round than its
own, and all warps must leave together."""
import ctypes
import itertools
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "z2_gauge_zfy_b200", "csrc")


@pytest.fixture(scope="module")
def first_word(tmp_path_factory):
    d = tmp_path_factory.mktemp("window")
    src, so = d / "w.cpp", d / "w.so"
    src.write_text('#include "z2_window.h"\n'
                   'extern "C" int w256(int base) { return z2_window_post<256>(base); }\n'
                   'extern "C" int w128(int base) { return z2_window_post<128>(base); }\n')
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-I", CSRC, "-o", str(so), str(src)],
                   check=True)
    lib = ctypes.CDLL(str(so))
    return {256: lib.w256, 128: lib.w128}


def _programs(nt, accepts, first_word, warps):
    """Each warp's steps: post, barrier, read per round; a second barrier after a
    round with a candidate.  A post or read names its round (window, round)."""
    out = []
    for w in range(warps):
        steps = []
        for win, n in enumerate(accepts):
            word = first_word[nt](win * nt)
            for r in range(n + 1):
                steps += [("post", word + w, (win, r)), ("bar",), ("read", word, (win, r))]
                if r < n:
                    steps.append(("bar",))
        out.append(tuple(steps))
    return out


def _explore(progs):
    """False as soon as some order of the warps lets one read another round's post."""
    warps = len(progs)
    seen = set()
    todo = [((0,) * warps, (0,) * warps, ())]     # positions, barriers passed, memory
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        pos, bars, mem = state
        m = dict(mem)
        for w in range(warps):
            if pos[w] == len(progs[w]):
                continue
            step = progs[w][pos[w]]
            nm, nb = m, bars
            if step[0] == "post":
                nm = dict(m)
                nm[step[1]] = step[2]
            elif step[0] == "read":
                if any(m.get(step[1] + k) != step[2] for k in range(warps)):
                    return False
            else:
                # a warp passes its k-th barrier once every warp has arrived there
                k = bars[w] + 1
                arrived = [bars[v] + (pos[v] < len(progs[v]) and progs[v][pos[v]][0] == "bar")
                           for v in range(warps)]
                if min(arrived) < k:
                    continue
                nb = bars[:w] + (k,) + bars[w + 1:]
            todo.append((pos[:w] + (pos[w] + 1,) + pos[w + 1:], nb, tuple(sorted(nm.items()))))
    return True


@pytest.mark.parametrize("nt,warps", [(256, 2), (256, 3), (128, 2)])
def test_no_round_reads_another_rounds_posts(first_word, nt, warps):
    for accepts in itertools.product((0, 1), repeat=3):       # three windows
        assert _explore(_programs(nt, accepts, first_word, warps)), accepts


def test_sets_fit_the_flags_and_do_not_overlap(first_word):
    for nt in (128, 256):
        words = [first_word[nt](win * nt) for win in range(4)]
        assert words[0] == words[2] and words[1] == words[3]
        assert abs(words[0] - words[1]) >= nt // 32
        assert 0 <= min(words) and max(words) + nt // 32 <= 16
