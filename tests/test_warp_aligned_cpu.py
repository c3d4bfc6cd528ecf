"""Instructions that a warp has to reach as one: cluster and named barriers, register hand-over, TMEM allocation, release, loads and stores (PTX `.aligned`;
bar.sync and bar.arrive are the aligned forms of barrier.*).  What they do while lanes of the warp are apart is undefined, and lanes come apart in any loop or
branch of theirs in front.  So the statement before each of them has to bring the warp together, whatever the caller did.  This reads the sources: a
kernel that breaks the rule may well run as intended, until a compiler lays its branches out differently."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "seq2seqsharp_b200", "csrc")
ALIGNED = re.compile(r"\.aligned\b|\bbar\.(sync|arrive|red)\b|\bbarrier\.cluster\b")
PRODUCTS = re.compile(r"\b(mma|wmma|ldmatrix|stmatrix|movmatrix)\.")      # in loops whose trip counts are the warp's


def statements(text):
    """Statements in order, comments gone, every string literal replaced by ALIGNED, PRODUCT or TEXT."""
    tokens = re.compile(r'//[^\n]*|/\*.*?\*/|"(?:\\.|[^"\\])*"|\'(?:\\.|[^\'\\])\'', re.S)

    def word(m):
        t = m.group(0)
        if t[0] == "/":
            return " "
        return " PRODUCT " if PRODUCTS.search(t) else (" ALIGNED " if ALIGNED.search(t) else " TEXT ")
    text = re.sub(r"^\s*#\s*pragma[^\n]*", "", text, flags=re.M)
    return [s.strip() for s in re.split(r"([;{}])", tokens.sub(word, text)) if s.strip() and s.strip() != ";"]


def offenders(text):
    last, out = "", []
    for s in statements(text):
        aligned = "ALIGNED" in s and "PRODUCT" not in s
        bare = aligned and s.startswith("asm")       # not the body of a condition
        if aligned and not (bare and (last == "aligned" or re.fullmatch(r"__sync(warp|threads)\(\)", last))):
            out.append(s)
        last = "aligned" if bare else s
    return out


def test_the_reader_sees_what_it_should():
    assert offenders('f(); asm volatile("bar.sync 1, 256;" ::: "memory");')
    assert offenders('__syncwarp(); if (x) asm volatile("barrier.cluster.arrive.aligned;");')
    assert not offenders('__syncwarp(); asm volatile("barrier.cluster.arrive.aligned;"); asm volatile("barrier.cluster.wait.aligned;");')
    assert not offenders('f(); asm volatile("mma.sync.aligned.m16n8k16;"); // bar.sync\n g("x; y");')


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_the_warp_is_together_before_aligned_instructions(name):
    with open(os.path.join(CSRC, name)) as f:
        assert offenders(f.read()) == []
