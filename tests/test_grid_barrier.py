"""The training kernel's grid barrier (no GPU): its word is one 64-bit object that is only ever accessed whole -- a release and
an acquire of different widths on the same bytes do not synchronise in the PTX memory model -- and counts right."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pink_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_every_access_to_the_barrier_word_has_its_width():
    struct = re.search(r"struct StepCtrl\s*\{(.*?)\}", _source("kernels.cuh"), re.S).group(1)
    assert re.search(r"unsigned long long bar\s*;", struct)
    members = re.findall(r"(\w+)(?:\[\w+\])?\s*;", struct)
    assert members[-1] == "bar"                   # nothing behind it that a wider access could share
    steps, ptx = _source("train_steps.cu"), _source("ptx.cuh")
    uses = re.findall(r"(\w+)\(&a\.ctrl->bar\b", steps)
    assert len(uses) >= 2 and len(uses) == len(re.findall(r"ctrl->bar\b", steps))
    for name in uses:
        body = re.search(r"\b%s\((?:const )?unsigned long long\* p\b.*?\n\}" % name, ptx, re.S).group(0)
        assert re.search(r"\.gpu\.global(?:\.add)?\.u64 ", body), name


def test_arrivals_and_failures_share_the_word():
    assert re.search(r"kBarArrived = 1ull, kBarFailed = 1ull << 32", _source("train_steps.cu"))
    wrap, arrived, failed, blocks = 1 << 64, 1, 1 << 32, 148
    word = wrap - 1                               # memset to 0xFF bytes
    for barrier in range(1, 33):                  # 16 images, two barriers each
        for _ in range(blocks):
            assert (word + 1) % wrap < barrier * blocks
            word = (word + arrived) % wrap
        assert barrier * blocks == (word + 1) % wrap < failed
    word = (word + arrived + failed) % wrap
    assert (word + 1) % wrap >= failed
