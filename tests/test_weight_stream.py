"""The rule that makes a step's weights a stream, on the CPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
L2 = 126 << 20


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cpp") / "weight_stream_main")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "linmt_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "weight_stream_main.cpp"), "-o", out], check=True)

    def run(layers, hp, vp, members, planes, vocab_planes, scoring, rows, l2=L2):
        line = f"{layers} {hp} {vp} {members} {planes} {vocab_planes} {l2} {scoring} {rows}\n"
        n, stream = subprocess.run([out], input=line, capture_output=True, text=True, check=True).stdout.split()
        return int(n), stream == "1"
    return run


def test_a_scoring_step_reads_no_vocabulary(ask):
    for members, planes, vocab_planes in ((1, 1, 1), (1, 2, 1), (4, 2, 2)):
        scored, decoded = (ask(4, 1024, 30080, members, planes, vocab_planes, s, 1)[0] for s in (1, 0))
        assert scored == members * planes * 2 * 36 * 1024 * 1024
        assert decoded - scored == members * vocab_planes * 2 * 30080 * 1024


@pytest.mark.parametrize("model,decoding,scoring_few,scoring_many", [
    ((4, 1024, 30080, 1, 1, 1), True, False, True),        # bf16: 75 MB recurrent, 137 MB with the vocabulary
    ((4, 1024, 30080, 1, 2, 1), True, True, True),         # fp32: 151 MB recurrent
    ((2, 128, 1024, 1, 2, 1), False, False, False),
    ((2, 512, 100096, 1, 1, 1), True, False, True),
    ((4, 1024, 30080, 2, 1, 1), True, True, True),         # two members in bf16
])
def test_what_is_a_stream(ask, model, decoding, scoring_few, scoring_many):
    for rows in (1, 64, 65, 256, 1536):
        assert ask(*model, 0, rows)[1] == decoding
        assert ask(*model, 1, rows)[1] == (scoring_few if rows <= 64 else scoring_many)
