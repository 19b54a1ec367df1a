"""The rule that chooses the encoder's form, on the CPU: against measured times, and at its edges."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def form(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cpp") / "encoder_form_main")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "linmt_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "encoder_form_main.cpp"), "-o", out], check=True)

    def ask(layers, hp, n, words, members=1, split=1):
        r = subprocess.run([out], input=f"{layers} {hp} {members} {split} {n} {words}\n", capture_output=True, text=True, check=True)
        return r.stdout.strip()
    return ask


# ms of a call with two decoder steps on a B200, fp32 weights: layers, hidden size, sentences, words, layer by layer, pipelined,
# position by position
MEASURED = [
    (2, 128, 33, 32, 0.606, 0.549, 0.646), (2, 128, 64, 96, 1.806, 1.078, 1.578), (2, 512, 48, 64, 1.017, 1.167, 1.492),
    (2, 1024, 33, 32, 0.755, 0.968, 1.116), (2, 1024, 48, 64, 1.395, 1.623, 1.984), (2, 1024, 64, 32, 0.942, 1.016, 1.161),
    (3, 256, 48, 32, 0.808, 0.672, 0.770), (3, 1024, 33, 32, 1.053, 1.328, 1.347), (3, 1024, 48, 64, 1.985, 2.126, 2.433),
    (3, 1024, 64, 96, 3.367, 3.008, 3.525), (4, 512, 33, 96, 2.560, 1.970, 2.618), (4, 768, 33, 32, 1.159, 1.339, 1.170),
    (4, 1024, 33, 32, 1.359, 1.568, 1.528), (4, 1024, 48, 32, 1.463, 1.582, 1.554), (4, 1024, 48, 96, 3.727, 3.275, 3.978),
    (4, 1024, 64, 64, 3.103, 2.524, 2.775), (5, 1024, 33, 32, 1.646, 2.036, 1.749), (5, 1024, 64, 96, 5.484, 4.373, 4.596),
    (4, 1280, 48, 96, 6.333, 4.537, 5.549), (2, 512, 96, 32, 0.874, 0.771, 0.920), (3, 768, 128, 64, 3.182, 1.934, 2.067),
    (4, 768, 96, 32, 1.857, 1.468, 1.328), (4, 1024, 128, 32, 2.631, 1.893, 1.743), (4, 1024, 96, 96, 5.681, 3.686, 4.347),
    (5, 512, 96, 32, 1.944, 1.357, 1.195), (5, 512, 128, 96, 6.051, 2.679, 2.894), (5, 1024, 128, 32, 3.260, 2.400, 1.993),
]


@pytest.mark.parametrize("layers,hp,n,words,by_layers,pipelined,wavefront", MEASURED)
def test_chosen_form_is_no_slower_than_the_plain_one(form, layers, hp, n, words, by_layers, pipelined, wavefront):
    """The plain form is layer by layer up to 64 sentences, position by position beyond.  Bound: two runs of one form differ by
    up to 3 %."""
    plain = by_layers if n <= 64 else wavefront
    taken = {"layers": by_layers, "pipelined": pipelined, "wavefront": wavefront}[form(layers, hp, n, words)]
    assert taken <= 1.03 * plain and taken <= 1.03 * min(plain, pipelined), (taken, plain, pipelined)


def test_edges_of_the_rule(form):
    for words in (1, 31, 32, 100, 5000):
        for n in (1, 32, 33, 64, 65, 128, 129, 500):
            plain = "layers" if n <= 64 else "wavefront"
            assert form(4, 1024, n, words, split=0) == plain          # bf16: the order of sums that it has
            assert form(4, 1024, n, words, members=2) == plain        # members run side by side
            assert form(1, 1024, n, words) == plain                   # no layers to run side by side
            if n <= 32 or n > 128 or words < 32:
                assert form(4, 512, n, words) == plain
            elif words >= 100:
                assert form(4, 512, n, words) == "pipelined"          # however long: in chunks


# ms of the encoder and two scored words, fp32 weights: layers, hidden size, sentences, words, layer by layer, layers side by side
BESIDE = [
    (2, 512, 1, 20, 0.333, 0.348), (2, 512, 1, 32, 0.437, 0.454), (2, 512, 1, 50, 0.588, 0.517), (2, 512, 4, 20, 0.344, 0.330),
    (2, 512, 16, 32, 0.474, 0.464), (4, 512, 1, 24, 0.629, 0.641), (4, 512, 1, 50, 1.088, 0.877), (5, 768, 1, 20, 0.732, 0.690),
    (2, 1024, 1, 20, 0.414, 0.411), (2, 1024, 48, 24, 0.732, 0.680), (2, 1024, 64, 20, 0.726, 0.745), (2, 1024, 64, 50, 1.376, 1.415),
    (4, 1024, 1, 20, 0.709, 0.660), (4, 1024, 48, 20, 1.125, 0.979), (4, 1024, 64, 20, 1.244, 1.260), (5, 1024, 64, 20, 1.498, 1.524),
    (4, 512, 64, 20, 0.879, 0.771), (5, 768, 64, 20, 1.297, 1.238), (3, 1280, 64, 20, 1.656, 1.418),
]


@pytest.fixture(scope="module")
def beside(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cpp") / "encoder_beside_main")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "linmt_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "encoder_beside_main.cpp"), "-o", out], check=True)

    def ask(cases):
        r = subprocess.run([out], input="".join("%d %d %d %d %d %d %d\n" % c for c in cases), capture_output=True, text=True, check=True)
        return [tuple(x == "1" for x in line.split()) for line in r.stdout.splitlines()]
    return ask


@pytest.mark.parametrize("layers,hp,n,words,turn,side", BESIDE)
def test_layers_side_by_side_where_that_is_no_slower(beside, layers, hp, n, words, turn, side):
    """Bound: two runs of one form differ by up to 1 %."""
    taken = side if beside([(layers, hp, 1, 1, n, words, 0)])[0][0] else turn
    assert taken <= 1.01 * min(turn, side)


def test_one_plane_is_encoded_in_one_order(beside):
    """Layers side by side, and products that leave room for the next one, add in another order: neither in one plane."""
    asked = [(layers, hp, members, split, n, words, shared) for layers in (1, 2, 5) for hp in (128, 448, 512, 1024) for members in (1, 2)
             for split in (0, 1) for n in (1, 32, 33, 48, 49, 64) for words in (1, 19, 20, 39, 40, 100) for shared in (0, 1)]
    for a, (side, room) in zip(asked, beside(asked), strict=True):
        layers, hp, members, split, n, words, shared = a
        if not split:
            assert not side and not room, a
        if members > 1 or layers == 1 or hp < 512 or shared or words < 20:
            assert not side, a
        assert room == (split and n <= (48 if side else 32)), a
