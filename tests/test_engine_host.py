"""The engine's host side on the CPU: a child process decodes with tests/cpp/fake_cudart.cpp in the place of the CUDA runtime, whose
kernels do nothing, and looks at what the engine asked the runtime for."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import ctypes as C, os, sys
fake = C.CDLL(os.environ["LD_PRELOAD"])
fake.fake_get.restype = fake.fake_launches.restype = C.c_long
sys.path.insert(0, %r)
import numpy as np
from linmt_b200 import decoder, synth

def put(key, x): fake.fake_set(key.encode(), C.c_long(x))
def get(key): return fake.fake_get(key.encode())
def launches(part): return fake.fake_launches(part.encode())

class refusing:
    "From the n-th request for memory on, all are refused."
    def __init__(self, n): self.n = n
    def __enter__(self): put("refuse_after", self.n); put("refusing", 1)
    def __exit__(self, *a): put("refusing", 0)

def no_memory(call, n):
    "Whether the call fails for memory when its n-th request and all after it are refused."
    try:
        with refusing(n): call()
    except decoder.LinmtError as e:
        assert "failed (4)" in str(e), e      # LINMT_ENOMEM
        return True
    return False

D = synth.ModelDesc(2, 256, 3000, 300, 1)
BLOB = synth.make_blob(D, 1)
OPT = dict(beam=2, max_batch=4, max_src_len=16, max_steps=20)
def make(**kw): return decoder.Decoder(D, [BLOB], **{**OPT, **kw})
def some(n, seed=3): return synth.make_sentences(n, 2, 9, D.Vs, 1.1, seed, lambda s: s + 3)
def words(n, m=2): return [np.arange(3, 3 + m)] * n
""" % ROOT


@pytest.fixture(scope="module")
def child(cuda_lib, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("cpp") / "fake_cudart.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-o", so], check=True)

    def run(body, **env):
        r = subprocess.run([sys.executable, "-c", HEAD + body + "\nassert get('violations') == 0, get('violations')\n"],
                           env={**os.environ, "LD_PRELOAD": so, **env}, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return run


def test_a_refused_request_is_not_reported_again(child):
    """A call, or the creation of a handle, that fails for memory leaves nothing that the next one would fail by."""
    child("""
dec = make()
dec.decode(some(2))
assert no_memory(lambda: dec.decode(some(2), trace=True), 0)
dec.decode(some(2))
n = 0
while no_memory(lambda: make().close(), n):
    dec.decode(some(2))
    n += 1
assert n > 100
dec.close()
assert get("used") == 0, get("used")
""")


def test_one_plane_makes_its_recurrent_products_in_place(child):
    """Apart from the rest of a gate they are another order of sums, which bf16 states show."""
    child("""
for precision, ahead in (("fp32", True), ("bf16", False)):
    before = launches("TcEpiParts")
    dec = make(precision=precision)
    dec.decode(some(2))
    assert (launches("TcEpiParts") > before) == ahead, precision
    dec.close()
""")


def test_a_buffer_that_could_not_grow_is_not_taken_for_the_old_one(child):
    """Calls that fail for memory at each request of theirs, and smaller ones after them: no copy goes to memory that is not there."""
    child("""
def all_refusals(dec, big, small):
    "`big` fails at its first request, its second, ... until it goes through; `small` works after each."
    small()
    n = 0
    while no_memory(big, n):
        small()
        n += 1
    return n
long = synth.make_sentences(4, 12, 16, D.Vs, 1.1, 3, lambda s: 20)
dec = make(nbest=2)
assert all_refusals(dec, lambda: dec.decode(long), lambda: dec.decode(some(1))) > 0
dec.close()
dec = make()
assert all_refusals(dec, lambda: dec.score(long, words(4, 20)), lambda: dec.score(some(1), words(1))) > 0
dec.close()
assert get("used") == 0, get("used")
""")


def test_scoring_fills_its_panels_ahead_of_the_kernels_that_write_them(child):
    """The engine's stream does not wait for a fill of the legacy stream: none of a call's is there."""
    child("""
for kw in (dict(), dict(precision="bf16"), dict(gemm_path="tensor3")):
    dec = make(**kw)
    put("races", 0)
    dec.score(some(3), words(3))
    dec.score(some(4), words(4, 12))       # (longer: the panels are made anew)
    assert get("races") == 0, kw
    dec.close()
""")


def test_a_refused_scoring_workspace_is_not_kept_in_part(child):
    """However often a call fails for memory, the handle holds what one that went through holds."""
    child("""
def held(refusals):
    dec = make(precision=precision)
    empty = get("used")
    for n in refusals:
        no_memory(lambda: dec.score(some(4), words(4, 12)), n)
    dec.score(some(4), words(4, 12))
    mine = get("used") - empty
    dec.close()
    return mine
for precision in ("fp32", "bf16"):
    dec, n = make(precision=precision), 0
    while no_memory(lambda: dec.score(some(4), words(4, 12)), n):
        n += 1
    dec.close()
    assert n > 1
    assert held(list(range(n)) * 3) == held([]), precision
""")


LANES = """
def calls(dec):
    dec.decode(some(18)); dec.score(some(18), words(18, 12)); dec.decode(long); dec.decode(some(2), trace=True)
long = synth.make_sentences(18, 12, 16, D.Vs, 1.1, 3, lambda s: 20)
os.environ["LINMT_LANES"] = "0"
dec = make(); created = get("used"); calls(dec); alone = get("used")
per_call = dec.stats()["sentence_steps"]
dec.close()
del os.environ["LINMT_LANES"]
"""


def test_a_call_goes_through_in_the_memory_that_one_engine_needs(child):
    """Whatever the device has beside that, and whenever the memory gets short: engines beside the handle's own are made of what is
    to spare, and given up where it does not suffice."""
    child(LANES + """
kept = 0
for early in (False, True):
    for extra in range(0, 1200 << 20, 48 << 20):
        dec = make()
        if early:
            dec.decode(some(18))
            assert get("used") > created + (100 << 20), "no lanes made"
        put("limit", max(get("used"), alone) + extra)
        calls(dec)
        calls(dec)
        kept += get("used") > alone
        put("limit", 0)
        dec.close()
        assert get("used") == 0
assert 0 < kept < 50, kept
""")


def test_no_single_refusal_fails_a_call_of_several_batches(child):
    child(LANES + """
n, refused = 1, True
while refused:
    dec = make()
    put("refuse_one", n)
    calls(dec)
    refused = get("refuse_one") == 0
    put("refuse_one", 0)
    assert dec.stats()["sentence_steps"] >= per_call
    calls(dec)
    dec.close()
    n += 1
assert get("used") == 0 and n > 30, n
""")


def test_streams_that_could_not_be_made_are_not_used(child):
    """The encoder's streams and those of ensemble members are made in a call: each refusal fails that one alone, for memory, and no
    kernel runs on the legacy stream."""
    child("""
def ensemble(**kw): return decoder.Decoder(D, [BLOB, synth.make_blob(D, 2)], **{**OPT, **kw})
for new in (lambda: make(gemm_path="tensor3"), ensemble, lambda: ensemble(gemm_path="tensor3")):
    n, more = 0, True
    while more:
        dec = new()
        more = no_memory(lambda: dec.decode(some(2)), n)
        put("legacy", 0)
        dec.decode(some(2))
        assert get("legacy") == 0, n
        dec.close()
        n += 1
    assert n > 4
""")


def test_host_memory_that_runs_out_in_one_of_several_batches(child):
    """Thrown in whichever engine's thread: the call goes through without the further engines; of a handle that has none it fails."""
    child(LANES + """
for n in range(1, 16):
    dec = make()
    put("throw_at", n)
    dec.decode(some(18)); dec.decode(some(18))
    assert get("throw_at") == 0, n
    dec.close()
os.environ["LINMT_LANES"] = "0"
dec = make()
put("throw_at", 3)
assert no_memory(lambda: dec.decode(some(18)), 10**9)
dec.decode(some(18))
dec.close()
""")


def test_a_batch_that_has_its_device_to_itself_runs_as_one_by_itself(child):
    """On several devices with a batch each, and where there is no memory for further engines: the launches of a handle without them.
    (Batches that share a device encode layer by layer, a batch by itself with the layers side by side.)"""
    child("""
D5 = synth.ModelDesc(3, 512, 3000, 300, 1)
B5 = synth.make_blob(D5, 1)
def counted(n, limited=False, **kw):
    dec = decoder.Decoder(D5, [B5], beam=2, max_batch=4, max_src_len=40, max_steps=20, **kw)
    s = synth.make_sentences(n, 24, 30, D5.Vs, 1.1, 3, lambda s: 9)
    dec.decode(synth.make_sentences(1, 24, 30, D5.Vs, 1.1, 3, lambda s: 9))
    if limited: put("limit", get("used") + (200 << 20))
    start = dec.stats()["kernel_launches"]
    dec.decode(s)
    one = dec.stats()["kernel_launches"] - start
    if not kw: dec.score(s, words(n, 5))
    put("limit", 0)
    both = dec.stats()["kernel_launches"] - start
    dec.close()
    return one, both
def alone(*a, **kw):
    os.environ["LINMT_LANES"] = "0"
    c = counted(*a, **kw)
    del os.environ["LINMT_LANES"]
    return c
assert counted(8) != alone(8)                   # (one device: they share it)
assert counted(8, devices=[0, 1]) == alone(8, devices=[0, 1])
assert counted(12, devices=[0, 1, 2, 3]) == alone(12, devices=[0, 1, 2, 3])
put("limit", 0)
got, want = counted(8, limited=True), alone(8, limited=True)
assert got == want, (got, want)
""")


def test_further_engines_are_made_beside_the_first_batches(child):
    """The first call of several batches does not wait for them: its thread asks for what it asks for without them, nothing waits for the
    whole device, and the two make a few requests each (an engine's creation is one)."""
    child("""
same = synth.make_sentences(16, 9, 9, D.Vs, 1.1, 3, lambda s: s + 3)        # four batches of one size
def asked(call):
    put("requests", 0); put("requests_beside", 0); put("device_waits", 0)
    call()
    assert get("device_waits") == 0
    return get("requests")
for entry in (lambda dec: dec.decode(same), lambda dec: dec.score(same, words(16, 12))):
    os.environ["LINMT_LANES"] = "0"
    dec = make()
    alone = asked(lambda: entry(dec))
    dec.close()
    del os.environ["LINMT_LANES"]
    dec = make()
    assert asked(lambda: entry(dec)) <= alone          # (less where the others have taken every batch)
    assert 0 < get("requests_beside") <= 2 * 12
    dec.close()
""")


def test_engines_of_a_call(child):
    """Three up to 64 rows, and beyond where L2 holds a step's weights, else two; one from 513 rows on, for one batch, for an ensemble, and
    while kernels are timed.  (An engine makes one stream; sources as short as these are encoded on that.)"""
    child("""
def engines(n, timing=False, **kw):
    put("streams", 0)
    dec = decoder.Decoder(d, blobs, max_src_len=16, max_steps=4, **kw)
    dec.set_kernel_timing(timing)
    dec.decode(synth.make_sentences(n, 2, 9, d.Vs, 1.1, 3, lambda s: 3))
    dec.decode(synth.make_sentences(n, 2, 9, d.Vs, 1.1, 3, lambda s: 3))
    dec.close()
    return get("streams")
d, blobs = D, [BLOB]
assert engines(31, beam=2, max_batch=4) == 3
assert engines(8, beam=2, max_batch=4) == 2
assert engines(4, beam=2, max_batch=4) == 1
assert engines(31, timing=True, beam=2, max_batch=4) == 1
assert engines(200, beam=8, max_batch=64) == 3
assert engines(200, beam=9, max_batch=57) == 1          # 513 rows
d = synth.ModelDesc(5, 768, 3000, 300, 1)               # 104 MB a step in fp32 precision, of 126 MB of L2
blobs = [synth.make_blob(d, 1)]
assert engines(100, beam=2, max_batch=32) == 3
assert engines(100, beam=2, max_batch=33) == 2
assert engines(100, beam=2, max_batch=33, precision="bf16") == 3
""")


def test_an_error_in_a_further_engine_is_the_call_s(child):
    """A sentence that cannot be decoded, in whichever of the batches: the code and the text that one engine gives, and a handle that
    goes on working."""
    child("""
def bad(i, what):
    s = some(18)
    lens = s.lengths().copy()
    lens[i] = 0 if what == "empty" else 17
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return synth.Sentences(np.full(int(off[-1]), 5, np.int32), off, np.full(18, 5, np.int32))
def error(call):
    try:
        call()
    except decoder.LinmtError as e:
        return str(e)
dec = make()
for i in range(18):
    for what, code in (("empty", "(1): empty source"), ("long", "(5): source sentence longer")):
        for call in (lambda: dec.decode(bad(i, what)), lambda: dec.score(bad(i, what), words(18))):
            assert code in str(error(call)), (i, error(call))
        dec.decode(some(18)); dec.score(some(18), words(18))
dec.close()
""")


def test_layers_side_by_side_of_more_words_than_the_panels_hold(child):
    """40 sentences of 500 words are 20000 rows, in two chunks of 409 and 91 positions: the layers side by side (512 units) make an input
    product for every eight of them, layer by layer (448 units) one a chunk."""
    child("""
def launched(H, n, longest):
    d = synth.ModelDesc(2, H, 3000, 300, 1)
    dec = decoder.Decoder(d, [synth.make_blob(d, 1)], beam=2, max_batch=n, max_src_len=longest, max_steps=4)
    before = dec.stats()["kernel_launches"]
    dec.score(synth.make_sentences(n, longest, longest, d.Vs, 1.1, 3, lambda s: 3), words(n, 1))
    count = dec.stats()["kernel_launches"] - before
    dec.close()
    return count
assert launched(512, 40, 500) - launched(448, 40, 500) == 2 * (52 + 12 - 2)
assert launched(512, 2, 20) - launched(448, 2, 20) == 2 * (3 - 1)
assert launched(512, 2, 19) == launched(448, 2, 19)
""")


def test_rows_whose_recurrent_products_are_made_ahead(child):
    """Up to 60, of few or narrow layers; up to 48 of more than 2 Mi layers x units x units; up to 32 of one slot each."""
    child("""
def ahead(dec, n, beam):
    before = launches("TcEpiParts")
    dec.decode(synth.make_sentences(n, 4, 4, D.Vs, 1.1, 3, lambda s: 5))      # (all end together)
    return launches("TcEpiParts") > before
for L, H, most in ((2, 256, 60), (3, 768, 60), (3, 840, 48)):
    d = synth.ModelDesc(L, H, 3000, 300, 1)
    blob = synth.make_blob(d, 1)
    for beam in (4, 1):
        dec = decoder.Decoder(d, [blob], beam=beam, max_batch=70 // beam, max_src_len=16, max_steps=8)
        bound = (32 if beam == 1 else most) // beam
        assert ahead(dec, bound, beam) and not ahead(dec, bound + 1, beam), (L, H, beam)
        dec.close()
""")


def test_host_memory_that_runs_out_between_two_launches(child):
    """Wherever in a call, on a layer's or a member's stream among them: that call fails for memory, and the next one runs as ever."""
    child("""
D5 = synth.ModelDesc(3, 512, 3000, 300, 1)
long = synth.make_sentences(2, 20, 20, D5.Vs, 1.1, 3, lambda s: 3)
def ensemble(): return decoder.Decoder(D, [BLOB, synth.make_blob(D, 2)], **OPT)
def side_by_side(): return decoder.Decoder(D5, [synth.make_blob(D5, 1)], beam=2, max_batch=4, max_src_len=20, max_steps=8)
for new, s in ((side_by_side, long), (lambda: make(gemm_path="tensor3"), some(2)), (ensemble, some(2))):
    dec = new()
    dec.decode(s)
    before = dec.stats()["kernel_launches"]
    dec.decode(s)
    count = dec.stats()["kernel_launches"] - before
    assert count > 20
    for n in list(range(1, count, 3)) + [count]:
        put("throw_launch", n)
        assert no_memory(lambda: dec.decode(s), 10**9), n
        before = dec.stats()["kernel_launches"]
        dec.decode(s)
        assert dec.stats()["kernel_launches"] - before == count, n
    dec.close()
assert get("used") == 0
""")
