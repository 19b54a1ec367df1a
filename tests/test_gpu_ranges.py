"""GPU tests at the far ends of what a handle takes: sizes and batches that no named configuration reaches."""
import numpy as np
import pytest

from linmt_b200 import synth
from parity import RTOL_FP32, compare_forced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,H,counts", [(2, 1600, (64, 49, 48)), (1, 2432, (1, 17, 64))])
def test_hidden_sizes_beyond_the_few_rows_kernel(cuda_lib, L, H, counts):
    """The weight-streaming kernel declines K slices of more than three k-blocks per leading accumulator: a recurrent
    product of 1600 units from 49 sentences on, of 2432 for any number.  The encoder's per-position products then run
    elsewhere, on rows in the middle of a panel.  Decode (forced) and scores against the CUDA-core path."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(L, H, 100, 60, 1)
    # Bound of the comparison: a CUDA-core logit is within 4e-6 of its terms' absolute sum, 0.04 x 0.5 x 2432 = 49, of the
    # exact one, 2e-4; log-probabilities of 100 words are near -4.6, 1e-4 of which is 4.6e-4.  (The peaked family's output
    # weights are 30 times as large, and the bound 6e-3 against rows of 40: 1.3e-4 relative was seen.)
    blob = synth.make_blob(d, 3)
    kw = dict(beam=2, max_batch=64, max_src_len=8, max_steps=12, cp_beta=0.0)
    tc = decoder.Decoder(d, [blob], **kw)
    ref = decoder.Decoder(d, [blob], gemm_path="simt", **kw)
    for n in counts:
        sents = synth.make_sentences(n, 2, 7, d.Vs, 1.1, n, lambda s: s + 2)
        r = ref.decode(sents, trace=True)
        e = tc.decode(sents, trace=True, force=r)
        worst, bad, skipped, compared = compare_forced(e, r, sents.steps, src_len=sents.lengths())
        assert worst <= RTOL_FP32 and bad == 0 and skipped <= 0.1 * (skipped + compared), (n, worst, bad, skipped, compared)
        rng = np.random.default_rng(n)
        targets = [rng.integers(3, d.V, size=int(m)) for m in rng.integers(1, 10, size=n)]
        a, b = tc.score(sents, targets), ref.score(sents, targets)
        scale = np.abs(b[1]).max(axis=1, keepdims=True)
        assert (np.abs(a[1] - b[1]) <= RTOL_FP32 * scale).all(), (n, float((np.abs(a[1] - b[1]) / scale).max()))
    tc.close(); ref.close()


@pytest.mark.parametrize("n", [1, 75])     # two rows, a CTA of 1024 threads each; 150 rows, CTAs of 512 threads
def test_global_attention_over_long_sources(oracle, cuda_lib, n):
    """A handle for sources of up to 12,250 words: with a row's vector, its scores pass 48 KB of shared memory."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(1, 64, 200, 100, 1)
    blob = synth.make_blob(d, 8)
    rng = np.random.default_rng(n)
    lens = np.concatenate([[12250], rng.integers(2, 20, size=n - 1)]).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    sents = synth.Sentences(synth.zipf_ids(rng, int(off[-1]), 1, d.Vs, 1.1), off, np.full(n, 4, np.int32))
    kw = dict(beam=2, attention="global_general", cp_beta=0.0, min_ratio=0.0)
    o = oracle.decode(d, [blob], sents, trace=True, **kw)
    dec = decoder.Decoder(d, [blob], max_batch=n, max_src_len=12250, max_steps=8, **kw)
    e = dec.decode(sents, trace=True, force=o)
    worst, bad, skipped, compared = compare_forced(e, o, sents.steps, src_len=sents.lengths())
    assert worst <= RTOL_FP32 and bad == 0 and skipped == 0, (worst, bad, skipped, compared)
    dec.close()


@pytest.mark.parametrize("attention", ["local_p_general", "global_general"])
def test_batches_of_other_lengths_on_one_handle(cuda_lib, attention):
    """The source lengths of a batch replace those of the batch before while kernels overlap at their boundaries: results
    on a handle that has just decoded longer or shorter sentences are those of a fresh handle, to the bit."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(2, 128, 500, 300, 1)
    blob = synth.make_blob(d, 5)
    kw = dict(beam=3, attention=attention, print_info=True, cp_beta=0.2, max_batch=8, max_src_len=64, max_steps=64)
    batches = [synth.make_sentences(n, lo, hi, d.Vs, 1.1, n, lambda s: 12) for n, lo, hi in ((8, 50, 60), (8, 1, 3), (3, 30, 64), (8, 20, 25))]
    fresh = []
    for b in batches:
        dec = decoder.Decoder(d, [blob], **kw)
        fresh.append(dec.decode(b, want_align=True))
        dec.close()
    kept = decoder.Decoder(d, [blob], **kw)
    for i in (0, 1, 2, 3, 1, 0, 3, 2):
        out = kept.decode(batches[i], want_align=True)
        for key in ("tok", "len", "score", "vit", "align"):
            assert np.array_equal(out[key], fresh[i][key]), (i, key)
    kept.close()
