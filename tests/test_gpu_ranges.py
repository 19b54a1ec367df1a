"""GPU tests at the far ends of what a handle takes: sizes and batches that no named configuration reaches."""
import os

import numpy as np
import pytest

from linmt_b200 import synth
from parity import RTOL_FP32, compare_forced, hyps

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
    blob = synth.make_blob(d, 8, family="peaked")
    rng = np.random.default_rng(n)
    lens = np.concatenate([[12250], rng.integers(2, 20, size=n - 1)]).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    sents = synth.Sentences(synth.zipf_ids(rng, int(off[-1]), 1, d.Vs, 1.1), off, np.full(n, 4, np.int32))
    kw = dict(beam=2, attention="global_general", cp_beta=0.0, min_ratio=0.0, print_info=1)
    o = oracle.decode(d, [blob], sents, trace=True, **kw)
    dec = decoder.Decoder(d, [blob], max_batch=n, max_src_len=12250, max_steps=8, **kw)
    e = dec.decode(sents, trace=True, force=o, want_align=True)
    worst, bad, skipped, compared = compare_forced(e, o, sents.steps, src_len=sents.lengths())
    assert worst <= RTOL_FP32 and bad == 0 and skipped == 0, (worst, bad, skipped, compared)
    # every position's weight (a source of 12,250 words has 8e-5 on each): a score is a 64-term fp32 sum, its exponential
    # and the sum of all of them good to a few 1e-6
    assert hyps(e, 0) == hyps(o, 0)
    for i in range(n):
        if hyps(e, i) == hyps(o, i):
            m, S = int(o["len"][i, 0]), int(lens[i])
            np.testing.assert_allclose(e["align"][i, 0, :m, :S], o["align"][i, 0, :m, :S], rtol=5e-5, atol=1e-10)
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


def _with_env(env, make):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        return make()
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v


@pytest.mark.parametrize("attention", ["local_p_general", "global_dot"])
def test_bf16_batch_of_more_than_1024_rows(oracle, cuda_lib, attention):
    """128 sentences x 12 beams in bf16: 1536 rows, whose gate products run as persistent CTA pairs until 1024 are left,
    behind the encoder of more than 64 sentences.  Against the oracle, forced; and the same bits without pairs, since the
    same products accumulate in the same order.

    Bound: where two implementations sum in different orders, a rounding of the state may fall to the other bf16
    neighbour, a step of 2^-9.  Logits are 128-term sums that spread by 0.07: 2^-9 of that is 1.4e-4 if every element of
    one state parts, ten states (layers, context, attentional state, the steps before) 4e-4 in the mean square, ten times
    that for the far tail.  (Seen: median 2.6e-4, 1.9e-3 at 99.9 %.  Another sentence's rows differ by 6e-2.)"""
    from linmt_b200 import decoder
    c = synth.configs()["C1"]
    blob = c.blobs(family="peaked")[0]
    sents = synth.make_sentences(128, 3, 20, c.desc.Vs, 1.1, 5, lambda s: min(s + 2, 16))
    kw = dict(beam=12, precision="bf16", attention=attention, cp_beta=0.0, min_ratio=0.0)
    o = oracle.decode(c.desc, [blob], sents, trace=True, **kw)

    def run():
        dec = decoder.Decoder(c.desc, [blob], max_batch=128, max_src_len=32, max_steps=32, **kw)
        forced, before = dec.decode(sents, trace=True, force=o), dec.stats()["pair_launches"]
        free = dec.decode(sents)
        dec.close()
        return forced, free, before

    forced, free, pairs = run()
    # a gate launch of every layer in every step of more than 1024 rows
    wide = sum(1 for t in range(int(sents.steps.max()) + 1) if 12 * int((sents.steps >= t).sum()) > 1024)
    assert wide >= 3 and pairs >= wide * c.desc.L
    err = np.concatenate([np.abs(forced["cand_logp"][i, t, :(1 if t == 0 else None)] - o["cand_logp"][i, t, :(1 if t == 0 else None)]).ravel()
                          for i in range(sents.n) for t in range(int(sents.steps[i]))])
    assert (err <= 4e-3).mean() >= 0.999 and err.max() <= 1.2e-2, (float((err <= 4e-3).mean()), float(np.median(err)), float(err.max()))
    forced1, free1, pairs1 = _with_env({"LINMT_TC_PAIR": "0"}, run)
    assert pairs1 == 0
    for a, b, keys in ((forced, forced1, ("cand_tok", "cand_logp", "final_logp")), (free, free1, ("tok", "len", "score"))):
        for key in keys:
            assert a[key].tobytes() == b[key].tobytes(), key


def test_full_size_gate_products_on_persistent_pairs(cuda_lib):
    """The same at the full model size, where a product's 32 k-blocks go round the ring several times and a pair walks over
    several tiles: 100 sentences x 12 beams, the bits of the one-tile kernels."""
    from linmt_b200 import decoder
    c = synth.configs()["C2"]
    blob = c.blobs()[0]
    sents = synth.make_sentences(100, 2, 8, c.desc.Vs, 1.1, 5, lambda s: 5)

    def run():
        dec = decoder.Decoder(c.desc, [blob], beam=12, precision="bf16", max_batch=100, max_src_len=8, max_steps=8, cp_beta=0.0)
        out = dec.decode(sents, trace=True)
        pairs = dec.stats()["pair_launches"]
        dec.close()
        return out, pairs

    a, pairs = run()
    b, none = _with_env({"LINMT_TC_PAIR": "0"}, run)
    assert pairs >= 6 * c.desc.L and none == 0
    for key in ("cand_tok", "cand_logp", "final_logp", "tok", "score"):
        assert a[key].tobytes() == b[key].tobytes(), key


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("n,longest", [(64, 300), (63, 600), (3, 6000)])
def test_encoder_in_chunks_of_positions(cuda_lib, precision, n, longest):
    """The layer-by-layer encoder takes 16,384 rows (positions x sentences) at a time: longer sources continue from the
    states the chunk before ended with, here after an even and an odd number of positions and more than once.  Against the
    encoder that runs position by position (the CUDA-core path in fp32; without the few-rows kernel in bf16)."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(2, 96, 300, 200, 1)
    blob = synth.make_blob(d, 6, family="peaked")
    rng = np.random.default_rng(n)
    lens = np.concatenate([[longest, longest - 1], rng.integers(1, longest, size=n - 2)]).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    sents = synth.Sentences(synth.zipf_ids(rng, int(off[-1]), 1, d.Vs, 1.1), off, np.full(n, 6, np.int32))
    kw = dict(beam=2, precision=precision, max_batch=n, max_src_len=longest, max_steps=8, cp_beta=0.0, min_ratio=0.0)
    if precision == "fp32":
        ref = decoder.Decoder(d, [blob], gemm_path="simt", **kw)
    else:
        ref = _with_env({"LINMT_TC_ROWS": "0"}, lambda: decoder.Decoder(d, [blob], **kw))
    r = ref.decode(sents, trace=True)
    dec = decoder.Decoder(d, [blob], **kw)
    e = dec.decode(sents, trace=True, force=r)
    if precision == "fp32":
        worst, bad, skipped, compared = compare_forced(e, r, sents.steps, src_len=sents.lengths())
        assert worst <= RTOL_FP32 and bad == 0 and skipped <= 0.1 * (skipped + compared), (worst, bad, skipped, compared)
    else:
        a, b = e["cand_logp"][:, 1:], r["cand_logp"][:, 1:]
        assert np.abs(a - b).max() <= 1.2e-2, float(np.abs(a - b).max())      # (as for 1536 rows above)
    ref.close(); dec.close()


@pytest.mark.parametrize("members,mode", [(5, "prob_mean"), (8, "logprob_mean")])
def test_ensembles_of_more_than_four(oracle, cuda_lib, members, mode):
    """The combining softmax keeps four members' loads in flight and takes the others in turn."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(1, 64, 1003, 300, 1)
    blobs = [synth.make_blob(d, 40 + m, family="peaked") for m in range(members)]
    sents = synth.make_sentences(5, 2, 12, d.Vs, 1.1, 3, lambda s: s + 3)
    kw = dict(beam=6, nbest=2, cp_beta=0.0, ensemble=mode)
    o = oracle.decode(d, blobs, sents, trace=True, **kw)
    dec = decoder.Decoder(d, blobs, max_batch=5, max_src_len=16, max_steps=20, **kw)
    e = dec.decode(sents, trace=True, force=o)
    worst, bad, skipped, compared = compare_forced(e, o, sents.steps, src_len=sents.lengths())
    assert worst <= RTOL_FP32 and bad == 0 and skipped <= 0.1 * (skipped + compared), (worst, bad, skipped, compared)
    dec.close()


@pytest.mark.parametrize("members,precision", [(1, "fp32"), (1, "bf16"), (2, "fp32")])
def test_rows_of_equal_logits(oracle, cuda_lib, members, precision):
    """All-zero weights: every class ties, more of them than the candidate lists hold, and the lowest ids win."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(1, 64, 3000, 50, 1)
    blobs = [np.zeros(synth.blob_floats(d), np.float32)] * members
    sents = synth.make_sentences(3, 2, 6, d.Vs, 1.1, 3, lambda s: s + 1)
    kw = dict(beam=4, cp_beta=0.0, precision=precision)
    o = oracle.decode(d, blobs, sents, trace=True, **kw)
    dec = decoder.Decoder(d, blobs, max_batch=3, max_src_len=8, max_steps=10, **kw)
    e = dec.decode(sents, trace=True)
    for i in range(sents.n):
        T = int(sents.steps[i])
        assert (e["cand_tok"][i, 0, 0] == np.arange(5)).all() and (e["cand_tok"][i, 1:T] == np.arange(5)).all()
        np.testing.assert_allclose(e["cand_logp"][i, 1:T], -np.log(3000.0), rtol=1e-6)
        assert (e["surv_tok"][i, :T] == o["surv_tok"][i, :T]).all() and (e["surv_parent"][i, :T] == o["surv_parent"][i, :T]).all()
    dec.close()


@pytest.mark.parametrize("steps", [300, 1500, 5900])     # 8 warps, 1 warp, and back-pointers that stay in global memory
def test_finalisation_of_long_hypotheses(oracle, cuda_lib, steps):
    """n-best lists with alignments and coverage penalty of hypotheses so long that fewer warps, and then no copy of the
    back-pointers, fit the shared memory of the finalisation."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(1, 32, 60, 50, 1)
    blob = synth.make_blob(d, 9, family="peaked")
    sents = synth.make_sentences(2, 9, 12, d.Vs, 1.1, 3, lambda s: steps if s > 10 else 7)
    sents.steps[:] = [steps, 7]
    kw = dict(beam=3, nbest=3, cp_beta=0.2, min_ratio=0.0, print_info=1)
    o = oracle.decode(d, [blob], sents, trace=True, **kw)
    dec = decoder.Decoder(d, [blob], max_batch=2, max_src_len=16, max_steps=steps, **kw)
    e = dec.decode(sents, trace=True, force=o, want_align=True)
    assert (e["len"] == o["len"]).all()
    for i in range(2):
        S = int(sents.lengths()[i])
        for q in range(3):
            n = int(o["len"][i, q])
            assert hyps(e, i, q) == hyps(o, i, q)
            assert (e["vit"][i, q, :n] == o["vit"][i, q, :n]).mean() >= 0.999
            assert abs(e["score"][i, q] - o["score"][i, q]) <= RTOL_FP32 * abs(o["score"][i, q])
            np.testing.assert_allclose(e["align"][i, q, :n, :S], o["align"][i, q, :n, :S], rtol=2e-4, atol=1e-6)
    dec.close()


@pytest.mark.parametrize("beam", [4, 7, 8, 15, 16, 17, 31])     # up to 64 candidates, two firsts of a row, one first
@pytest.mark.parametrize("n,family,diversity", [(2, "peaked", 0.0), (60, "peaked", 0.5), (3, "zero", 0.0)])    # 1024 and 256 threads; ties
def test_selection_from_the_candidates_of_a_step(cuda_lib, beam, n, family, diversity):
    """A step's survivors follow from its candidates: score descending, then beam, then word; START is skipped, EOS leaves
    without taking a slot.  Recomputed from the engine's own candidates in fp32 and in its order of operations (the product with a diversity of one half is exact): no tolerance."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(1, 64, 1000, 100, 1)
    blob = synth.make_blob(d, 5, family="peaked") if family == "peaked" else np.zeros_like(synth.make_blob(d, 5))
    sents = synth.make_sentences(n, 2, 6, d.Vs, 1.1, 9, lambda s: 8)
    dec = decoder.Decoder(d, [blob], beam=beam, max_batch=n, max_src_len=8, max_steps=8, cp_beta=0.0, diversity=diversity)
    e, k, f = dec.decode(sents, trace=True), dec.k, np.float32
    dec.close()
    assert k == beam
    for i in range(n):
        score = np.zeros(k, f)
        for t in range(8):
            cand = []
            for b in range(1 if t == 0 else k):
                for q in range(k + 1):
                    v, lp = int(e["cand_tok"][i, t, b, q]), e["cand_logp"][i, t, b, q]
                    cand.append((-((lp + score[b]) - f(q + 1) * f(diversity)), b, v))
            want = [(v, b, -s) for s, b, v in sorted(cand) if v not in (0, 1)][:k]
            want += [(2, 0, f(-1e30))] * (k - len(want))       # fewer that survive than slots
            got = list(zip(e["surv_tok"][i, t].tolist(), e["surv_parent"][i, t].tolist(), e["surv_score"][i, t]))
            assert got == want, (i, t)
            score = e["surv_score"][i, t].copy()


@pytest.mark.parametrize("attention", ["local_p_general", "global_general", "global_dot"])
@pytest.mark.parametrize("L,H,n,precision", [(1, 64, 1, "fp32"), (3, 250, 70, "fp32"), (2, 512, 150, "bf16")])   # few rows, one tile, two
def test_rows_that_continue_themselves_take_turns_in_two_panels(cuda_lib, attention, L, H, n, precision):
    """Greedy search and scoring leave a step's states where the next step reads them; a forced search copies them through
    its parents.  The products are the same, so log-probabilities are the same bits."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(L, H, 400, 300, 1)
    blob = synth.make_blob(d, 7, family="peaked")
    sents = synth.make_sentences(n, 1, 9, d.Vs, 1.1, 4, lambda s: s + 3)
    dec = decoder.Decoder(d, [blob], beam=1, max_batch=n, max_src_len=16, max_steps=16, cp_beta=0.0, attention=attention, precision=precision)
    free = dec.decode(sents, trace=True)
    forced = dec.decode(sents, trace=True, force=free)
    for key in ("cand_tok", "cand_logp", "final_logp"):
        assert free[key].tobytes() == forced[key].tobytes(), key
    targets = [free["surv_tok"][i, :s, 0] for i, s in enumerate(sents.steps)]
    total, per_token = dec.score(sents, targets)
    dec.close()
    for i, s in enumerate(sents.steps):      # the chosen word is a candidate of its step, unless that is START or EOS before it
        t = np.arange(s)
        hit = (free["cand_tok"][i, t, 0] == free["surv_tok"][i, t, 0][:, None])
        want = np.where(hit, free["cand_logp"][i, t, 0], 0).sum(axis=1)
        scale = np.maximum(1, np.abs(free["cand_logp"][i, t, 0]).max(axis=1))
        tol = (2e-2 if precision == "bf16" else RTOL_FP32) * scale       # scoring multiplies other row counts: sums in another order
        assert (np.abs(per_token[i, :s] - want) <= tol)[hit.any(axis=1)].all(), i


@pytest.mark.parametrize("n,longest", [(33, 32), (64, 45), (65, 33), (128, 40)])     # a last stretch of 8, 5, 1 and 8 positions
def test_encoder_layers_side_by_side(cuda_lib, n, longest):
    """Batches of 33 to 128 sentences of 32 and more words in fp32 precision encode with the layers a few positions behind each
    other; with LINMT_TC_ROWS=0 they do so position by position.  Scores of both agree to the sums' rounding."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(3, 128, 300, 200, 1)
    blob = synth.make_blob(d, 11, family="peaked")
    sents = synth.make_sentences(n, 1, longest, d.Vs, 1.1, 6, lambda s: 4)
    lens = sents.lengths()
    assert lens.max() >= 32
    kw = dict(beam=2, max_batch=n, max_src_len=48, max_steps=8, cp_beta=0.0)
    rng = np.random.default_rng(n)
    targets = [rng.integers(3, d.V, size=int(m)) for m in rng.integers(1, 7, size=n)]
    dec = decoder.Decoder(d, [blob], **kw)
    ref = _with_env({"LINMT_TC_ROWS": "0"}, lambda: decoder.Decoder(d, [blob], **kw))
    a, again, b = dec.score(sents, targets), dec.score(sents, targets), ref.score(sents, targets)
    dec.close(); ref.close()
    assert np.array_equal(a[1], again[1])
    scale = np.maximum(1, np.abs(b[1]).max(axis=1, keepdims=True))
    assert (np.abs(a[1] - b[1]) <= RTOL_FP32 * scale).all(), float((np.abs(a[1] - b[1]) / scale).max())


@pytest.mark.parametrize("hidden", [128, 500])
@pytest.mark.parametrize("n,longest", [(33, 496), (33, 497), (40, 1000), (64, 256), (64, 257), (100, 200)])     # 16,384 rows, just more, three chunks
def test_encoder_of_long_sources_takes_chunks(cuda_lib, n, longest, hidden):
    """33 and more sentences so long that the layers' panels do not hold all positions are encoded in chunks, in whichever form
    reads half of a layer's weights per position, and not position by position: that is told from the launches, L a position
    against L + 1.  Scores agree to the sums' rounding."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(2, hidden, 300, 200, 1)
    blob = synth.make_blob(d, 11, family="peaked")
    rng = np.random.default_rng(n)
    lens = np.concatenate([[longest, longest - 1], rng.integers(1, longest, size=n - 2)]).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    sents = synth.Sentences(synth.zipf_ids(rng, int(off[-1]), 1, d.Vs, 1.1), off, np.full(n, 1, np.int32))
    targets = [rng.integers(3, d.V, size=int(m)) for m in rng.integers(1, 4, size=n)]
    kw = dict(beam=1, max_batch=n, max_src_len=longest, max_steps=8, cp_beta=0.0)
    dec = decoder.Decoder(d, [blob], **kw)
    ref = _with_env({"LINMT_TC_ROWS": "0"}, lambda: decoder.Decoder(d, [blob], **kw))
    launches = []
    for h in (dec, ref):
        before = h.stats()["kernel_launches"]
        h.decode(sents)
        launches.append(h.stats()["kernel_launches"] - before)
    a, again, b = dec.score(sents, targets), dec.score(sents, targets), ref.score(sents, targets)
    dec.close(); ref.close()
    assert launches[1] >= 3 * longest > launches[0] >= 2 * longest, launches
    assert np.array_equal(a[1], again[1])
    scale = np.maximum(1, np.abs(b[1]).max(axis=1, keepdims=True))
    assert (np.abs(a[1] - b[1]) <= RTOL_FP32 * scale).all(), float((np.abs(a[1] - b[1]) / scale).max())


@pytest.mark.parametrize("layers,members,hidden,longest", [(1, 1, 512, 128), (2, 2, 512, 128), (3, 1, 1024, 24)])
def test_encoder_panels_only_for_forms_that_run(cuda_lib, layers, members, hidden, longest):
    """One-layer models, ensembles and handles for short sources never run the layers side by side, so a handle for 128
    sentences has no larger panels than one for 64: it grows by its encoder states, 12 bytes an element of a position's
    state, and not by the panels' 20 + 4 L."""
    import torch
    from linmt_b200 import decoder
    d = synth.ModelDesc(layers, hidden, 100, 60, 1)
    blobs = [synth.make_blob(d, 3 + m) for m in range(members)]

    def held(max_batch):
        before = torch.cuda.mem_get_info()[0]
        dec = decoder.Decoder(d, blobs, beam=1, max_batch=max_batch, max_src_len=longest, max_steps=8)
        after = torch.cuda.mem_get_info()[0]
        dec.close()
        return before - after

    held(64)      # (the context's own memory)
    grown = held(128) - held(64)
    elements = members * 64 * longest * hidden
    assert 6 * elements <= grown <= (12 + (20 + 4 * layers) // 2) * elements, grown / elements


@pytest.mark.parametrize("hidden,n,longest", [(512, 64, 80), (512, 96, 64), (512, 128, 41)])
def test_attention_output_over_encoder_states_runs_on_pairs(cuda_lib, hidden, n, longest):
    """The product over all encoder states that follows the layers side by side is the only one of these calls whose shape
    takes CTA pairs; the same products accumulate in the same order without them."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(2, hidden, 300, 200, 1)
    blob = synth.make_blob(d, 11, family="peaked")
    sents = synth.make_sentences(n, longest, longest, d.Vs, 1.1, 6, lambda s: 3)

    def run():
        dec = decoder.Decoder(d, [blob], beam=1, max_batch=n, max_src_len=longest, max_steps=8, cp_beta=0.0)
        out = dec.decode(sents, trace=True)
        pairs = dec.stats()["pair_launches"]
        dec.close()
        return out, pairs

    a, pairs = run()
    b, none = _with_env({"LINMT_TC_PAIR": "0"}, run)
    assert pairs == 1 and none == 0
    for key in ("cand_tok", "cand_logp", "final_logp"):
        assert a[key].tobytes() == b[key].tobytes(), key


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("n", [33, 64])     # 132 and 256 rows: the few that two row tiles hold, and all of them
def test_vocabulary_beyond_l2_on_persistent_pairs(cuda_lib, n, precision):
    """Weights that L2 cannot hold beside the states (102 MB of vocabulary in one plane) are loaded as a stream, by the
    persistent pairs of 129 to 256 rows too: the bits of the kernels without pairs."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(1, 512, 100000, 100, 1)
    blob = synth.make_blob(d, 4, family="peaked")
    sents = synth.make_sentences(n, 2, 6, d.Vs, 1.1, 5, lambda s: 3)

    def run():
        dec = decoder.Decoder(d, [blob], beam=4, precision=precision, max_batch=n, max_src_len=8, max_steps=8, cp_beta=0.0)
        out = dec.decode(sents, trace=True)
        pairs = dec.stats()["pair_launches"]
        dec.close()
        return out, pairs

    a, pairs = run()
    b, none = _with_env({"LINMT_TC_PAIR": "0"}, run)
    assert pairs >= 4 and none == 0
    for key in ("cand_tok", "cand_logp", "final_logp", "tok", "score"):
        assert a[key].tobytes() == b[key].tobytes(), key


@pytest.mark.parametrize("members,n,beam", [(2, 9, 7), (2, 13, 5), (3, 20, 7), (4, 43, 7)])      # 63, 65, 140 and 301 rows
def test_members_side_by_side(oracle, cuda_lib, members, n, beam):
    """Members decode on a stream each, beyond 64 rows in products shaped for half of the SMs: forced, against the oracle,
    and the same bits in every call."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(2, 128, 20000, 300, 1)
    blobs = [synth.make_blob(d, 40 + m, family="peaked") for m in range(members)]
    sents = synth.make_sentences(n, 2, 12, d.Vs, 1.1, 3, lambda s: 2 + s // 3)
    kw = dict(beam=beam, cp_beta=0.0, min_ratio=0.0)
    o = oracle.decode(d, blobs, sents, trace=True, **kw)
    dec = decoder.Decoder(d, blobs, max_batch=n, max_src_len=16, max_steps=20, **kw)
    e = dec.decode(sents, trace=True, force=o)
    worst, bad, skipped, compared = compare_forced(e, o, sents.steps, src_len=sents.lengths())
    assert worst <= RTOL_FP32 and bad == 0 and skipped <= 0.1 * (skipped + compared), (worst, bad, skipped, compared)
    for _ in range(3):
        again = dec.decode(sents, trace=True, force=o)
        for key in ("cand_tok", "cand_logp", "final_logp"):
            assert e[key].tobytes() == again[key].tobytes(), key
    dec.close()


@pytest.mark.parametrize("attention", ["local_p_general", "global_dot"])
@pytest.mark.parametrize("members,n,beam", [(3, 12, 5), (2, 40, 5), (3, 45, 7)])      # 60, 200 and 315 rows
def test_members_side_by_side_in_one_plane(cuda_lib, members, n, beam, attention):
    """bf16 members on a stream each run the products that they run one after another, as they do while kernels are timed:
    the same bits, decoded and scored."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(2, 128, 20000, 300, 1)
    blobs = [synth.make_blob(d, 40 + m, family="peaked") for m in range(members)]
    sents = synth.make_sentences(n, 2, 12, d.Vs, 1.1, 3, lambda s: s + 2)
    rng = np.random.default_rng(n)
    targets = [rng.integers(3, d.V, size=int(m)) for m in rng.integers(1, 10, size=n)]
    dec = decoder.Decoder(d, blobs, beam=beam, precision="bf16", attention=attention, max_batch=n, max_src_len=16, max_steps=20, cp_beta=0.0)
    side = dec.decode(sents, trace=True), dec.score(sents, targets)
    dec.set_kernel_timing(True)
    turn = dec.decode(sents, trace=True), dec.score(sents, targets)
    dec.close()
    for key in ("cand_tok", "cand_logp", "final_logp", "tok", "len", "score"):
        assert side[0][key].tobytes() == turn[0][key].tobytes(), key
    assert side[1][1].tobytes() == turn[1][1].tobytes()


@pytest.mark.parametrize("L,H,n,beam,attention,feed", [
    (2, 256, 1, 1, "local_p_general", 1), (3, 250, 5, 1, "global_general", 1), (5, 300, 1, 12, "local_p_general", 1),
    (2, 260, 4, 15, "global_dot", 1),                    # 60 rows, and 45 once a sentence has ended
    (4, 256, 16, 4, "local_p_general", 0),               # 64 rows, then 60 and fewer
    (3, 256, 33, 1, "local_p_general", 1)])              # 33 rows, then 32 and fewer
def test_recurrent_products_ahead_of_their_step(oracle, cuda_lib, L, H, n, beam, attention, feed):
    """Up to 60 rows (32 of one slot each) the recurrent products of a step are made behind the step before, by the rows that they continue:
    forced, against the oracle, and against the steps that make them in place; free, the same bits in every call."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(L, H, 2000, 300, feed)
    blob = synth.make_blob(d, 40, family="peaked")
    sents = synth.make_sentences(n, 2, 12, d.Vs, 1.1, 3, lambda s: s + 3)
    kw = dict(beam=beam, attention=attention, cp_beta=0.0, min_ratio=0.0)
    o = oracle.decode(d, [blob], sents, trace=True, **kw)
    cap = dict(max_batch=n, max_src_len=16, max_steps=20)
    dec = decoder.Decoder(d, [blob], **kw, **cap)
    e = dec.decode(sents, trace=True, force=o)
    worst, bad, skipped, compared = compare_forced(e, o, sents.steps, src_len=sents.lengths())
    assert worst <= RTOL_FP32 and bad == 0 and skipped <= 0.1 * (skipped + compared), (worst, bad, skipped, compared)
    first = dec.decode(sents)
    for _ in range(3):
        again = dec.decode(sents)
        assert first["tok"].tobytes() == again["tok"].tobytes() and first["score"].tobytes() == again["score"].tobytes()
    before = dec.stats()["kernel_launches"]
    dec.decode(sents)
    launches = dec.stats()["kernel_launches"] - before
    dec.close()
    ref = _with_env({"LINMT_AHEAD": "0"}, lambda: decoder.Decoder(d, [blob], **kw, **cap))
    r = ref.decode(sents)
    before = ref.stats()["kernel_launches"]
    ref.decode(sents)
    assert (L == 2 and beam > 1) or ref.stats()["kernel_launches"] - before != launches      # (it ran the other way)
    ref.close()
    # scores: sums of up to 15 log-probabilities of the same tokens
    for i in range(n):
        if hyps(first, i) == hyps(r, i):
            np.testing.assert_allclose(first["score"][i, 0], r["score"][i, 0], rtol=RTOL_FP32)


@pytest.mark.parametrize("n,beam", [(1, 5), (4, 12), (24, 2)])
def test_recurrent_products_ahead_in_one_plane(cuda_lib, n, beam):
    """The same in bf16, forced to the beams of the steps that make them in place: within the bar of bf16 log-probabilities."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(3, 512, 2000, 300, 1)
    blob = synth.make_blob(d, 40)
    sents = synth.make_sentences(n, 2, 12, d.Vs, 1.1, 3, lambda s: s + 3)
    kw = dict(beam=beam, precision="bf16", attention="global_general", cp_beta=0.0, max_batch=n, max_src_len=16, max_steps=20)
    ref = _with_env({"LINMT_AHEAD": "0"}, lambda: decoder.Decoder(d, [blob], **kw))
    r = ref.decode(sents, trace=True)
    dec = decoder.Decoder(d, [blob], **kw)
    e = dec.decode(sents, trace=True, force=r)
    ref.close(); dec.close()
    for i in range(n):
        T = int(sents.steps[i])
        a, b = np.sort(e["cand_logp"][i, 1:T]), np.sort(r["cand_logp"][i, 1:T])
        assert (np.abs(a - b) <= 2e-2).all(), float(np.abs(a - b).max())


@pytest.mark.parametrize("precision,beam,max_batch,n,info", [("fp32", 1, 4, 31, False), ("fp32", 5, 8, 17, True), ("bf16", 3, 16, 70, False),
                                                             ("fp32", 16, 32, 65, False), ("fp32", 2, 3, 4, False)])     # (the fourth: 512 rows)
def test_device_batches_of_a_call_at_once(cuda_lib, precision, beam, max_batch, n, info):
    """A call of several device batches runs some of them at once, decoding and scoring: the same bits in every call, the
    results of one after another (in other shapes of products: to fp32 rounding, or to the bar of bf16 log-probabilities), and
    the counters of all of them."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(2, 256, 3000, 300, 1)
    blob = synth.make_blob(d, 40, family="peaked" if precision == "fp32" else "flat")
    sents = synth.make_sentences(n, 1, 14, d.Vs, 1.1, 3, lambda s: s + 3)
    rng = np.random.default_rng(n)
    targets = [rng.integers(3, d.V, size=int(m)) for m in rng.integers(1, 12, size=n)]
    kw = dict(beam=beam, precision=precision, max_batch=max_batch, max_src_len=16, max_steps=20, print_info=info, cp_beta=0.2 if info else 0.0)
    dec = decoder.Decoder(d, [blob], **kw)
    one = _with_env({"LINMT_LANES": "0"}, lambda: decoder.Decoder(d, [blob], **kw))
    b, y = one.decode(sents, want_align=info), one.score(sents, targets)
    first = None
    for call in range(3):
        a, x = dec.decode(sents, want_align=info), dec.score(sents, targets)
        first = first or (a, x)
        for key in ("tok", "len", "score") + (("vit", "align") if info else ()):
            assert a[key].tobytes() == first[0][key].tobytes(), (call, key)
        assert x[0].tobytes() == first[1][0].tobytes() and x[1].tobytes() == first[1][1].tobytes(), call
    a, x = first
    if precision == "fp32":
        scale = np.maximum(1, np.abs(y[1]).max(axis=1, keepdims=True))
        assert (np.abs(x[1] - y[1]) <= RTOL_FP32 * scale).all(), float((np.abs(x[1] - y[1]) / scale).max())
        same = [i for i in range(n) if hyps(a, i) == hyps(b, i)]
        assert len(same) >= 0.95 * n, len(same)       # (a tie may go the other way)
        for i in same:
            np.testing.assert_allclose(a["score"][i, 0], b["score"][i, 0], rtol=RTOL_FP32)
    else:
        assert (np.abs(x[1] - y[1]) <= 2e-2).all(), float(np.abs(x[1] - y[1]).max())
    assert dec.stats()["sentence_steps"] == 3 * one.stats()["sentence_steps"]
    short = synth.make_sentences(1, 3, 3, d.Vs, 1.1, 3, lambda s: s + 3)      # one batch, after many
    assert dec.decode(short)["tok"].tobytes() == one.decode(short)["tok"].tobytes()
    dec.close(); one.close()


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("L,H,n,longest,max_src", [(2, 512, 1, 20, 64), (5, 500, 3, 41, 48), (3, 512, 32, 33, 33), (4, 448, 64, 21, 24), (2, 512, 7, 500, 512), (3, 512, 2, 21, 21)])
def test_encoder_of_few_sentences_side_by_side(cuda_lib, precision, L, H, n, longest, max_src):
    """Sources of 20 words and more of at most 64 sentences: the layers side by side from 449 units on (rounded to 512), one after
    another below, against the encoder position by position; log-probabilities of given words to fp32 rounding, or within the
    bar of bf16."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(L, H, 300, 200, 1)
    blob = synth.make_blob(d, 11, family="peaked" if precision == "fp32" else "flat")
    rng = np.random.default_rng(n)
    lens = np.concatenate([[longest], rng.integers(1, longest + 1, size=n - 1)]).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    sents = synth.Sentences(synth.zipf_ids(rng, int(off[-1]), 1, d.Vs, 1.1), off, np.full(n, 3, np.int32))
    targets = [rng.integers(3, d.V, size=int(m)) for m in rng.integers(1, 4, size=n)]
    kw = dict(beam=2, precision=precision, max_batch=n, max_src_len=max_src, max_steps=8, cp_beta=0.0)
    dec = decoder.Decoder(d, [blob], **kw)
    ref = _with_env({"LINMT_TC_ROWS": "0"}, lambda: decoder.Decoder(d, [blob], **kw))
    a, again, b = dec.score(sents, targets), dec.score(sents, targets), ref.score(sents, targets)
    dec.close(); ref.close()
    assert np.array_equal(a[1], again[1])
    if precision == "fp32":
        scale = np.maximum(1, np.abs(b[1]).max(axis=1, keepdims=True))
        assert (np.abs(a[1] - b[1]) <= RTOL_FP32 * scale).all(), float((np.abs(a[1] - b[1]) / scale).max())
    else:
        assert (np.abs(a[1] - b[1]) <= 2e-2).all(), float(np.abs(a[1] - b[1]).max())


@pytest.mark.parametrize("L,H,n,beam,max_batch,longest", [
    (3, 512, 1, 5, 8, 30), (2, 300, 40, 1, 40, 30),                            # one device batch
    (3, 512, 9, 12, 3, 25), (2, 512, 70, 2, 32, 12), (2, 256, 200, 4, 96, 12)])    # several, of 36, 64 and 384 rows; scoring 3, 32 and 96
def test_one_plane_has_one_order_of_sums(cuda_lib, L, H, n, beam, max_batch, longest):
    """bf16 results do not go by what runs beside a step or beside a device batch: the same bits with and without."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(L, H, 2000, 300, 1)
    blob = synth.make_blob(d, 40)
    sents = synth.make_sentences(n, 2, longest, d.Vs, 1.1, 3, lambda s: s // 2 + 3)
    rng = np.random.default_rng(n)
    targets = [rng.integers(3, d.V, size=int(m)) for m in rng.integers(1, 15, size=n)]
    kw = dict(beam=beam, precision="bf16", cp_beta=0.0, max_batch=max_batch, max_src_len=32, max_steps=20)
    dec = decoder.Decoder(d, [blob], **kw)
    ref = _with_env({"LINMT_AHEAD": "0", "LINMT_LANES": "0"}, lambda: decoder.Decoder(d, [blob], **kw))
    a, b = dec.decode(sents), ref.decode(sents)
    x, y = dec.score(sents, targets), ref.score(sents, targets)
    dec.close(); ref.close()
    for key in ("tok", "len", "score"):
        assert a[key].tobytes() == b[key].tobytes(), key
    assert x[1].tobytes() == y[1].tobytes()


@pytest.mark.parametrize("L,H,beam,max_batch,n,lo,hi", [
    (5, 768, 3, 32, 100, 2, 12),       # a step's weights are more than L2 keeps: two engines, of 96 rows
    (3, 256, 1, 96, 200, 20, 40)])     # three engines, each with a pipelined encoder (96 sentences of 32 words and more)
def test_engines_of_a_call_beyond_l2_and_with_pipelined_encoders(cuda_lib, L, H, beam, max_batch, n, lo, hi):
    """Device batches at once: the same bits in every call, and the results of one batch after another to fp32 rounding."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(L, H, 3000, 300, 1)
    blob = synth.make_blob(d, 40, family="peaked")
    sents = synth.make_sentences(n, lo, hi, d.Vs, 1.1, 3, lambda s: s // 2 + 3)
    rng = np.random.default_rng(n)
    targets = [rng.integers(3, d.V, size=int(m)) for m in rng.integers(1, 12, size=n)]
    kw = dict(beam=beam, max_batch=max_batch, max_src_len=hi, max_steps=24, cp_beta=0.0)
    one = _with_env({"LINMT_LANES": "0"}, lambda: decoder.Decoder(d, [blob], **kw))
    b, y = one.decode(sents), one.score(sents, targets)
    one.close()
    dec = decoder.Decoder(d, [blob], **kw)
    a, x = dec.decode(sents), dec.score(sents, targets)
    for _ in range(3):
        again, z = dec.decode(sents), dec.score(sents, targets)
        assert a["tok"].tobytes() == again["tok"].tobytes() and a["score"].tobytes() == again["score"].tobytes()
        assert x[1].tobytes() == z[1].tobytes()
    dec.close()
    scale = np.maximum(1, np.abs(y[1]).max(axis=1, keepdims=True))
    assert (np.abs(x[1] - y[1]) <= RTOL_FP32 * scale).all(), float((np.abs(x[1] - y[1]) / scale).max())
    same = [i for i in range(n) if hyps(a, i) == hyps(b, i)]
    assert len(same) >= 0.95 * n, len(same)       # (a tie may go the other way)
    for i in same:
        np.testing.assert_allclose(a["score"][i, 0], b["score"][i, 0], rtol=RTOL_FP32)


def test_encoder_layers_side_by_side_in_two_chunks(cuda_lib):
    """40 sentences of up to 500 words are more rows than the panels hold (16384): against the encoder position by position."""
    from linmt_b200 import decoder
    d = synth.ModelDesc(2, 512, 300, 200, 1)
    blob = synth.make_blob(d, 11, family="peaked")
    sents = synth.make_sentences(40, 380, 500, d.Vs, 1.1, 3, lambda s: 3)
    rng = np.random.default_rng(4)
    targets = [rng.integers(3, d.V, size=int(m)) for m in rng.integers(1, 4, size=40)]
    kw = dict(beam=2, max_batch=40, max_src_len=500, max_steps=8, cp_beta=0.0)
    dec = decoder.Decoder(d, [blob], **kw)
    ref = _with_env({"LINMT_TC_ROWS": "0"}, lambda: decoder.Decoder(d, [blob], **kw))
    a, b = dec.score(sents, targets), ref.score(sents, targets)
    dec.close(); ref.close()
    scale = np.maximum(1, np.abs(b[1]).max(axis=1, keepdims=True))
    assert (np.abs(a[1] - b[1]) <= RTOL_FP32 * scale).all(), float((np.abs(a[1] - b[1]) / scale).max())
