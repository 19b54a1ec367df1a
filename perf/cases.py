"""Performance cases of the decoding library: calls a translation program makes through ``linmt_b200.decoder``.

A case names a model shape, the options of the handle that a program keeps for it, one call on that handle
(``decode``: beam search; ``score``: log-probabilities of given translations) and the sentences of the call.  Source
ids are Zipf-distributed, lengths spread evenly between two bounds, steps 1.5 S + 10 as in the repository's configurations.

The weights behave like a trained model's in what decides speed and comparability: activations of ordinary size, a
decaying memory, and a peaked next-word distribution that names a definite word after every word (and a definite
first word for the source word read last), so that one-best hypotheses do not hang on the last bit of a sum.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from linmt_b200 import decoder, synth

# Model shapes and seeds of the repository's configurations: C1's, the 4 x 1000 / 30k model of C2, C3 and C5 (C5: four
# of them), C4's 4 x 1024 / 80k; and sizes off every tile boundary as its tests use them.
SMALL = dict(layers=2, hidden=128, vocab=1000)
BASE = dict(layers=4, hidden=1000, vocab=30000)
LARGE_VOCAB = dict(layers=4, hidden=1024, vocab=80000)
ODD = dict(layers=3, hidden=250, vocab=5003)


def _case(model, **kw):
    c = dict(model, entry="decode", members=1, precision="fp32", attention="local_p_general", beam=12, nbest=1,
             print_info=False, cp_beta=0.0, max_batch=64, n=1, len_lo=10, len_hi=50)
    c.update(kw)
    return c


def listed():
    return [
        # a small model answering one sentence at a time, greedily: nothing but latency
        _case(SMALL, name="small_greedy_one", beam=1, len_lo=5, len_hi=20),
        # an n-best list with alignments and coverage penalty for a handful of sentences, sizes off every tile
        _case(ODD, name="odd_nbest_align", beam=7, nbest=3, print_info=True, cp_beta=0.2, max_batch=16, n=11, len_lo=1, len_hi=40),
        # the reference's sentence API: one sentence on the full-size model
        _case(BASE, name="one_sentence", n=1),
        # a server's small ragged batch: one word to a long paragraph
        _case(BASE, name="ragged_eight", n=8, beam=5, nbest=2, print_info=True, cp_beta=0.2, len_lo=1, len_hi=100),
        # the headline configuration (C2)
        _case(BASE, name="batch64", n=64),
        # greedy translation of a file that does not fit one device batch
        _case(BASE, name="greedy_file", n=300, beam=1, len_lo=5, len_hi=80),
        # scoring given translations (rescoring, perplexity) on the handle that translates
        _case(BASE, name="score64", entry="score", n=64),
        # bf16, one sentence, attention over the whole source
        _case(BASE, name="one_bf16_global", precision="bf16", attention="global_general", n=1, beam=5, max_batch=8),
        # the throughput configuration (C3): a length-bucketed bf16 batch
        _case(BASE, name="batch128_bf16", precision="bf16", n=128, len_lo=40, len_hi=60, max_batch=128),
        # scoring in bf16 on a handle kept for it, more sentences than a device batch
        _case(BASE, name="score_bf16", entry="score", precision="bf16", n=200, beam=1, max_batch=128),
        # the output-bound configuration (C4): 80k words, global dot attention
        _case(LARGE_VOCAB, name="large_vocab_bf16", precision="bf16", attention="global_dot", n=128, beam=5, len_lo=20, len_hi=100,
              max_batch=128),
        # the ensemble configuration (C5)
        _case(BASE, name="ensemble4", members=4, n=32, len_lo=10, len_hi=60),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice([SMALL, ODD, BASE, BASE, LARGE_VOCAB, None])
    if model is None:   # a size of nobody's configuration
        model = dict(layers=rng.randint(1, 5), hidden=spread(96, 1024), vocab=spread(1000, 60000))
    precision = rng.choice(["fp32", "fp32", "bf16"]) if model["hidden"] >= 500 else "fp32"   # bf16 is for the large models
    members = rng.choice([1, 1, 1, 1, 2, 3]) if model["vocab"] <= 30000 else 1
    entry = rng.choice(["decode", "decode", "decode", "score"])
    info = entry == "decode" and precision == "fp32" and rng.random() < 0.3
    hi = spread(8, 100)
    c = _case(model, entry=entry, members=members, precision=precision,
              attention=rng.choice(["local_p_general", "local_p_general", "global_general", "global_dot"]),
              beam=spread(1, 16), nbest=1, print_info=info, cp_beta=0.2 if info else 0.0, n=spread(1, 256),
              len_lo=rng.randint(1, hi), len_hi=hi, max_batch=rng.choice([32, 64, 64, 128]))
    if info:
        c["nbest"] = rng.randint(1, min(3, c["beam"]))
    # no more than the largest listed case: arithmetic, and device batches times their steps
    most = 0.7 * max(work(x)["flops"] for x in listed())
    while c["n"] > 1 and (work(c)["flops"] > most or -(-c["n"] // c["max_batch"]) * members * _steps(hi) > 600):
        c["n"] //= 2
    return c


def _steps(s):
    return int(1.5 * s) + 10


# ---- the model -------------------------------------------------------------------------------------------------
# Scales of the groups of matrices against uniform [-0.08, 0.08] at hidden size 1000.
_EMB, _RECURRENT, _INPUT, _FEED, _CONTEXT, _FORGET_BIAS = 5.0, 0.5, 3.0, 0.3, 0.3, -1.0
_PEAK = 25.0    # logit of the next word above the rest


def _cell(w, prefix, x, h, c):
    z = {g: x @ w[f"{prefix}.M_{g}"] + w[f"{prefix}.b_{g}"].T.reshape(1, -1) for g in "ifco"}
    if h is not None:
        z = {g: z[g] + h @ w[f"{prefix}.W_h{g}"] for g in "ifco"}
    c_new = torch.sigmoid(z["i"]) * torch.tanh(z["c"])
    if c is not None:
        c_new = c_new + torch.sigmoid(z["f"]) * c
    return torch.sigmoid(z["o"]) * torch.tanh(c_new), c_new


def _weights(desc, seed):
    """A weight blob whose output rows answer to the attentional states that single words leave."""
    blob = synth.make_blob(desc, seed)
    w, off = {}, {}
    at = 0
    for name, r, c in synth.blob_layout(desc):
        off[name] = (at, r * c)
        leaf = name.split(".")[1]
        part = blob[at:at + r * c]
        if leaf == "W_emb":
            part *= np.float32(_EMB)
            if name.startswith("tgt"):
                part[:r] = 0.0        # START carries nothing: the first word comes from the source
        elif leaf == "b_f":
            part[:] = _FORGET_BIAS
        elif leaf[:2] in ("W_", "M_", "Q_") and not name.startswith(("sm.", "att.v")):
            by = {"W_h": _RECURRENT, "W_c1": _CONTEXT}.get(leaf if leaf == "W_c1" else leaf[:3], 1.0)
            if leaf[0] == "M" and not name.startswith(("src0", "tgt0")):
                by = _INPUT
            if leaf[0] == "Q":
                by = _FEED
            part *= np.float32(by * math.sqrt(1000.0 / desc.H))
        if name != "sm.D":
            w[name] = torch.from_numpy(part.reshape(c, r)).cuda()     # stored [in][out]
        at += r * c

    # what one source word, then START, leaves; and what one target word leaves on its own
    def states(prefix, x, below):
        out = []
        for l in range(desc.L):
            x, c = _cell(w, f"{prefix}{l}", x, *(below[l] if below else (None, None)))
            out.append((x, c))
        return out

    first, following = [], []
    for lo in range(0, desc.Vs, 16384):
        enc = states("src", w["src0.W_emb"][lo:lo + 16384], None)
        top = states("tgt", torch.zeros_like(enc[0][0]), enc)[-1][0]
        first.append(torch.tanh(enc[-1][0] @ w["att.W_c1"] + top @ w["att.W_c2"]))
    for lo in range(0, desc.V, 16384):
        top = states("tgt", w["tgt0.W_emb"][lo:lo + 16384], None)[-1][0]
        following.append(torch.tanh(top @ w["att.W_c2"]))
    first, following = torch.cat(first), torch.cat(following)
    size = float(following.norm(dim=1).mean())
    unit = torch.nn.functional.normalize
    words = torch.arange(3, desc.V, device="cuda")        # START, EOS and UNK follow nothing
    rows = torch.empty(desc.V, desc.H, device="cuda")
    rows[:3] = 0.2 * _PEAK / size * unit(torch.from_numpy(np.random.default_rng(seed + 1).standard_normal((3, desc.H), np.float32)).cuda())
    rows[3:] = _PEAK / size * (unit(following[3 + (words * 7919 + 11) % (desc.V - 3)]) + unit(first[words % desc.Vs]))
    lo, size = off["sm.D"]
    blob[lo:lo + size] = rows.T.contiguous().cpu().numpy().reshape(-1)      # [H][V]
    return blob


_blobs, _handles = {}, {}     # the models and the handle of the last case: a program keeps them between calls


def _handle(case):
    model = (case["layers"], case["hidden"], case["vocab"], case["members"])
    options = dict(beam=case["beam"], nbest=case["nbest"], attention=case["attention"], print_info=int(case["print_info"]),
                   precision=case["precision"], max_batch=case["max_batch"], cp_beta=case["cp_beta"])
    key = model + tuple(sorted(options.items()))
    if key not in _handles:
        _handles.clear()
        desc = synth.ModelDesc(case["layers"], case["hidden"], case["vocab"], case["vocab"], 1)
        if model not in _blobs:
            _blobs.clear()
            _blobs[model] = [_weights(desc, 10 + m if case["members"] > 1 else 1) for m in range(case["members"])]
            torch.cuda.empty_cache()
        _handles[key] = decoder.Decoder(desc, _blobs[model], **options)
    return _handles[key]


def prepare(case, seed):
    # every seed draws the same spread of lengths, in an order of its own
    rng = np.random.default_rng(seed)
    n, lo, hi = case["n"], case["len_lo"], case["len_hi"]
    lens = rng.permutation(lo + ((np.arange(n) + 0.5) * (hi + 1 - lo) / n).astype(np.int32))
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    sents = synth.Sentences(synth.zipf_ids(rng, int(off[-1]), 1, case["vocab"], 1.1), off, np.array([_steps(int(s)) for s in lens], np.int32))
    state = {"decoder": _handle(case), "sents": sents, "align": case["print_info"]}
    if case["entry"] == "score":
        state["targets"] = [synth.zipf_ids(rng, int(1.1 * s) + 2, 3, case["vocab"], 1.1) for s in lens]
    return state


def run(state):
    if "targets" in state:
        total, per_token = state["decoder"].score(state["sents"], state["targets"])
        return {"total": total, "per_token": per_token}
    out = state["decoder"].decode(state["sents"], want_align=state["align"])
    got = {k: out[k] for k in ("tok", "len", "score")}
    if state["align"]:
        got.update(vit=out["vit"], align=out["align"])
    return got


def work(case):
    L, H, V, m, n = case["layers"], case["hidden"], case["vocab"], case["members"], case["n"]
    s = 0.5 * (case["len_lo"] + case["len_hi"])
    score = case["entry"] == "score"
    steps = 1.1 * s + 3 if score else 1.5 * s + 11
    k = 1 if score else case["beam"]
    window = min(s, 21.0) if case["attention"] == "local_p_general" else s
    # per decoder row: LSTM stack (input, recurrent, feed-input), attention and its output layer, vocabulary
    per_row = 2.0 * (8 * L * H * H + 4 * H * H + (2 if case["attention"] == "global_dot" else 4) * H * H + 2 * window * H + H * V)
    flops = m * n * (s * 16.0 * L * H * H + k * steps * per_row)
    width = 2 if case["precision"] == "bf16" else 4
    weights = 16 * L * H * H + 8 * H * H + H * V + min(n * s, V) * H + min(n * k * steps, V) * H
    return {"bytes": m * weights * width + 4.0 * n * (s + case["nbest"] * steps), "flops": flops}


def tolerance(case):
    # bf16: the recurrent state is rounded to 8 bits at every step; fp32: the recurrence carries a sum's rounding on.
    # Tokens: a pair of hypotheses may be closer to each other than that.
    if case["precision"] == "bf16":
        return {"rel": 1e-2, "max": 0.2, "differ": 0.005}
    return {"rel": 5e-5, "max": 2e-3, "differ": 0.005}
