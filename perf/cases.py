"""The work that a user of this framework has it do, as cases that can be timed and compared.

Four kinds of call, all through the package's public functions:
  decode    one token through mlstm_recurrent_step__b200 (what mLSTMBackend's step kernel does per generated token)
  sequence  a handful of tokens through mlstm_recurrent_sequence__b200 (tail of a prompt, several tokens at once)
  prefill   a prompt through the chunkwise forward, without gradients, last states returned for the decode that follows
  train     the chunkwise forward and backward: H and the gradients of q, k, v, i, f from an upstream gradient of H

Inputs have the distributions of the repository's benchmark and tests: q, k, v, i ~ N(0, 1), forget logits 3 + N(0, 1),
upstream gradient N(0, 1), states C ~ N(0, 0.1), n ~ |N(0, 1)|, m ~ N(0, 1).
"""

import math

import torch

import mlstm_kernels_b200 as mk

_DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16, "f32": torch.float32}
_BYTES = {"bf16": 2, "fp16": 2, "f32": 4}

# Head geometries (DHQK, DHHV) of the repository's benchmark, tests and configurations.
_HEADS = [(64, 128), (96, 192), (128, 128), (128, 256), (192, 384), (256, 256), (256, 512)]


def listed():
    return [
        # one user generating text at the 7B head geometry: the smallest call, launch latency and host time count
        dict(name="decode_b1", kind="decode", B=1, NH=8, DHQK=256, DHHV=512, dtype="bf16", gates="bf16", state="f32"),
        # a handful of users sharing a GPU
        dict(name="decode_b8", kind="decode", B=8, NH=8, DHQK=256, DHHV=512, dtype="bf16", gates="f32", state="f32"),
        # a full serving batch: 2.1 GB of state traffic per token
        dict(name="decode_b256", kind="decode", B=256, NH=8, DHQK=256, DHHV=512, dtype="bf16", gates="bf16", state="f32"),
        # the last few tokens of four prompts, or several proposed tokens checked at once, in one launch
        dict(name="sequence_t13", kind="sequence", B=4, NH=8, S=13, DHQK=256, DHHV=512, dtype="bf16", gates="bf16",
             init=True),
        # one short prompt of any length
        dict(name="prefill_s500", kind="prefill", B=1, NH=8, S=500, DHQK=256, DHHV=512, dtype="bf16", gates="bf16",
             variant="exp", chunk=128, init=False),
        # the next turn of four conversations: a prompt that starts from the states the last turn left
        dict(name="prefill_continue", kind="prefill", B=4, NH=8, S=1234, DHQK=256, DHHV=512, dtype="bf16", gates="f32",
             variant="exp", chunk=128, init=True),
        # a batch of long prompts of a length that is no multiple of anything
        dict(name="prefill_s8077", kind="prefill", B=8, NH=16, S=8077, DHQK=256, DHHV=256, dtype="bf16", gates="bf16",
             variant="exp", chunk=128, init=False),
        # one very long document
        dict(name="prefill_s131072", kind="prefill", B=1, NH=8, S=131072, DHQK=256, DHHV=512, dtype="bf16", gates="bf16",
             variant="exp", chunk=256, init=False),
        # a layer of a small model trained in half precision, head dims off the powers of two, normalised sigmoid gate
        dict(name="train_small_fp16", kind="train", B=4, NH=4, S=1024, DHQK=96, DHHV=192, dtype="fp16", gates="fp16",
             variant="sig", chunk=128, recompute=True),
        # a training step of one layer with the sigmoid input gate (no normaliser), states recomputed (the default)
        dict(name="train_sig", kind="train", B=16, NH=16, S=2048, DHQK=128, DHHV=256, dtype="bf16", gates="f32",
             variant="sig_nonorm", chunk=128, recompute=True),
        # the benchmark's step: 65 536 tokens, exponential input gate, per-chunk states kept for the backward
        dict(name="train_64k", kind="train", B=8, NH=16, S=8192, DHQK=256, DHHV=256, dtype="bf16", gates="bf16",
             variant="exp", chunk=128, recompute=False),
        # single precision, the functions' default kernel dtype: the configuration that parity is checked on
        dict(name="train_f32", kind="train", B=2, NH=4, S=512, DHQK=128, DHHV=256, dtype="f32", gates="f32",
             variant="exp", chunk=64, recompute=True),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "sequence", "prefill", "prefill", "train", "train", "train_f32"])
    heads = rng.choice(_HEADS)
    if rng.random() < 0.2:   # any head dims that are multiples of 8
        heads = (8 * rng.randint(4, 32), 8 * rng.randint(4, 64))
    case = dict(kind=kind, NH=rng.choice([4, 8, 16]), DHQK=heads[0], DHHV=heads[1],
                dtype=rng.choice(["bf16", "bf16", "bf16", "fp16"]))
    case["gates"] = rng.choice([case["dtype"], "f32"])
    if kind == "decode":
        most = max(1, 256 * 8 * 256 * 512 // (case["NH"] * case["DHQK"] * case["DHHV"]))
        case.update(B=_log_int(rng, 1, min(512, most)), state=rng.choice(["f32", "f32", "f32", "bf16"]))
    elif kind == "sequence":
        case.update(B=_log_int(rng, 1, 16), S=_log_int(rng, 2, 64), init=rng.random() < 0.7)
    elif kind == "train_f32":
        chunk = rng.choice([64, 128])
        case.update(kind="train", dtype="f32", gates="f32", B=_log_int(rng, 1, 4), NH=4, chunk=chunk,
                    S=chunk * _log_int(rng, 1, 2048 // chunk), DHQK=min(128, case["DHQK"]), DHHV=min(256, case["DHHV"]),
                    variant=rng.choice(["exp", "sig"]), recompute=rng.random() < 0.7)
    else:
        case.update(variant=rng.choice(["exp", "exp", "exp", "sig", "sig_nonorm"]), chunk=rng.choice([64, 128, 256]))
        # tokens of one call, at most the work of the largest listed one: about 2^20 (batch, head, token) at 256 / 256
        most = int(0.9 * (1 << 20) * 256 * 512 / (case["DHQK"] * case["DHHV"] + 256 * 256)) // case["NH"]
        most = min(most, 131072)
        case["S"] = _log_int(rng, 100, min(most, 131072 if kind == "prefill" else 16384))
        case["B"] = _log_int(rng, 1, max(1, min(32, most // case["S"])))
        if kind == "prefill":
            case["init"] = case["variant"] == "exp" and rng.random() < 0.4
        else:
            case["recompute"] = rng.random() < 0.7
    return case


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt, gdt = _DTYPE[case["dtype"]], _DTYPE[case["gates"]]
    B, NH, DHQK, DHHV = case["B"], case["NH"], case["DHQK"], case["DHHV"]

    def randn(*shape, dtype):
        return torch.randn(shape, generator=gen, device="cuda", dtype=dtype)

    tok = () if case["kind"] == "decode" else (case["S"],)
    gate = (1,) if case["kind"] == "decode" else tok
    s = dict(case=case, q=randn(B, NH, *tok, DHQK, dtype=dt), k=randn(B, NH, *tok, DHQK, dtype=dt),
             v=randn(B, NH, *tok, DHHV, dtype=dt), i=randn(B, NH, *gate, dtype=gdt),
             f=3 + randn(B, NH, *gate, dtype=gdt))
    if case["kind"] == "decode" or case.get("init"):
        sdt = _DTYPE[case.get("state", "f32")]
        s.update(c=0.1 * randn(B, NH, DHQK, DHHV, dtype=sdt), n=randn(B, NH, DHQK, dtype=sdt).abs(),
                 m=randn(B, NH, 1, dtype=sdt))
    if case["kind"] == "train":
        for x in "qkvif":
            s[x].requires_grad_(True)
        s["dh"] = randn(B, NH, *tok, DHHV, dtype=dt)
    return s


def _chunkwise(s, **kw):
    case = s["case"]
    if case["variant"] == "exp":
        return mk.mlstm_chunkwise__b200_xl_chunk(s["q"], s["k"], s["v"], s["i"], s["f"], chunk_size=case["chunk"], **kw)
    return mk.mlstm_siging_chunkwise__b200_xl_chunk(s["q"], s["k"], s["v"], s["i"], s["f"], chunk_size=case["chunk"],
                                                    normalize=case["variant"] == "sig", **kw)


def run(s):
    case = s["case"]
    if case["kind"] == "decode":
        h, (c, n, m) = mk.mlstm_recurrent_step__b200(s["q"], s["k"], s["v"], s["i"], s["f"], s["c"], s["n"], s["m"],
                                                     dtype_state=_DTYPE[case["state"]])
        return {"h": h, "c": c, "n": n, "m": m}
    if case["kind"] == "sequence":
        h, (c, n, m) = mk.mlstm_recurrent_sequence__b200(s["q"], s["k"], s["v"], s["i"], s["f"], s.get("c"), s.get("n"),
                                                         s.get("m"), return_last_states=True)
        return {"h": h, "c": c, "n": n, "m": m}
    if case["kind"] == "prefill":
        with torch.no_grad():
            h, last = _chunkwise(s, c_initial=s.get("c"), n_initial=s.get("n"), m_initial=s.get("m"),
                                 return_last_states=True)
        return {"h": h, **dict(zip("cnm", last))}
    h = _chunkwise(s, recompute_states_in_bw=case["recompute"])
    grads = torch.autograd.grad(h, [s[x] for x in "qkvif"], s["dh"])
    return {"h": h, **dict(zip(("dq", "dk", "dv", "di", "df"), grads))}


def work(case):
    el, gel = _BYTES[case["dtype"]], _BYTES[case["gates"]]
    units, DHQK, DHHV = case["B"] * case["NH"], case["DHQK"], case["DHHV"]
    T = case.get("S", 1)
    state = units * (DHQK * DHHV + DHQK + 1) * _BYTES[case.get("state", "f32")]
    token = (2 * DHQK + 2 * DHHV) * el + 2 * gel   # q, k, v, i, f in, h out
    if case["kind"] in ("decode", "sequence"):
        # per token: k v^T added to the decayed state, q times the new state
        return {"bytes": units * T * token + state * (2 if case["kind"] == "decode" or case["init"] else 1),
                "flops": units * T * 4 * DHQK * DHHV}
    # chunks of 128 (one chunk of T when T is smaller): states in, states out, the causal half of both L x L products
    L = min(128, T)
    flops = units * T * (4 * DHQK * DHHV + L * (DHQK + DHHV))
    if case["kind"] == "prefill":
        return {"bytes": units * T * token + state * (2 if case["init"] else 1), "flops": flops}
    # backward: the gradient's recurrence, three products with the states, the causal halves of five L x L products
    flops += units * T * (8 * DHQK * DHHV + L * (3 * DHQK + 2 * DHHV))
    # q, k, v, dh and the gates in, h and five gradients out
    return {"bytes": units * T * 2 * token, "flops": flops}


def tolerance(case):
    # Rounding of the 16-bit results is 1.7e-3 (bf16) and 3e-4 (fp16) by itself.  The chunkwise kernels may also keep
    # per-chunk states and gated tiles in 16 bits (2.4e-3 against exact arithmetic), and the forget-gate gradient is a
    # running sum of nearly cancelling terms (6e-3 in bf16, 7e-4 in fp16); two such results differ by up to twice that.
    # Single precision: sums of a few hundred terms in another order (7e-7; 3e-6 in the forget-gate gradient).
    if case["dtype"] == "f32":
        return {"rel": 1e-5}
    rel = {"decode": 4e-3, "sequence": 4e-3, "prefill": 6e-3, "train": 1.5e-2}[case["kind"]]
    return {"rel": rel / 8 if case["dtype"] == "fp16" and case.get("state") != "bf16" else rel}
