"""The work that users of this package have it do, as measurable cases.

Every case goes through the public functions of the package on the current CUDA stream:

  decode        recurrent_forward, one token per sequence, the state updated where it lies
  decode_layer  one token through the whole mixer: causal_conv1d, recurrent_forward, gated_rmsnorm
  verify        recurrent_forward over a few draft tokens per sequence
  prefill       chunked_forward on padded batches
  packed        chunked_forward on packed sequences of unequal length
  layer         a prompt through the whole mixer: causal_conv1d, fused_gdn_gating, chunked_forward, gated_rmsnorm

Sizes are those of the benchmark configurations and of the tests (16 key heads, 32 value heads, head dim 128
and their shards; head dims 64 to 256), or odd neighbours of them.  Inputs follow the distributions the benchmark
uses: q, k, v ~ N(0, 1) (q, k L2-normalised where the call does not do it), beta = sigmoid(N(0, 1)),
gate = -exp(A_log) softplus(a + dt_bias), states ~ N(0, 0.02).
"""
import math
import os

import torch

import h100_gdn_cuda_b200 as gdn

CHUNK = 64
_ready = False


def listed():
    return [
        # one user's next token through the whole mixer: three short calls, launches and host time are all there is
        dict(name="decode_layer_b1", op="decode_layer", B=1, kh=16, vh=32, d=128),
        # a serving engine's running batch: states in a pool, one slot per sequence
        dict(name="decode_pool_b24", op="decode", B=24, kh=16, vh=32, d=128, state="bf16", where="pool", gating="inside"),
        # the benchmark's decode step: 268 MB of states updated in place
        dict(name="decode_b256", op="decode", B=256, kh=16, vh=32, d=128, state="bf16", where="inplace", gating="inside"),
        # states kept in fp32 between steps, an odd batch, beta and the gate given by the caller
        dict(name="decode_fp32_b93", op="decode", B=93, kh=16, vh=32, d=128, state="f32", where="inplace", gating="given"),
        # the benchmark's speculative verify: the state advances by the accepted tokens of each sequence
        dict(name="verify_b64_t4", op="verify", B=64, T=4, kh=16, vh=32, d=128, steps=False),
        # draft tokens scored with a state kept per token, so that the caller can roll back
        dict(name="verify_steps_b13_t5", op="verify", B=13, T=5, kh=16, vh=32, d=128, steps=True),
        # the smallest configuration: a short prompt, head dim 64, no state yet
        dict(name="prefill_b1_t256_d64", op="prefill", B=1, T=256, kh=4, vh=4, d=64, norm=False, state=False),
        # the benchmark's padded prefill
        dict(name="prefill_b4_t4096", op="prefill", B=4, T=4096, kh=16, vh=32, d=128, norm=False, state=True),
        # a wide-head layer, ragged length
        dict(name="prefill_b2_t1500_d256", op="prefill", B=2, T=1500, kh=4, vh=8, d=256, norm=False, state=True),
        # the benchmark's packed batch: 16 prompts of log-normal lengths
        dict(name="packed_16x32768", op="packed", n=16, tokens=32768, kh=16, vh=32, d=128),
        # one GPU's share of the long-context layer whose value heads are spread over eight
        dict(name="prefill_b2_t131072_h4", op="prefill", B=2, T=131072, kh=2, vh=4, d=128, norm=False, state=True),
        # one slice of a long prompt through the whole mixer, continuing from the state of the slice before
        dict(name="layer_b1_t7919", op="layer", B=1, T=7919, kh=16, vh=32, d=128),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["decode", "decode", "decode_layer", "verify", "prefill", "prefill", "packed", "long", "layer", "wide"])
    kh, vh = rng.choice([(16, 32), (16, 32), (8, 16), (4, 8), (2, 4)])
    if op == "decode":
        state = rng.choice(["bf16", "bf16", "f32"])
        return dict(op="decode", B=_log(rng, 1, 256 if state == "bf16" else 128), kh=kh, vh=vh, d=rng.choice([128, 128, 64]),
                    state=state, where=rng.choice(["inplace", "pool", "new"]), gating=rng.choice(["inside", "given"]))
    if op == "decode_layer":
        return dict(op="decode_layer", B=_log(rng, 1, 64), kh=kh, vh=vh, d=128)
    if op == "verify":
        steps = rng.random() < 0.5
        T = rng.randint(2, 8)
        return dict(op="verify", B=_log(rng, 1, 96 // T if steps else 64), T=T, kh=kh, vh=vh, d=128, steps=steps)
    if op == "prefill":
        B = _log(rng, 1, 8)
        return dict(op="prefill", B=B, T=_log(rng, 33, 16384 // B), kh=kh, vh=vh, d=rng.choice([128, 128, 96, 64]),
                    norm=rng.random() < 0.5, state=rng.random() < 0.7)
    if op == "packed":
        n = _log(rng, 2, 32)
        return dict(op="packed", n=n, tokens=_log(rng, 64 * n, 32768), kh=kh, vh=vh, d=128)
    if op == "long":
        B = rng.choice([1, 2])
        return dict(op="prefill", B=B, T=_log(rng, 16384, 131072), kh=2, vh=4, d=128, norm=rng.random() < 0.5, state=rng.random() < 0.7)
    if op == "layer":
        B = rng.choice([1, 1, 2, 4])
        return dict(op="layer", B=B, T=_log(rng, 64, 8192 // B), kh=kh, vh=vh, d=128)
    return dict(op="prefill", B=rng.choice([1, 2]), T=_log(rng, 65, 1500), kh=rng.choice([2, 4]), vh=rng.choice([4, 8]),
                d=rng.choice([256, 256, 192, 200]), norm=rng.random() < 0.5, state=rng.random() < 0.7)


# ------------------------------------------------------------------ inputs
def _init():
    global _ready
    if not _ready:
        gdn.init(os.getcwd(), os.environ.get("CUDA_HOME", "/usr/local/cuda"))
        _ready = True


class _Inputs:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, std=1.0):
        return (torch.randn(*shape, device="cuda", generator=self.g) * std).bfloat16()

    def unit(self, *shape):
        x = torch.randn(*shape, device="cuda", generator=self.g)
        return (x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6)).bfloat16()

    def gate_params(self, vh):
        A_log = torch.log(torch.rand(vh, device="cuda", generator=self.g) * 15.0 + 1.0)
        dt_bias = torch.randn(vh, device="cuda", generator=self.g) * 0.1
        return A_log.bfloat16(), dt_bias.bfloat16()

    def beta_gate(self, *lead, vh):
        A_log, dt_bias = self.gate_params(vh)
        a, b = self.normal(*lead, vh), self.normal(*lead, vh)
        gate = -torch.exp(A_log.float()) * torch.nn.functional.softplus(a.float() + dt_bias.float())
        return torch.sigmoid(b.float()).bfloat16(), gate

    def lengths(self, n, total):
        """n log-normal lengths of at least one token that sum to `total`"""
        x = torch.exp(torch.randn(n, device="cuda", generator=self.g) + 7.0).cpu()
        lens = [max(1, int(v * total / x.sum())) for v in x.tolist()]
        while sum(lens) != total:
            i = max(range(n), key=lens.__getitem__)
            lens[i] += max(1 - lens[i], total - sum(lens))
        return lens


def prepare(case, seed):
    _init()
    r, c = _Inputs(seed), case
    kh, vh, d, op = c["kh"], c["vh"], c["d"], c["op"]
    s = dict(op=op, case=c)
    if op in ("layer", "decode_layer"):
        B, T = c["B"], c.get("T", 1)
        ch = (2 * kh + vh) * d
        s.update(x=r.normal(B, T, ch), z=r.normal(B, T, vh, d), a=r.normal(B, T, vh), b=r.normal(B, T, vh),
                 conv_w=r.normal(ch, 4, std=0.5), norm_w=(1.0 + 0.1 * r.normal(d).float()).bfloat16(),
                 conv_state=r.normal(B, 3, ch), state=r.normal(B, vh, d, d, std=0.02))
        s["A_log"], s["dt_bias"] = r.gate_params(vh)
    elif op in ("decode", "verify"):
        B, T = c["B"], c.get("T", 1)
        s.update(q=r.normal(B, T, kh, d), k=r.normal(B, T, kh, d), v=r.normal(B, T, vh, d), beta=None, gate=None, gating=None)
        if c.get("gating", "inside") == "inside":
            A_log, dt_bias = r.gate_params(vh)
            s["gating"] = (A_log, dt_bias, r.normal(B, T, vh), r.normal(B, T, vh))
        else:
            s["beta"], s["gate"] = r.beta_gate(B, T, vh=vh)
        slots = B + B // 4 + 1 if c.get("where") == "pool" else B
        s["state"] = r.normal(slots, vh, d, d, std=0.02)
        if c.get("state") == "f32":
            s["state"] = s["state"].float()
        if c.get("where") == "pool":
            s["slots"] = torch.randperm(slots, device="cuda", generator=r.g)[:B].int()
        if op == "verify" and not c["steps"]:
            s["accepted"] = torch.randint(1, T + 1, (B,), device="cuda", generator=r.g).int()
    else:
        lead = (c["tokens"],) if op == "packed" else (c["B"], c["T"])
        seqs = c["n"] if op == "packed" else c["B"]
        qk = r.normal if c.get("norm") else r.unit
        s.update(q=qk(*lead, kh, d), k=qk(*lead, kh, d), v=r.normal(*lead, vh, d))
        s["beta"], s["gate"] = r.beta_gate(*lead, vh=vh)
        s["state"] = r.normal(seqs, vh, d, d, std=0.02) if c.get("state", True) else None
        if op == "packed":
            lens = r.lengths(c["n"], c["tokens"])
            cu, cc, ci = [0], [0], []
            for i, n in enumerate(lens):
                nc = (n + CHUNK - 1) // CHUNK
                cu.append(cu[-1] + n)
                cc.append(cc[-1] + nc)
                for j in range(nc):
                    ci += [i, j]
            s["cu"], s["cc"], s["ci"] = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in (cu, cc, ci))
            s["chunks"] = cc[-1]
    return s


# ------------------------------------------------------------------ one pass
def _split(qkv, kh, vh, d):
    return (qkv[..., :kh * d].unflatten(-1, (kh, d)), qkv[..., kh * d:2 * kh * d].unflatten(-1, (kh, d)),
            qkv[..., 2 * kh * d:].unflatten(-1, (vh, d)))


def run(s):
    c, op = s["case"], s["op"]
    if op == "prefill":
        return gdn.chunked_forward(s["q"], s["k"], s["v"], s["beta"], s["gate"], None, s["state"], is_qk_norm=c["norm"])
    if op == "packed":
        return gdn.chunked_forward(s["q"], s["k"], s["v"], s["beta"], s["gate"], None, s["state"], s["cu"], s["ci"], s["cc"], s["chunks"])
    if op == "decode":
        return gdn.recurrent_forward(s["q"], s["k"], s["v"], s["state"], s["beta"], s["gate"], inference_mode=gdn.Decode,
                                     is_qk_norm=True, gating=s["gating"], inplace_state=c["where"] == "inplace",
                                     state_indices=s.get("slots"))
    if op == "verify":
        o, state = gdn.recurrent_forward(s["q"], s["k"], s["v"], s["state"], None, None, None, s.get("accepted"),
                                         gdn.SpecVerify if c["steps"] else gdn.Decode, True, gating=s["gating"])
        # with accepted-token caps the call's purpose is the advanced state; output rows past a cap are not written
        return (o, state) if c["steps"] else state
    kh, vh, d = c["kh"], c["vh"], c["d"]
    if op == "decode_layer":
        qkv, conv_state = gdn.causal_conv1d(s["x"], s["conv_w"], None, s["conv_state"], final_state=s["conv_state"])
        q, k, v = _split(qkv, kh, vh, d)
        o, state = gdn.recurrent_forward(q, k, v, s["state"], None, None, inference_mode=gdn.Decode, is_qk_norm=True,
                                         gating=(s["A_log"], s["dt_bias"], s["a"], s["b"]), inplace_state=True)
    else:
        qkv, conv_state = gdn.causal_conv1d(s["x"], s["conv_w"], None, s["conv_state"], return_final_state=True)
        q, k, v = _split(qkv, kh, vh, d)
        beta, gate = gdn.fused_gdn_gating(s["A_log"], s["dt_bias"], s["a"], s["b"])
        o, state = gdn.chunked_forward(q, k, v, beta, gate, None, s["state"], is_qk_norm=True)
    return gdn.gated_rmsnorm(o, s["z"], s["norm_w"]), state, conv_state


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c = case
    kh, vh, d, op = c["kh"], c["vh"], c["d"], c["op"]
    T = c.get("T", 1)
    tokens = c["tokens"] if op == "packed" else c["B"] * T
    seqs = c["n"] if op == "packed" else c["B"]
    state = vh * d * d * (4 if c.get("state") == "f32" else 2)
    if op in ("decode", "verify", "decode_layer"):
        # the token recurrence: S k, the rank-one update with its decay, S q
        flops = tokens * vh * 7.0 * d * d
        out_states = tokens if c.get("steps") else seqs
    else:
        # the chunked form: five C x C x d and three C x d x d contractions and a triangular inverse per chunk and head
        flops = tokens / CHUNK * vh * (2.0 * CHUNK * (5 * CHUNK * d + 3 * d * d) + 2.0 / 3.0 * CHUNK ** 3)
        out_states = seqs
    nbytes = tokens * vh * (2 + (4 if op in ("prefill", "packed") or c.get("gating") == "given" else 2)) + out_states * state
    nbytes += seqs * state if c.get("state", True) else 0
    if op in ("layer", "decode_layer"):  # projections in, gate z in, result out, the convolution's state in and out
        ch = (2 * kh + vh) * d
        nbytes += tokens * 2 * (ch + 2 * vh * d) + seqs * 2 * 2 * 3 * ch
        flops += tokens * (2.0 * 4 * ch + 10.0 * vh * d)
    else:
        nbytes += tokens * 2 * (2 * kh * d + 2 * vh * d)
    return {"bytes": float(nbytes), "flops": flops}


def tolerance(case):
    # bf16 results; inside the chunked form the operands of the matrix products are bf16 as well
    return {"rel": 1e-2, "max": 0.25}
