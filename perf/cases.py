"""The work a training or evaluation program has this framework do, as timed cases.

A case is one call, or one forward + backward, through a public entry point: the ops that the
hybrid models are made of (``nsa_optim_b200.ops``), the MLP module, the optimizer and a whole model.
``listed()`` gives one case per kind of work, from a few microseconds to the long sequences the
framework is for; ``draw()`` gives other sizes of the same kinds.

Shapes are those of the models this repository configures: the 1B hybrid (d_model 2048, FFN 5632,
vocabulary 32000, 32 query / 2 KV heads of 128, Mamba-2 with 64 heads of 64 and d_state 128,
Gated DeltaNet with 16 heads of 128 / 256) and its smaller and wider relatives.  Activations and
weights are bf16, gates and step sizes fp32, as the models pass them.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from nsa_optim_b200 import ops
from nsa_optim_b200.models.hybrid import HybridConfig, create_hybrid_model
from nsa_optim_b200.models.kernels import MLP
from nsa_optim_b200.optimizers import AdamW, AdamWLowBit

DEV = "cuda"
BF = torch.bfloat16


def listed():
    return [
        # evaluation of a short prompt batch: two sequences of odd length, no gradient
        dict(name="attention_eval_short", kind="attention", B=2, T=300, Hq=16, Hkv=8, D=64, window=0, train=False),
        # the dense attention layer of a training step at 8K context
        dict(name="attention_train_8k", kind="attention", B=1, T=8192, Hq=32, Hkv=2, D=128, window=0, train=True),
        # the sparse attention layer of the 1B hybrid (compressed + selected + window) at 16K
        dict(name="nsa_train_16k", kind="nsa", B=1, T=16384, Hq=32, Hkv=2, D=128),
        # the Mamba-2 scan of the 1B hybrid, one layer
        dict(name="ssd_train_16k", kind="ssd", B=1, T=16384, H=64),
        # the Gated DeltaNet recurrence of the 1B hybrid, one layer
        dict(name="gdn_train_16k", kind="gdn", B=1, T=16384, H=16),
        # the causal convolution in front of the Mamba-2 scan, on a column slice of the in-projection
        dict(name="conv_train_16k", kind="conv", B=1, T=16384, C=4352, pitch=8512, bias=True),
        # residual add + norm between the mixer and the MLP of a block
        dict(name="add_norm_train", kind="norm", mode="add", rows=16384, d=2048),
        # the SwiGLU MLP of a block
        dict(name="mlp_train", kind="mlp", rows=8192, d=2048, f=5632),
        # the output head and loss
        dict(name="head_train", kind="head", rows=8192, d=2048, V=32000),
        # the optimizer step over the weights of a few blocks, 8-bit state
        dict(name="adamw8bit_step", kind="adamw", bits=8, d=2048, f=5632, blocks=2),
        # the optimizer step of a small model with fp32 state and master weights
        dict(name="adamw_master_step", kind="adamw", bits=32, d=768, f=2048, blocks=2),
        # evaluation logits of a small three-block hybrid on a short context
        dict(name="hybrid_logits", kind="model", B=1, T=1000, d=1024, pattern="MDA", V=32000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "nsa", "ssd", "gdn", "conv", "norm", "mlp", "head", "adamw", "model"])
    if kind == "attention":
        Hq, Hkv, D = rng.choice([(32, 2, 128), (16, 8, 128), (32, 8, 128), (16, 2, 128), (16, 8, 64), (8, 2, 64)])
        T = _log(rng, 64, 8192)
        B = rng.choice([1, 2, 4])
        while B > 1 and B * T > 8192:
            B //= 2
        return dict(kind=kind, B=B, T=T, Hq=Hq, Hkv=Hkv, D=D, window=rng.choice([0, 0, 512]), train=rng.random() < 0.7)
    if kind == "nsa":
        Hq, Hkv, D = rng.choice([(32, 2, 128), (16, 2, 128), (32, 4, 128)])
        return dict(kind=kind, B=1, T=_log(rng, 512, 16384), Hq=Hq, Hkv=Hkv, D=D)
    if kind == "ssd":
        T = _log(rng, 100, 16384)
        return dict(kind=kind, B=rng.choice([1, 2]) if T <= 8192 else 1, T=T, H=rng.choice([24, 32, 48, 64]))
    if kind == "gdn":
        T = _log(rng, 100, 16384)
        return dict(kind=kind, B=rng.choice([1, 2]) if T <= 8192 else 1, T=T, H=rng.choice([4, 8, 16]))
    if kind == "conv":
        T, C = _log(rng, 100, 16384), 8 * _log(rng, 96, 544)
        return dict(kind=kind, B=rng.choice([1, 2]) if T <= 8192 else 1, T=T, C=C,
                    pitch=rng.choice([C, C + 4160]), bias=rng.random() < 0.5)
    if kind == "norm":
        mode = rng.choice(["plain", "add", "gated_before", "gated_after"])
        d = rng.choice([256, 768, 1024, 1536, 2048, 2560, 4096])
        return dict(kind=kind, mode=mode, rows=min(_log(rng, 64, 65536), 16384 * 2048 // d), d=d)
    if kind == "mlp":
        d = rng.choice([768, 1024, 1536, 2048])
        return dict(kind=kind, rows=_log(rng, 64, 8192), d=d, f=64 * math.ceil(d * 8 / 3 / 64))
    if kind == "head":
        return dict(kind=kind, rows=_log(rng, 128, 8192), d=rng.choice([768, 1024, 1536, 2048]), V=32000)
    if kind == "adamw":
        d = rng.choice([512, 768, 1024, 1536, 2048])
        return dict(kind=kind, bits=rng.choice([8, 8, 32]), d=d, f=64 * math.ceil(d * 8 / 3 / 64), blocks=rng.choice([1, 2]))
    return dict(kind=kind, B=rng.choice([1, 2]), T=_log(rng, 64, 2048), d=rng.choice([512, 1024]),
                pattern=rng.choice(["MDA", "MA", "DA", "AM"]), V=32000)


# ------------------------------------------------------------------------------------- inputs
class _Draws:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=BF):
        return (torch.randn(*shape, generator=self.g, device=DEV) * std).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(*shape, generator=self.g, device=DEV) * (hi - lo) + lo


def _step_sizes(r, B, T, H):
    """softplus(dt + bias) with the bias log-uniform in [1e-3, 1e-1] per head, and A = -U(1, 16)."""
    dt0 = torch.exp(r.uniform(H, lo=math.log(1e-3), hi=math.log(1e-1)))
    bias = dt0 + torch.log(-torch.expm1(-dt0))
    return F.softplus(r.normal(B, T, H, dtype=torch.float32) * 0.5 + bias), -r.uniform(H, lo=1.0, hi=16.0)


def _weight_shapes(case):
    """The parameters of a Mamba-2 block and its MLP: projections, convolution, norms, per-head vectors."""
    d, f = case["d"], case["f"]
    heads = 2 * d // 64
    one = [(4 * d + 256 + heads, d), (d, 2 * d), (f, d), (f, d), (d, f), (2 * d + 256, 1, 4), (2 * d + 256,), (2 * d,),
           (d,), (d,), (heads,), (heads,), (heads,)]
    return one * case["blocks"]


def _model_config(case):
    d = case["d"]
    return HybridConfig(d_model=d, vocab_size=case["V"], block_pattern=case["pattern"], block_repeats=1,
                        deltanet_head_dim=128, num_attention_heads=d // 128, num_key_value_heads=2, head_dim=128,
                        max_position_embeddings=4096)


def prepare(case, seed):
    r, k = _Draws(seed), case["kind"]
    s = dict(case=case)
    if k in ("attention", "nsa"):
        B, T, Hq, Hkv, D = (case[n] for n in ("B", "T", "Hq", "Hkv", "D"))
        s["in"] = [r.normal(B, T, Hq, D), r.normal(B, T, Hkv, D), r.normal(B, T, Hkv, D)]
        if k == "nsa":
            s["in"].append(r.normal(B, T, 3 * Hq))
        s["dy"] = r.normal(B, T, Hq, D)
    elif k == "ssd":
        # x, B and C are the column groups of the convolution's output, as in the mixer
        B, T, H = case["B"], case["T"], case["H"]
        xbc = F.silu(r.normal(B, T, H * 64 + 256))
        dt, A = _step_sizes(r, B, T, H)
        s["in"] = [xbc[..., :H * 64].view(B, T, H, 64), dt, A, xbc[..., H * 64:H * 64 + 128].view(B, T, 1, 128),
                   xbc[..., H * 64 + 128:].view(B, T, 1, 128), 1 + 0.1 * r.normal(H, dtype=torch.float32)]
        # with a common component: per-head sums over all tokens (dA) would otherwise be cancellation alone
        s["dy"] = r.normal(B, T, H, 64) + 0.5
    elif k == "gdn":
        B, T, H = case["B"], case["T"], case["H"]
        unit = lambda t: F.normalize(t.float(), dim=-1).to(BF)  # noqa: E731
        dt, A = _step_sizes(r, B, T, H)
        s["in"] = [unit(F.silu(r.normal(B, T, H, 128))), unit(F.silu(r.normal(B, T, H, 128))),
                   F.silu(r.normal(B, T, H, 256)), A * dt, torch.sigmoid(r.normal(B, T, H, dtype=torch.float32))]
        s["dy"] = r.normal(B, T, H, 256)
    elif k == "conv":
        B, T, C = case["B"], case["T"], case["C"]
        off = 0 if case["pitch"] == C else (case["pitch"] - C) // 16 * 8
        s["in"] = [r.normal(B, T, case["pitch"])[..., off:off + C], r.normal(C, 4, std=0.3)]
        if case["bias"]:
            s["in"].append(r.normal(C, std=0.3))
        s["dy"] = r.normal(B, T, C)
    elif k == "norm":
        n, d = case["rows"], case["d"]
        s["in"] = [r.normal(n, d), 1 + 0.1 * r.normal(d)]
        if case["mode"] != "plain":
            s["in"].insert(1, r.normal(n, d))
        s["dy"] = r.normal(n, d)
        s["dh"] = r.normal(n, d)
    elif k == "mlp":
        n, d, f = case["rows"], case["d"], case["f"]
        with torch.device("meta"):
            m = MLP(d, f)
        m = m.to(BF).to_empty(device=DEV)
        for p in m.parameters():
            p.data = r.normal(*p.shape, std=0.02)
        s["mlp"], s["in"], s["dy"] = m, [r.normal(n, d)], r.normal(n, d)
    elif k == "head":
        n, d, V = case["rows"], case["d"], case["V"]
        s["in"] = [r.normal(n, d), r.normal(V, d, std=0.02)]
        s["labels"] = torch.randint(0, V, (n,), generator=r.g, device=DEV)
        s["labels"][::50] = -100
    elif k == "adamw":
        params = [torch.nn.Parameter(r.normal(*sh, std=0.02)) for sh in _weight_shapes(case)]
        s["opt"] = (AdamWLowBit(params, lr=1e-4, weight_decay=0.1, bits=8) if case["bits"] == 8
                    else AdamW(params, lr=1e-4, weight_decay=0.1, master_weights=True))
        s["in"] = params
        for _ in range(2):                       # a program is in the middle of training: the state is not zero
            for p in params:
                p.grad = r.normal(*p.shape, std=1e-3)
            s["opt"].step()
        for p in params:
            p.grad = r.normal(*p.shape, std=1e-3)
    else:
        torch.manual_seed(seed)
        with torch.device(DEV):
            m = create_hybrid_model(_model_config(case))
        s["model"] = m.to(BF).eval()
        s["ids"] = torch.randint(0, case["V"], (case["B"], case["T"]), generator=r.g, device=DEV)
    if k not in ("adamw", "model") and case.get("train", True):
        s["in"] = [t.detach().requires_grad_() for t in s["in"]]
    return s


# ------------------------------------------------------------------------------------- one pass
def _gate_before(case):
    return case["mode"] == "gated_before"


def run(s):
    case, k = s["case"], s["case"]["kind"]
    if k == "adamw":
        s["opt"].step()
        out = []
        for p in s["in"][:13]:                   # every kind of parameter; all are updated
            st = s["opt"].state[p]
            out += [p.detach()] + [st[n] for n in ("exp_avg", "exp_avg_sq", "master") if n in st and p.dim() == 2]
        return out
    if k == "model":
        with torch.no_grad():
            return s["model"](s["ids"])[0]
    x = s["in"]
    if k == "attention":
        if not case["train"]:
            with torch.no_grad():
                return ops.attention(*x, causal=True, window=case["window"])
        y = ops.attention(*x, causal=True, window=case["window"])
    elif k == "nsa":
        y = ops.nsa_attention(*x[:3], None, None, None, gate_logits=x[3])
    elif k == "ssd":
        y = ops.ssd_scan(*x)
    elif k == "gdn":
        y = ops.gated_delta_rule(*x)
    elif k == "conv":
        y = ops.causal_conv1d(x[0], x[1], x[2] if case["bias"] else None)
    elif k == "norm":
        if case["mode"] == "add":
            h, y = ops.add_rms_norm(*x)
            return [h.detach(), y.detach()] + list(torch.autograd.grad([h, y], [x[0], x[2]], [s["dh"], s["dy"]]))
        y = ops.rms_norm(*x) if case["mode"] == "plain" else ops.gated_rms_norm(*x, norm_before_gate=_gate_before(case))
    elif k == "mlp":
        y = s["mlp"](x[0])
        x = x + list(s["mlp"].parameters())
    else:
        loss = ops.linear_cross_entropy(x[0], x[1], s["labels"])
        return [loss.detach()] + list(torch.autograd.grad(loss, x))
    return [y.detach()] + list(torch.autograd.grad(y, x, s["dy"]))


# ------------------------------------------------------------------------------------- cost and accuracy
def _pairs(T, window=0):
    """Query-key pairs of a causal sequence."""
    if window and window < T:
        return window * (window + 1) // 2 + (T - window) * window
    return T * (T + 1) // 2


def work(case):
    k = case["kind"]
    if k in ("attention", "nsa"):
        B, T, Hq, Hkv, D = (case[n] for n in ("B", "T", "Hq", "Hkv", "D"))
        q, kv = B * T * Hq * D * 2, B * T * Hkv * D * 2
        train = case.get("train", True)
        bytes_ = 2 * q + 2 * kv + (2 * q + 2 * kv if train else 0)
        if k == "attention":
            return dict(bytes=bytes_, flops=B * Hq * D * _pairs(T, case["window"]) * (14 if train else 4))
        nc = max(0, (T - 32) // 16 + 1)
        cmp_ = nc * (T - 31) - 16 * nc * (nc - 1) // 2
        sel = min(T, 1024)
        sel = sel * (sel + 1) // 2 + (T - sel) * 1024 if T > sel else _pairs(T)
        return dict(bytes=bytes_, flops=B * Hq * D * 14 * (cmp_ + sel + _pairs(T, 512)))
    if k in ("ssd", "gdn"):
        n = case["B"] * case["T"]
        if k == "ssd":
            H = case["H"]
            # state update and read-out, forward and backward: 128 x 64 state per head
            return dict(bytes=n * (H * 64 * 2 * 4 + 128 * 2 * 4 + H * 4 * 2), flops=n * H * 128 * 64 * 4 * 3)
        H = case["H"]
        return dict(bytes=n * H * (128 * 2 * 4 + 256 * 2 * 4 + 4 * 4), flops=n * H * 128 * 256 * 6 * 3)
    if k == "conv":
        return dict(bytes=case["B"] * case["T"] * case["C"] * 2 * 4, flops=case["B"] * case["T"] * case["C"] * 40)
    if k == "norm":
        n = case["rows"] * case["d"]
        tensors = {"plain": 4, "add": 7, "gated_before": 6, "gated_after": 6}[case["mode"]]
        return dict(bytes=n * 2 * tensors, flops=n * 12)
    if k == "mlp":
        n, d, f = case["rows"], case["d"], case["f"]
        return dict(bytes=2 * (4 * n * d + 2 * 3 * d * f), flops=2 * n * d * f * 9)
    if k == "head":
        n, d, V = case["rows"], case["d"], case["V"]
        return dict(bytes=2 * (2 * n * d + 2 * V * d), flops=2 * n * d * V * 3)
    if k == "adamw":
        n = sum(math.prod(sh) for sh in _weight_shapes(case))
        return dict(bytes=n * (10 if case["bits"] == 8 else 28), flops=n * 20)
    d, V, n = case["d"], case["V"], case["B"] * case["T"]
    f = 64 * math.ceil(int(d * 8 / 3) / 64)
    per = {"M": d * (4 * d + 256 + d // 32) + 2 * d * d, "D": 2 * d * d + 2 * d * 2 * d + 2 * d * d + 2 * d * (d // 128),
           "A": 2 * d * d + 2 * d * 256}
    w = sum(per[c] + 3 * d * f for c in case["pattern"]) + V * d
    return dict(bytes=2 * w + 2 * n * V, flops=2 * n * w)


def tolerance(case):
    k = case["kind"]
    if k == "adamw":
        return {"rel": 2e-3, "max": 0.1, "differ": 1e-3}
    # measured against 64 bits: 0.002 to 0.005 for one op in bf16, 0.004 for the three sparse branches,
    # 0.008 for a whole model; two implementations differ by up to the sum of their errors
    return {"rel": {"model": 2.5e-2, "nsa": 1.6e-2}.get(k, 1e-2), "max": 0.5}


# ------------------------------------------------------------------------------------- 64-bit results
class _Attend64(torch.autograd.Function):
    """One head: softmax(q k^T scale, masked) v with the probabilities recomputed in the backward."""

    @staticmethod
    def forward(ctx, q, k, v, mask, scale):
        p = _probs64(q, k, mask, scale)
        ctx.save_for_backward(q, k, v, mask)
        ctx.scale = scale
        return p @ v

    @staticmethod
    def backward(ctx, do):
        q, k, v, mask = ctx.saved_tensors
        p = _probs64(q, k, mask, ctx.scale)
        dv = p.t() @ do
        ds = do @ v.t()
        ds = (ds - (ds * p).sum(-1, keepdim=True)).mul_(p).mul_(ctx.scale)
        return ds @ k, ds.t() @ q, dv, None, None


def _probs64(q, k, mask, scale):
    p = (q @ k.t()).mul_(scale).masked_fill_(~mask, -math.inf)
    p = p.sub_(p.amax(-1, keepdim=True).clamp_min(-1e300)).exp_()
    return p.div_(p.sum(-1, keepdim=True).clamp_min(1e-300))


def _causal(T, window=0):
    t = torch.arange(T, device=DEV)
    m = t[None, :] <= t[:, None]
    return m & (t[None, :] > t[:, None] - window) if window else m


def _attention64(q, k, v, window=0):
    B, T, Hq, D = q.shape
    G, mask = Hq // k.shape[2], _causal(T, window)
    return torch.stack([torch.stack([_Attend64.apply(q[b, :, h], k[b, :, h // G], v[b, :, h // G], mask, D ** -0.5)
                                     for h in range(Hq)], 1) for b in range(B)])


def _nsa64(q, k, v, logits):
    """Compressed (mean of 32 every 16, kept in bf16 like the tensors it pools), selected (16 blocks of
    64: the first, the query's own, the one before it and the most important) and window (512) branches."""
    B, T, Hq, D = q.shape
    G, sc = Hq // k.shape[2], D ** -0.5
    nS, t = -(-T // 64), torch.arange(T, device=DEV)
    pool = lambda x: x.unfold(0, 32, 16).mean(-1)                                    # noqa: E731
    near = lambda x: x + (x.to(BF).double() - x).detach()                            # noqa: E731
    swa = _causal(T, 512)
    outs = []
    for b in range(B):
        heads = []
        for g in range(k.shape[2]):
            kk, vv = k[b, :, g], v[b, :, g]
            kc, vc = near(pool(kk)), near(pool(vv))
            start = torch.arange(kc.shape[0], device=DEV) * 16
            vis = (start + 31)[None, :] <= t[:, None]
            with torch.no_grad():
                p = sum(_probs64(q[b, :, h], kc, vis, sc) for h in range(g * G, (g + 1) * G))
                lo, hi = torch.arange(nS, device=DEV) * 64, torch.arange(nS, device=DEV) * 64 + 64
                share = (torch.minimum(hi[None], start[:, None] + 32) - torch.maximum(lo[None], start[:, None])).clamp_min(0) / 16
                imp = p @ share.double()
                own, j = (t // 64)[:, None], torch.arange(nS, device=DEV)[None]
                imp = imp.masked_fill((j == 0) | (j == own) | (j == own - 1), math.inf).masked_fill(j > own, -math.inf)
                top = imp.sort(dim=-1, descending=True, stable=True)
                blk = torch.zeros(T, nS, dtype=torch.bool, device=DEV)
                blk.scatter_(1, top.indices[:, :16], top.values[:, :16] > -math.inf)
                slc = blk.repeat_interleave(64, 1)[:, :T] & _causal(T)
            for h in range(g * G, (g + 1) * G):
                qq, gate = q[b, :, h], torch.sigmoid(logits[b])
                heads.append(gate[:, h, None] * _Attend64.apply(qq, kc, vc, vis, sc)
                             + gate[:, Hq + h, None] * _Attend64.apply(qq, kk, vv, slc, sc)
                             + gate[:, 2 * Hq + h, None] * _Attend64.apply(qq, kk, vv, swa, sc))
        outs.append(torch.stack(heads, 1))
    return torch.stack(outs)


def _chunks(t, C):
    """(B, T, ...) -> (B, n, C, ...), zero-padded."""
    pad = -t.shape[1] % C
    if pad:
        t = torch.cat([t, t.new_zeros(t.shape[0], pad, *t.shape[2:])], 1)
    return t.reshape(t.shape[0], -1, C, *t.shape[2:])


def _decay64(cum):
    """exp(cum_i - cum_j) for i >= j, else 0, over the last dimension."""
    C = cum.shape[-1]
    keep = torch.ones(C, C, dtype=torch.bool, device=cum.device).tril()
    return (cum[..., :, None] - cum[..., None, :]).masked_fill(~keep, -math.inf).exp()


def _ssd64(x, dt, A, Bm, Cm, D):
    T, C = x.shape[1], 64
    xc, dc, Bc, Cc = (_chunks(t, C) for t in (x * dt[..., None], dt, Bm[:, :, 0], Cm[:, :, 0]))
    cum = (dc * A).cumsum(2).transpose(2, 3)                                          # (B, n, H, C)
    y = torch.einsum("bnis,bnjs,bnhij,bnjhp->bnihp", Cc, Bc, _decay64(cum), xc)
    h, ys = x.new_zeros(x.shape[0], x.shape[2], 128, 64), []
    new = torch.einsum("bnjs,bnhj,bnjhp->bnhsp", Bc, (cum[..., -1:] - cum).exp(), xc)
    for n in range(xc.shape[1]):
        ys.append(torch.einsum("bis,bhi,bhsp->bihp", Cc[:, n], cum[:, n].exp(), h))
        h = cum[:, n, :, -1].exp()[..., None, None] * h + new[:, n]
    return (y + torch.stack(ys, 1)).flatten(1, 2)[:, :T] + x * D[:, None]


def _gdn64(q, k, v, g, beta):
    T, C = q.shape[1], 64
    q, k, v, g, beta = (_chunks(t, C).transpose(2, 3) for t in (q * 128 ** -0.5, k, v, g, beta))   # (B, n, H, C, .)
    cum = g.cumsum(-1)
    dec, eg = _decay64(cum), cum.exp()[..., None]
    kk = k @ k.transpose(-1, -2)
    A = (beta[..., None] * kk * dec).tril(-1) + torch.eye(C, device=DEV, dtype=q.dtype)
    uw = torch.linalg.solve_triangular(A, beta[..., None] * torch.cat([v, k * eg], -1), upper=False, unitriangular=True)
    u, w = uw.split([v.shape[-1], k.shape[-1]], -1)
    qk, tail = (q @ k.transpose(-1, -2)) * dec, k * (cum[..., -1:] - cum).exp()[..., None]
    S, out = q.new_zeros(q.shape[0], q.shape[2], q.shape[-1], v.shape[-1]), []
    for n in range(q.shape[1]):
        new = u[:, n] - w[:, n] @ S
        out.append((q[:, n] * eg[:, n]) @ S + qk[:, n] @ new)
        S = eg[:, n, :, -1:] * S + tail[:, n].transpose(-1, -2) @ new
    return torch.stack(out, 1).transpose(2, 3).flatten(1, 2)[:, :T]


def _conv64(x, w, bias):
    T = x.shape[1]
    xp = F.pad(x, (0, 0, 3, 0))
    y = sum(xp[:, i:i + T] * w[:, i] for i in range(4))
    return F.silu(y if bias is None else y + bias)


def _rms64(x, w, eps=1e-6):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt() * w


def _rope64(x, theta):
    T, D = x.shape[1], x.shape[-1]
    inv = theta ** (-torch.arange(0, D, 2, device=DEV, dtype=torch.float64) / D)
    a = (torch.arange(T, device=DEV)[:, None] * inv)[None, :, None]
    x1, x2 = x.chunk(2, -1)
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin()], -1)


def _model64(case, w, ids):
    d = case["d"]
    h = w["embed_tokens.weight"][ids]
    B, T = ids.shape
    unit = lambda t: t * (t.square().sum(-1, keepdim=True) + 1e-6).rsqrt()            # noqa: E731
    for i, c in enumerate(case["pattern"]):
        p = lambda n, i=i: w["layers.%d.%s" % (i, n)]                                  # noqa: E731
        u = _rms64(h, p("norm.weight"))
        if c == "M":
            H = 2 * d // 64
            z, xbc, dt = (u @ p("mixer.in_proj.weight").t()).split([2 * d, 2 * d + 256, H], -1)
            xbc = _conv64(xbc, p("mixer.conv1d.weight")[:, 0], p("mixer.conv1d.bias"))
            x, Bm, Cm = xbc.split([2 * d, 128, 128], -1)
            y = _ssd64(x.reshape(B, T, H, 64), F.softplus(dt + p("mixer.dt_bias")), -p("mixer.A_log").exp(), Bm[:, :, None],
                       Cm[:, :, None], p("mixer.D"))
            y = _rms64(y.reshape(B, T, 2 * d) * F.silu(z), p("mixer.norm.weight"), 1e-5) @ p("mixer.out_proj.weight").t()
        elif c == "D":
            H = d // 128
            proj = lambda n: _conv64(u @ p("mixer.%s_proj.weight" % n).t(), p("mixer.%s_conv1d.weight" % n)[:, 0], None)  # noqa: E731,B023
            q, k, v = proj("q").view(B, T, H, 128), proj("k").view(B, T, H, 128), proj("v").view(B, T, H, 256)
            g = -p("mixer.A_log").exp() * F.softplus(u @ p("mixer.a_proj.weight").t() + p("mixer.dt_bias"))
            o = _gdn64(unit(q), unit(k), v, g, torch.sigmoid(u @ p("mixer.b_proj.weight").t()))
            o = _rms64(o, p("mixer.o_norm.weight"), 1e-5) * F.silu((u @ p("mixer.g_proj.weight").t()).view(B, T, H, 256))
            y = o.reshape(B, T, -1) @ p("mixer.o_proj.weight").t()
        else:
            q, k, v = ((u @ p(n + "_proj.weight").t()).view(B, T, -1, 128) for n in "qkv")
            y = _attention64(_rope64(q, 100000.0), _rope64(k, 100000.0), v).reshape(B, T, -1) @ p("o_proj.weight").t()
        h = h + y
        u = _rms64(h, p("post_attn_norm.weight" if c == "A" else "post_mixer_norm.weight"))
        h = h + (F.silu(u @ p("mlp.gate_proj.weight").t()) * (u @ p("mlp.up_proj.weight").t())) @ p("mlp.down_proj.weight").t()
    return _rms64(h, w["norm.weight"]) @ w["lm_head.weight"].t()


def _codebook64(signed, device):
    """The 256-entry dynamic map: per decade 10^(i-6), 2^i (2^(i+1) unsigned) midpoints of a uniform
    grid over [0.1, 1], mirrored when signed, plus 0 and 1."""
    vals = [0.0, 1.0]
    for i in range(7):
        n = 2 ** i if signed else 2 ** (i + 1)
        mids = [10.0 ** (i - 6) * (0.1 + 0.9 * (j + 0.5) / n) for j in range(n)]
        vals += mids + ([-m for m in mids] if signed else [])
    return torch.tensor(sorted(vals + [0.0] * (256 - len(vals))), dtype=torch.float64, device=device)


def _adamw64(s):
    lr, b1, b2, eps, wd, out = 1e-4, 0.9, 0.95, 1e-8, 0.1, []
    for p in s["in"][:13]:
        st = s["opt"].state[p]
        m, v = st["exp_avg"], st["exp_avg_sq"]
        quantised = m.dtype == torch.uint8
        if quantised:
            m = (_codebook64(True, DEV)[m.long()].view(-1, 256) * st["exp_avg_absmax"].double()[:, None]).view(p.shape)
            v = (_codebook64(False, DEV)[v.long()].view(-1, 256) * st["exp_avg_sq_absmax"].double()[:, None]).view(p.shape)
        t, gr = st["step"] + 1, p.grad.double()
        w = st["master"].double() if "master" in st else p.detach().double()
        m, v = b1 * m.double() + (1 - b1) * gr, b2 * v.double() + (1 - b2) * gr * gr
        w = w * (1 - lr * wd) - lr / (1 - b1 ** t) * m / (v.sqrt() / math.sqrt(1 - b2 ** t) + eps)
        out.append(w)
        if p.dim() == 2:
            out += [None, None] if quantised else [m, v] + ([w] if "master" in st else [])
    return out


def exact(case, seed):
    s, k = prepare(case, seed), case["kind"]
    if k == "adamw":
        return _adamw64(s)
    if k == "model":
        with torch.no_grad():
            return _model64(case, {n: t.double() for n, t in s["model"].state_dict().items()}, s["ids"])
    x = [t.detach().double().requires_grad_(t.requires_grad) for t in s["in"]]
    dy = s["dy"].double() if "dy" in s else None
    if k == "attention":
        y = _attention64(*x, window=case["window"])
        if not case["train"]:
            return y
    elif k == "nsa":
        y = _nsa64(*x)
    elif k == "ssd":
        y = _ssd64(*x)
    elif k == "gdn":
        y = _gdn64(*x)
    elif k == "conv":
        y = _conv64(x[0], x[1], x[2] if case["bias"] else None)
    elif k == "norm":
        if case["mode"] == "add":
            h = x[0] + x[1]
            y = _rms64(h, x[2])
            return [h.detach(), y.detach()] + list(torch.autograd.grad([h, y], [x[0], x[2]], [s["dh"].double(), dy]))
        if case["mode"] == "plain":
            y = _rms64(*x)
        else:
            y = _rms64(x[0], x[2]) * F.silu(x[1]) if _gate_before(case) else _rms64(x[0] * F.silu(x[1]), x[2])
    elif k == "mlp":
        x += [p.detach().double().requires_grad_() for p in s["mlp"].parameters()]
        y = (F.silu(x[0] @ x[1].t()) * (x[0] @ x[2].t())) @ x[3].t()
    else:
        loss = F.cross_entropy(x[0] @ x[1].t(), s["labels"], ignore_index=-100)
        return [loss.detach()] + list(torch.autograd.grad(loss, x))
    return [y.detach()] + list(torch.autograd.grad(y, x, dy))
