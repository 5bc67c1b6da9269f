"""Performance cases: the work that programs built on this backend spend their time in, each through a public entry
point -- the layers of a Llama-style decoder in training (one block, its attention, its feed-forward, the loss), prompt
processing and graph-captured decoding, packed variable-length attention, the experts of a mixture-of-experts layer, an
fp8 linear layer and a convolution of ResNet-50 with its batch norm.

``listed()`` has the fixed cases, ``draw(rng)`` another one of the same ranges.  ``prepare`` builds what a program holds
before the call, ``run`` makes one pass, ``work`` counts the bytes and operations that pass cannot do without,
``exact`` gives the outputs in 64 bits from plain PyTorch, ``tolerance`` how far another correct implementation at the
same precision may be off.
"""
import math

import torch
import torch.nn.functional as F

import torch_musa_b200 as bw  # noqa: F401  (registers the device)
from torch_musa_b200.models import Llama, LlamaConfig
from torch_musa_b200.models.decode import LlamaDecoder
from torch_musa_b200.models.llama import Block, FeedForward, RopeTables
from torch_musa_b200.models.moe import Experts
from torch_musa_b200.ops import functional as BF

DEV = "blackwell"
BF16 = torch.bfloat16
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
# the dimensions of this repository's configurations: Llama-7B, the mixture-of-experts decoder's attention and experts
DIM, HEADS, FFN, VOCAB, HD = 4096, 32, 11008, 32000, 128
MOE_KV, MOE_FFN = 8, 14336


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # residual add + RMS norm of one decode step's rows: the smallest calls a server makes, launch latency counts
        {"name": "norm_decode_rows", "kind": "norm", "rows": 32, "dim": DIM, "train": False},
        # the norm in front of every block of a training step at sequence length 4096
        {"name": "norm_train", "kind": "norm", "rows": 4096, "dim": DIM, "train": True},
        # attention of the headline training step: one sequence of 4096, causal
        {"name": "attn_train_4096", "kind": "attn", "B": 1, "Sq": 4096, "H": 32, "Hkv": 32, "causal": True, "dtype": "bf16", "train": True},
        # prompt processing with grouped-query heads, a ragged prompt length, fp16
        {"name": "attn_prefill_1531_gqa", "kind": "attn", "B": 4, "Sq": 1531, "H": 32, "Hkv": 8, "causal": True, "dtype": "fp16", "train": False},
        # a packed batch of documents of mixed lengths in training (grouped-query heads)
        {"name": "varlen_train_mixed", "kind": "varlen", "lens": "4096,1024,3000,72", "H": 32, "Hkv": 8, "causal": True, "train": True},
        # feed-forward of the training step: the three largest GEMMs of a layer in every direction
        {"name": "mlp_train_4096", "kind": "mlp", "tokens": 4096, "dim": DIM, "ffn": FFN, "train": True},
        # one whole decoder block in training on a batch whose length is no multiple of anything
        {"name": "block_train_2x1000", "kind": "block", "B": 2, "S": 1000, "Hkv": 32, "ffn": FFN},
        # the loss over the 32000-word vocabulary, forward and backward
        {"name": "loss_train_4096", "kind": "loss", "rows": 4096, "vocab": VOCAB},
        # one token for 32 sequences with 2048 keys each, replayed from the captured graph (two layers and the head)
        {"name": "decode_32x2048", "kind": "decode", "B": 32, "kv": 2048, "layers": 2, "Hkv": 32, "ffn": FFN},
        # the experts of one expert-parallel rank in training: ragged groups, counts on the device
        {"name": "experts_train", "kind": "experts", "counts": "2300,1900,2200,1792", "ffn": MOE_FFN, "train": True},
        # an fp8 linear layer: 1 x 128 quantisation of the activations and the block-scaled product
        {"name": "fp8_linear_4096", "kind": "fp8", "rows": 4096, "n": 14336, "k": 4096},
        # a 3x3 convolution of ResNet-50's second stage with its batch norm, in training under bf16 autocast, channels last.  No
        # ReLU: where a pre-activation rounds to the other side of zero, a ReLU lets one whole gradient value through or not,
        # and no tolerance on single values could be stated.
        {"name": "conv3x3_bn_train_256", "kind": "conv", "B": 256, "cin": 128, "cout": 128, "size": 28, "k": 3, "stride": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["norm", "attn", "varlen", "mlp", "block", "loss", "decode", "experts", "fp8", "conv"])
    if kind == "norm":
        return {"kind": kind, "rows": _log_int(rng, 1, 8192), "dim": rng.choice([1024, 2048, DIM, 8192]), "train": rng.random() < 0.5}
    if kind == "attn":
        s = _log_int(rng, 96, 4096)
        return {"kind": kind, "B": max(1, min(8, 4096 // s)), "Sq": s, "H": 32, "Hkv": rng.choice([8, 32]),
                "causal": rng.random() < 0.75, "dtype": rng.choice(["bf16", "bf16", "fp16"]), "train": rng.random() < 0.6}
    if kind == "varlen":
        lens = [_log_int(rng, 24, 4096) for _ in range(rng.randint(2, 6))]
        while sum(lens) > 8192:
            lens.pop()
        return {"kind": kind, "lens": ",".join(map(str, lens)), "H": 32, "Hkv": rng.choice([8, 32]), "causal": rng.random() < 0.75,
                "train": rng.random() < 0.6}
    if kind == "mlp":
        return {"kind": kind, "tokens": _log_int(rng, 1, 6000), "dim": DIM, "ffn": rng.choice([FFN, MOE_FFN]), "train": rng.random() < 0.5}
    if kind == "block":
        s = _log_int(rng, 128, 2500)
        return {"kind": kind, "B": rng.randint(1, max(1, min(4, 2500 // s))), "S": s, "Hkv": rng.choice([MOE_KV, HEADS]), "ffn": FFN}
    if kind == "loss":
        return {"kind": kind, "rows": _log_int(rng, 64, 6000), "vocab": rng.choice([VOCAB, VOCAB, 50257, 4001])}
    if kind == "decode":
        kv = _log_int(rng, 64, 4000)
        return {"kind": kind, "B": max(1, min(_log_int(rng, 1, 64), 65536 // kv)), "kv": kv, "layers": 2, "Hkv": rng.choice([MOE_KV, HEADS]),
                "ffn": rng.choice([FFN, MOE_FFN])}
    if kind == "experts":
        n = _log_int(rng, 64, 2000)
        return {"kind": kind, "counts": ",".join(str(rng.randint(n // 2, n)) for _ in range(rng.choice([2, 4]))), "ffn": MOE_FFN,
                "train": rng.random() < 0.6}
    if kind == "fp8":
        return {"kind": kind, "rows": _log_int(rng, 16, 6000), "n": rng.choice([4096, FFN, MOE_FFN]), "k": rng.choice([2048, 4096, MOE_FFN])}
    width, size = rng.choice([(64, 56), (128, 28), (256, 14), (512, 7)])          # the four stages of ResNet-50
    cin, cout, size, kk, stride = rng.choice([(width, width, size, 3, 1), (width, width, 2 * size, 3, 2), (4 * width, width, size, 1, 1),
                                              (width, 4 * width, size, 1, 1)])
    return {"kind": "conv", "B": _log_int(rng, 8, 256 if stride == 1 else 128), "cin": cin, "cout": cout, "size": size, "k": kk, "stride": stride}


# ------------------------------------------------------------------------------------------------ inputs
# Everything random is drawn on the plain CUDA device from the seed and then handed to the backend, so that `exact`
# starts from the very same numbers without touching the backend.
class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)

    def normal(self, *shape, std=1.0, dtype=BF16):
        return (torch.randn(*shape, device="cuda", generator=self.g) * std).to(dtype)

    def ints(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, device="cuda", generator=self.g)


def _ints(text):
    return [int(t) for t in text.split(",")]


def _block_config(c, layers=1, max_len=4096):
    return LlamaConfig(vocab_size=VOCAB, dim=DIM, n_layers=layers, n_heads=HEADS, n_kv_heads=c["Hkv"], ffn_dim=c["ffn"], max_seq_len=max_len)


def _inputs(c, seed):
    r, k = _Rand(seed), c["kind"]
    if k == "norm":
        d = {"x": r.normal(c["rows"], c["dim"]), "res": r.normal(c["rows"], c["dim"], std=2.0), "w": 1 + r.normal(c["dim"], std=0.1)}
        if c["train"]:
            d.update(dy=r.normal(c["rows"], c["dim"]), dh=r.normal(c["rows"], c["dim"]))
        return d
    if k == "attn":
        dt = DTYPES[c["dtype"]]
        d = {n: r.normal(c["B"], c["Sq"], h, HD, dtype=dt) for n, h in (("q", c["H"]), ("k", c["Hkv"]), ("v", c["Hkv"]))}
        if c["train"]:
            d["do"] = r.normal(c["B"], c["Sq"], c["H"], HD, dtype=dt)
        return d
    if k == "varlen":
        n = sum(_ints(c["lens"]))
        d = {name: r.normal(n, h, HD) for name, h in (("q", c["H"]), ("k", c["Hkv"]), ("v", c["Hkv"]))}
        if c["train"]:
            d["do"] = r.normal(n, c["H"], HD)
        return d
    if k == "mlp":
        d = {"x": r.normal(c["tokens"], c["dim"]), "w13": r.normal(2 * c["ffn"], c["dim"], std=0.02), "w2": r.normal(c["dim"], c["ffn"], std=0.02)}
        if c["train"]:
            d["dy"] = r.normal(c["tokens"], c["dim"])
        return d
    if k in ("block", "decode"):
        kv = c["Hkv"]

        def layer():
            return {"attn_norm.weight": 1 + r.normal(DIM, std=0.1), "attn.wqkv.weight": r.normal((HEADS + 2 * kv) * HD, DIM, std=0.02),
                    "attn.wo.weight": r.normal(DIM, HEADS * HD, std=0.02), "ffn_norm.weight": 1 + r.normal(DIM, std=0.1),
                    "ffn.w13.weight": r.normal(2 * c["ffn"], DIM, std=0.02), "ffn.w2.weight": r.normal(DIM, c["ffn"], std=0.02)}

        if k == "block":
            return {"p": layer(), "x": r.normal(c["B"], c["S"], DIM), "dy": r.normal(c["B"], c["S"], DIM)}
        p = {"tok_emb.weight": r.normal(VOCAB, DIM, std=1.0), "norm.weight": 1 + r.normal(DIM, std=0.1), "lm_head.weight": r.normal(VOCAB, DIM, std=0.02)}
        for i in range(c["layers"]):
            p.update({"layers.%d.%s" % (i, n): t for n, t in layer().items()})
        caches = [r.normal(c["B"], kv, c["kv"], HD) for _ in range(2 * c["layers"])]
        return {"p": p, "caches": caches, "tokens": r.ints(0, VOCAB, c["B"], 1)}
    if k == "loss":
        t = r.ints(0, c["vocab"], c["rows"])
        t[r.ints(0, 20, c["rows"]) == 0] = -100        # padding positions
        return {"logits": r.normal(c["rows"], c["vocab"], std=2.0), "target": t}
    if k == "experts":
        n = _ints(c["counts"])
        d = {"x": r.normal(sum(n), DIM), "w13": r.normal(len(n), 2 * c["ffn"], DIM, std=0.02), "w2": r.normal(len(n), DIM, c["ffn"], std=0.02)}
        if c["train"]:
            d["dy"] = r.normal(sum(n), DIM)
        return d
    if k == "fp8":
        w = r.normal(c["n"], c["k"], std=0.02).float().view(c["n"] // 128, 128, c["k"] // 128, 128)
        scale = w.abs().amax(dim=(1, 3)) / 448.0
        q = (w / scale[:, None, :, None]).clamp(-448, 448).view(c["n"], c["k"]).to(torch.float8_e4m3fn)
        return {"x": r.normal(c["rows"], c["k"]), "wq": q, "ws": scale}
    so = c["size"] // c["stride"]
    return {"x": r.normal(c["B"], c["cin"], c["size"], c["size"]).relu(), "dy": r.normal(c["B"], c["cout"], so, so),
            "w": r.normal(c["cout"], c["cin"], c["k"], c["k"], std=math.sqrt(2.0 / (c["cout"] * c["k"] ** 2)), dtype=torch.float32),
            "g": 1 + r.normal(c["cout"], std=0.1, dtype=torch.float32), "b": r.normal(c["cout"], std=0.1, dtype=torch.float32)}


def _dev(t):
    return t.to(DEV)


def _leaf(t):
    return t.to(DEV).requires_grad_()


def _load(module, params):
    module.to_empty(device=DEV)
    with torch.no_grad():
        for n, p in module.named_parameters():
            p.copy_(params[n])
    return module


def prepare(case, seed):
    c, k = case, case["kind"]
    d = _inputs(c, seed)
    s = {"case": c}
    if k == "norm":
        mk = _leaf if c["train"] else _dev
        s.update(x=mk(d["x"]), res=mk(d["res"]), w=mk(d["w"]))
        if c["train"]:
            s.update(dy=_dev(d["dy"]), dh=_dev(d["dh"]))
    elif k in ("attn", "varlen"):
        mk = _leaf if c["train"] else _dev
        s.update({n: mk(d[n]) for n in "qkv"})
        if c["train"]:
            s["do"] = _dev(d["do"])
        if k == "varlen":
            lens = _ints(c["lens"])
            cu = [0]
            for n in lens:
                cu.append(cu[-1] + n)
            s.update(cu=torch.tensor(cu, dtype=torch.int32).to(DEV), longest=max(lens))
    elif k == "mlp":
        with torch.device("meta"):
            m = FeedForward(LlamaConfig(dim=c["dim"], ffn_dim=c["ffn"])).to(BF16)
        s.update(m=_load(m, {"w13.weight": d["w13"], "w2.weight": d["w2"]}), x=(_leaf if c["train"] else _dev)(d["x"]))
        if c["train"]:
            s["dy"] = _dev(d["dy"])
    elif k == "block":
        rope = RopeTables()
        rope.cos, rope.sin = BF.precompute_rope_cache(c["S"], HD, device=DEV)
        with torch.device("meta"):
            m = Block(_block_config(c), rope).to(BF16)
        s.update(m=_load(m, d["p"]), x=_leaf(d["x"]), dy=_dev(d["dy"]))
    elif k == "loss":
        s.update(logits=_leaf(d["logits"]), target=_dev(d["target"]))
    elif k == "decode":
        cfg = _block_config(c, c["layers"], c["kv"] + 8)
        with torch.device("meta"):
            m = Llama(cfg).to(BF16)
        m = _load(m, d["p"]).eval()
        m.init_rope_cache(DEV)
        m.lm_head.register_forward_hook(lambda mod, i, o: s.update(logits=o))     # the step's logits, for the caller's sampler
        dec = LlamaDecoder(m, c["B"], c["kv"] + 8, device=DEV)
        for i in range(c["layers"]):
            dec.k_cache[i, :, :, :c["kv"]].copy_(d["caches"][2 * i])
            dec.v_cache[i, :, :, :c["kv"]].copy_(d["caches"][2 * i + 1])
        s.update(dec=dec, tokens=_dev(d["tokens"]))
        dec.tokens.copy_(s["tokens"])
        dec.pos.fill_(c["kv"])
        dec.capture()
    elif k == "experts":
        with torch.device("meta"):
            m = Experts(len(_ints(c["counts"])), DIM, c["ffn"]).to(BF16)
        s.update(m=_load(m, {"w13": d["w13"], "w2": d["w2"]}), x=(_leaf if c["train"] else _dev)(d["x"]),
                 counts=torch.tensor(_ints(c["counts"]), dtype=torch.int32).to(DEV))
        if c["train"]:
            s["dy"] = _dev(d["dy"])
    elif k == "fp8":
        s.update({n: _dev(t) for n, t in d.items()})
    else:
        cl = torch.channels_last
        with torch.device("meta"):
            conv = torch.nn.Conv2d(c["cin"], c["cout"], c["k"], stride=c["stride"], padding=c["k"] // 2, bias=False)
            bn = torch.nn.BatchNorm2d(c["cout"])
        s.update(conv=_load(conv, {"weight": d["w"]}).to(memory_format=cl), bn=_load(bn, {"weight": d["g"], "bias": d["b"]}))
        bn.reset_running_stats()
        s.update(x=_dev(d["x"]).contiguous(memory_format=cl).requires_grad_(), dy=_dev(d["dy"]).contiguous(memory_format=cl))
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _forward_backward(y, dy, x, m):
    return [y.detach(), *torch.autograd.grad(y, [x, *m.parameters()], dy)]


def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "norm":
        y, h = BF.rms_norm_residual(s["x"], s["res"], s["w"], 1e-5)
        if not c["train"]:
            return [y, h]
        return [y.detach(), h.detach(), *torch.autograd.grad([y, h], [s["x"], s["res"], s["w"]], [s["dy"], s["dh"]])]
    if k == "attn":
        o = F.scaled_dot_product_attention(s["q"].transpose(1, 2), s["k"].transpose(1, 2), s["v"].transpose(1, 2), is_causal=c["causal"],
                                           enable_gqa=c["H"] != c["Hkv"]).transpose(1, 2)
        return [o.detach(), *torch.autograd.grad(o, [s["q"], s["k"], s["v"]], s["do"])] if c["train"] else [o]
    if k == "varlen":
        o = BF.flash_attn_varlen_func(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["longest"], s["longest"], causal=c["causal"])
        return [o.detach(), *torch.autograd.grad(o, [s["q"], s["k"], s["v"]], s["do"])] if c["train"] else [o]
    if k == "mlp":
        if not c["train"]:
            with torch.no_grad():
                return [s["m"](s["x"])]
        return _forward_backward(s["m"](s["x"]), s["dy"], s["x"], s["m"])
    if k == "block":
        return _forward_backward(s["m"](s["x"]), s["dy"], s["x"], s["m"])
    if k == "loss":
        loss = BF.fused_cross_entropy(s["logits"], s["target"])
        return [loss.detach(), *torch.autograd.grad(loss, [s["logits"]])]
    if k == "decode":
        dec = s["dec"]
        dec.tokens.copy_(s["tokens"])
        dec.pos.fill_(c["kv"])
        dec.decode(1)
        return [s["logits"], dec.k_cache[:, :, :, c["kv"]], dec.v_cache[:, :, :, c["kv"]]]     # the logits and the rows the step wrote
    if k == "experts":
        if not c["train"]:
            with torch.no_grad():
                return [s["m"](s["x"], s["counts"])]
        return _forward_backward(s["m"](s["x"], s["counts"]), s["dy"], s["x"], s["m"])
    if k == "fp8":
        q, scales = torch.ops.blackwell.quantize_fp8_1x128(s["x"])
        return [torch.ops.blackwell.scaled_mm(q, s["wq"], scales, s["ws"], None, None, None, BF16), scales]
    conv, bn = s["conv"], s["bn"]
    with torch.autocast(DEV, dtype=BF16):
        y = BF.batch_norm_act(conv(s["x"]), bn.weight, bn.bias, bn.running_mean, bn.running_var, relu=False)
    return [y.detach(), *torch.autograd.grad(y, [s["x"], conv.weight, bn.weight, bn.bias], s["dy"]), bn.running_mean, bn.running_var]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _attn_flops(lens, heads, causal, train):
    pairs = sum(n * (n + 1) / 2 if causal else n * n for n in lens)
    return pairs * heads * HD * 2 * (2 + (5 if train else 0))


def work(case):
    c, k = case, case["kind"]
    if k == "norm":
        n, d = c["rows"], c["dim"]
        return {"bytes": 2 * (n * d * (4 + (4 if c["train"] else 0)) + d), "flops": n * d * (6 + (12 if c["train"] else 0))}
    if k in ("attn", "varlen"):
        lens = [c["Sq"]] * c["B"] if k == "attn" else _ints(c["lens"])
        n, q, kv = sum(lens), c["H"] * HD, c["Hkv"] * HD
        return {"bytes": 2 * n * (2 * q + 2 * kv + ((2 * q + 2 * kv) if c["train"] else 0)), "flops": _attn_flops(lens, c["H"], c["causal"], c["train"])}
    if k == "mlp":
        w, t = 3 * c["dim"] * c["ffn"], c["tokens"]
        return {"bytes": 2 * (w * (2 if c["train"] else 1) + t * c["dim"] * (4 if c["train"] else 2)), "flops": 2 * t * w * (3 if c["train"] else 1)}
    if k in ("block", "decode"):
        w = DIM * (HEADS + 2 * c["Hkv"]) * HD + DIM * DIM + 3 * DIM * c["ffn"]
        if k == "block":
            t = c["B"] * c["S"]
            return {"bytes": 2 * (2 * w + 4 * t * DIM), "flops": 6 * t * w + _attn_flops([c["S"]] * c["B"], HEADS, True, True)}
        cache = 2 * c["B"] * c["Hkv"] * c["kv"] * HD
        w = c["layers"] * w + VOCAB * DIM
        return {"bytes": 2 * (w + c["layers"] * cache + c["B"] * VOCAB), "flops": 2 * c["B"] * w + c["layers"] * 4 * c["B"] * HEADS * c["kv"] * HD}
    if k == "loss":
        n = c["rows"] * c["vocab"]
        return {"bytes": 2 * n * 2, "flops": 8 * n}
    if k == "experts":
        n = _ints(c["counts"])
        w = 3 * DIM * c["ffn"]
        return {"bytes": 2 * (len(n) * w * (2 if c["train"] else 1) + sum(n) * DIM * (4 if c["train"] else 2)),
                "flops": 2 * sum(n) * w * (3 if c["train"] else 1)}
    if k == "fp8":
        m, n, kk = c["rows"], c["n"], c["k"]
        return {"bytes": 2 * m * kk + n * kk + 2 * m * n, "flops": 2 * m * n * kk}
    px, pin = c["B"] * (c["size"] // c["stride"]) ** 2, c["B"] * c["size"] ** 2
    w = c["cin"] * c["cout"] * c["k"] ** 2
    return {"bytes": 2 * (2 * pin * c["cin"] + 2 * px * c["cout"]) + 8 * w, "flops": 6 * px * w}


def tolerance(case):
    return {"rel": TOLERANCE[case["kind"]]}


# about four times the error against 64 bits that the outputs of each kind show (block and decode: three times)
TOLERANCE = {"norm": 0.01, "attn": 0.01, "varlen": 0.01, "mlp": 0.014, "block": 0.028, "loss": 0.01, "decode": 0.022, "experts": 0.014,
             "fp8": 0.014, "conv": 0.02}


# ------------------------------------------------------------------------------------------------ 64-bit results (plain PyTorch)
# Gradients are written out: autograd of plain CUDA tensors is not available in a process that has loaded the backend.
def _probs64(q, k, causal):
    s = q @ k.t() / math.sqrt(HD)
    if causal:
        s.masked_fill_(torch.ones(s.shape, dtype=torch.bool, device=s.device).triu_(1), float("-inf"))
    return torch.softmax(s, -1)


def _attention64(q, k, v, causal, do=None):
    """Attention of one sequence, head by head: q [S, H, D], k / v [S, Hkv, D]; (out, dq, dk, dv)."""
    g = q.shape[1] // k.shape[1]
    o, dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
    for h in range(q.shape[1]):
        qh, kh, vh = q[:, h], k[:, h // g], v[:, h // g]
        p = _probs64(qh, kh, causal)
        o[:, h] = p @ vh
        if do is not None:
            dv[:, h // g] += p.t() @ do[:, h]
            dp = do[:, h] @ vh.t()
            ds = p * (dp - (dp * p).sum(-1, keepdim=True)) / math.sqrt(HD)
            dq[:, h] = ds @ kh
            dk[:, h // g] += ds.t() @ qh
    return o, dq, dk, dv


def _norm64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w


def _norm64_backward(dy, x, w):
    r = torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5)
    g = dy * w
    return r * (g - x * r.square() * (g * x).mean(-1, keepdim=True)), (dy * x * r).flatten(0, -2).sum(0)


def _rope64(x, first=0, sign=1.0):
    """x [B, S, H, D] at positions first, first + 1, ...; the tables are rounded to fp32 like a user's; sign -1 turns back."""
    inv = 1.0 / (10000.0 ** (torch.arange(0, HD, 2, dtype=torch.float32) / HD))
    f = torch.outer(torch.arange(first + x.shape[1], dtype=torch.float32), inv)[first:]
    cs, sn = f.cos().double().to(x.device)[None, :, None], sign * f.sin().double().to(x.device)[None, :, None]
    a, b = x[..., :HD // 2], x[..., HD // 2:]
    return torch.cat((a * cs - b * sn, b * cs + a * sn), -1)


def _ffn64(x, w13, w2):
    g, u = (x @ w13.t()).chunk(2, -1)
    return (F.silu(g) * u) @ w2.t()


def _ffn64_backward(dy, x, w13, w2):
    g, u = (x @ w13.t()).chunk(2, -1)
    s = torch.sigmoid(g)
    a, da = g * s * u, dy @ w2
    dgu = torch.cat((da * u * s * (1 + g * (1 - s)), da * g * s), -1)
    return dgu @ w13, dgu.t() @ x, dy.t() @ a


def _conv64_backward(dy, x, w, stride, padding):
    return torch.ops.aten.convolution_backward(dy, x, w, None, [stride, stride], [padding, padding], [1, 1], False, [0, 0], 1, [True, True, False])[:2]


def _bn64(x, w, b):
    mean, var = x.mean((0, 2, 3), keepdim=True), x.var((0, 2, 3), unbiased=False, keepdim=True)
    return (x - mean) * torch.rsqrt(var + 1e-5) * w[:, None, None] + b[:, None, None]


def _bn64_backward(dy, x, w):
    mean, var = x.mean((0, 2, 3), keepdim=True), x.var((0, 2, 3), unbiased=False, keepdim=True)
    r = torch.rsqrt(var + 1e-5)
    xh = (x - mean) * r
    db, dw = dy.sum((0, 2, 3)), (dy * xh).sum((0, 2, 3))
    n = x.numel() // x.shape[1]
    return w[:, None, None] * r * (dy - db[:, None, None] / n - xh * dw[:, None, None] / n), dw, db


@torch.no_grad()
def exact(case, seed):
    c, k = case, case["kind"]
    d = {n: t.double() if torch.is_tensor(t) and t.dtype in (BF16, torch.float16) else t for n, t in _inputs(c, seed).items()}
    if "p" in d:
        d["p"] = {n: t.double() for n, t in d["p"].items()}
    if k == "norm":
        h = d["x"] + d["res"]
        y = _norm64(h, d["w"])
        if not c["train"]:
            return [y, h]
        dh, dw = _norm64_backward(d["dy"], h, d["w"])
        return [y, h, dh + d["dh"], dh + d["dh"], dw]
    if k in ("attn", "varlen"):
        q, kk, v, do = d["q"], d["k"], d["v"], d.get("do")
        if k == "attn":
            parts = [_attention64(q[b], kk[b], v[b], c["causal"], do[b] if do is not None else None) for b in range(c["B"])]
            out = [torch.stack(t) for t in zip(*parts)]
        else:
            n = _ints(c["lens"])
            dos = do.split(n) if do is not None else [None] * len(n)
            out = [torch.cat(t) for t in zip(*[_attention64(*a, c["causal"], g) for *a, g in zip(q.split(n), kk.split(n), v.split(n), dos)])]
        return out if c["train"] else out[:1]
    if k == "mlp":
        y = _ffn64(d["x"], d["w13"], d["w2"])
        return [y, *_ffn64_backward(d["dy"], d["x"], d["w13"], d["w2"])] if c["train"] else [y]
    if k == "block":
        p, B, S, kv = d["p"], c["B"], c["S"], c["Hkv"]
        x, dy = d["x"].view(B * S, DIM), d["dy"].view(B * S, DIM)
        wn1, wqkv, wo, wn2, w13, w2 = [p[n] for n in ("attn_norm.weight", "attn.wqkv.weight", "attn.wo.weight", "ffn_norm.weight", "ffn.w13.weight",
                                                     "ffn.w2.weight")]
        hn = _norm64(x, wn1)
        q, kk, v = (hn @ wqkv.t()).view(B, S, HEADS + 2 * kv, HD).split([HEADS, kv, kv], 2)
        q, kk = _rope64(q), _rope64(kk)
        o = torch.stack([_attention64(q[b], kk[b], v[b], True)[0] for b in range(B)]).view(B * S, -1)
        h = x + o @ wo.t()
        fn = _norm64(h, wn2)
        y = h + _ffn64(fn, w13, w2)
        dfn, dw13, dw2 = _ffn64_backward(dy, fn, w13, w2)
        dh, dwn2 = _norm64_backward(dfn, h, wn2)
        dh = dh + dy
        do = (dh @ wo).view(B, S, HEADS, HD)
        dq, dk, dv = [torch.stack(t) for t in list(zip(*[_attention64(q[b], kk[b], v[b], True, do[b]) for b in range(B)]))[1:]]
        dqkv = torch.cat((_rope64(dq, sign=-1.0), _rope64(dk, sign=-1.0), dv), 2).view(B * S, -1)
        dx, dwn1 = _norm64_backward(dqkv @ wqkv, x, wn1)
        return [y.view(B, S, DIM), (dx + dh).view(B, S, DIM), dwn1, dqkv.t() @ hn, dh.t() @ o, dwn2, dw13, dw2]
    if k == "loss":
        z, t = d["logits"], d["target"]
        valid = t != -100
        n = valid.sum()
        g = torch.softmax(z, -1)
        g[valid.nonzero()[:, 0], t[valid]] -= 1
        return [F.cross_entropy(z, t, ignore_index=-100), g * valid[:, None] / n]
    if k == "decode":
        B, kv, n = c["B"], c["Hkv"], c["kv"]
        p, rows_k, rows_v = d["p"], [], []
        x = p["tok_emb.weight"][d["tokens"][:, 0]]
        for i in range(c["layers"]):
            w = {m: p["layers.%d.%s" % (i, m)] for m in ("attn_norm.weight", "attn.wqkv.weight", "attn.wo.weight", "ffn_norm.weight", "ffn.w13.weight",
                                                         "ffn.w2.weight")}
            q, kn, vn = (_norm64(x, w["attn_norm.weight"]) @ w["attn.wqkv.weight"].t()).view(B, 1, HEADS + 2 * kv, HD).split([HEADS, kv, kv], 2)
            q, kn = _rope64(q.transpose(0, 1).reshape(1, 1, -1, HD), n).view(B, HEADS, HD), _rope64(kn.reshape(1, 1, -1, HD), n).view(B, kv, HD)
            vn = vn[:, 0]
            rows_k.append(kn)
            rows_v.append(vn)
            o = []
            for b in range(B):
                kk = torch.cat((d["caches"][2 * i][b].double(), kn[b][:, None]), 1)
                vv = torch.cat((d["caches"][2 * i + 1][b].double(), vn[b][:, None]), 1)
                qb = q[b].view(kv, HEADS // kv, HD)
                o.append((torch.softmax(qb @ kk.transpose(1, 2) / math.sqrt(HD), -1) @ vv).reshape(-1))
            x = x + torch.stack(o) @ w["attn.wo.weight"].t()
            x = x + _ffn64(_norm64(x, w["ffn_norm.weight"]), w["ffn.w13.weight"], w["ffn.w2.weight"])
        logits = _norm64(x, p["norm.weight"]) @ p["lm_head.weight"].t()
        return [logits.view(B, 1, -1), torch.stack(rows_k), torch.stack(rows_v)]
    if k == "experts":
        n = _ints(c["counts"])
        xs = d["x"].split(n)
        y = torch.cat([_ffn64(x, d["w13"][e], d["w2"][e]) for e, x in enumerate(xs)])
        if not c["train"]:
            return [y]
        dx, dw13, dw2 = zip(*[_ffn64_backward(g, x, d["w13"][e], d["w2"][e]) for e, (g, x) in enumerate(zip(d["dy"].split(n), xs))])
        return [y, torch.cat(dx), torch.stack(dw13), torch.stack(dw2)]
    if k == "fp8":
        x = d["x"].float().view(c["rows"], -1, 128)
        scale = x.abs().amax(-1).clamp_min(1e-12) / 448.0
        q = (x / scale[..., None]).clamp(-448, 448).to(torch.float8_e4m3fn).double() * scale[..., None].double()
        w = d["wq"].double().view(c["n"] // 128, 128, -1, 128) * d["ws"].double()[:, None, :, None]
        return [q.view(c["rows"], -1) @ w.view(c["n"], -1).t(), scale.double()]
    st = c["stride"]
    x, w, g = d["x"], d["w"].double(), d["g"].double()
    t = F.conv2d(x, w, stride=st, padding=c["k"] // 2)
    dt, dg, db = _bn64_backward(d["dy"], t, g)
    return [_bn64(t, g, d["b"].double()), *_conv64_backward(dt, x, w, st, c["k"] // 2), dg, db, 0.1 * t.mean((0, 2, 3)),
            0.9 + 0.1 * t.var((0, 2, 3))]
