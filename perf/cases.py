"""What a user of this library has it do, as measurable cases: single projections, projections of several columns, decode
attention, and whole passes of the 9B-shape model (greedy decode, a sampled token at long context, prompt prefill, a pipeline
stage, a serving step). Every case goes through the public entry points of bonsai_vk_b200 (Context, Model); inputs, weights
and caches are made on the GPU from the seed.

  listed()             the named cases            draw(rng)    one more case of the same ranges
  prepare(case, seed)  the state before the call  run(state)   one pass and its outputs
  work(case)           bytes and flops that a pass cannot do without
  tolerance(case)      how far another correct implementation may be from the outputs
"""
import ctypes as C
import math

import torch

from bonsai_vk_b200 import Context, Model, lib, synth

HEAD_DIM, BLOCK_BYTES = 256, 28
_ctx = None
_tables = None


def listed():
    return [
        # The smallest projection of a decode step: the k (or v) rows of an attention block. Launches and latency count.
        {"name": "gemv k rows", "kind": "gemv", "M": 1024, "K": 4096},
        # The largest one: the output head of the 9B shape, read once per token.
        {"name": "gemv output head", "kind": "gemv", "M": 248320, "K": 4096},
        # FFN gate | up of a 16-token prompt block, weights laid out once for the multi-column kernel.
        {"name": "gemm ffn 16 tokens", "kind": "gemm", "M": 24576, "K": 4096, "ncol": 16, "tiled": True, "hat": 4096},
        # Weights as the file holds them, a height that is no whole number of tiles, a width and a column count in between.
        {"name": "gemm ragged", "kind": "gemm", "M": 3000, "K": 5120, "ncol": 11, "tiled": False, "hat": 1024},
        # One decode-attention layer at the two contexts of the benchmark, q8_0 keys and values.
        {"name": "attention 4096", "kind": "attn", "keys": 4096, "cap": 4096, "n_head": 16, "n_kv": 4, "k_mode": 0, "v_mode": 0},
        {"name": "attention 32768", "kind": "attn", "keys": 32768, "cap": 32768, "n_head": 16, "n_kv": 4, "k_mode": 0, "v_mode": 0},
        # A partly filled cache in the reference's own layout: fp16 keys, q8_0 values.
        {"name": "attention fp16 keys", "kind": "attn", "keys": 1501, "cap": 8192, "n_head": 16, "n_kv": 4, "k_mode": 1, "v_mode": 0},
        # The headline: greedy decode of one sequence after a 16-token prompt, 48 tokens chained on the device.
        {"name": "decode 48", "kind": "decode", "layers": 32, "cap": 256, "pos": 16, "steps": 48},
        # One token of a long conversation whose next id a host-side sampler takes from the logits.
        {"name": "sampled token 30k", "kind": "decode", "layers": 32, "cap": 32768, "pos": 30000, "steps": 1},
        # A prompt in blocks of 32 tokens, the last one ragged.
        {"name": "prefill 100", "kind": "prefill", "layers": 32, "cap": 512, "pos": 0, "tokens": 100, "block": 32},
        # A server's step: eight conversations of different lengths through the whole model, one of them sampled on the host.
        {"name": "serve 8", "kind": "stage", "layers": 32, "b0": 0, "b1": 32, "cap": 2048, "ncol": 8},
        # A stage of the eight-GPU pipeline: four blocks, eight of the 64 sequences at context 8192, hidden states in and out.
        {"name": "pipeline stage", "kind": "stage", "layers": 32, "b0": 4, "b1": 8, "cap": 8192, "ncol": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemv", "gemv", "gemm", "gemm", "attn", "attn", "decode", "prefill", "stage", "stage"])
    if kind == "gemv":
        return {"kind": kind, "M": _log(rng, 64, 248320), "K": 128 * _log(rng, 4, 96)}
    if kind == "gemm":
        return {"kind": kind, "M": _log(rng, 128, 24576), "K": 1024 * rng.randint(1, 12), "ncol": rng.randint(1, 32),
                "tiled": rng.random() < 0.5, "hat": rng.choice([0, 256, 1024])}
    if kind == "attn":
        keys = _log(rng, 64, 32768)
        cap = min(32768, int(keys * rng.uniform(1.0, 3.0)) + 2) & ~1
        k_mode, v_mode = rng.choice([(0, 0), (0, 0), (1, 0), (1, 1)])
        n_head, n_kv = rng.choice([(16, 4), (16, 4), (8, 4), (8, 1)])
        return {"kind": kind, "keys": min(keys, cap), "cap": cap, "n_head": n_head, "n_kv": n_kv, "k_mode": k_mode, "v_mode": v_mode}
    layers = 4 * rng.randint(1, 8)
    if kind == "decode":
        steps, pos = _log(rng, 1, 48), _log(rng, 16, 16000)
        return {"kind": kind, "layers": layers, "cap": (pos + steps + _log(rng, 2, 16000)) & ~1, "pos": pos, "steps": steps}
    if kind == "prefill":
        tokens, pos = _log(rng, 2, 100), _log(rng, 1, 4096) - 1
        return {"kind": kind, "layers": layers, "cap": (pos + tokens + 65) & ~1, "pos": pos, "tokens": tokens, "block": rng.choice([8, 16, 32])}
    b0 = rng.randint(0, 27)
    return {"kind": kind, "layers": 32, "b0": b0, "b1": min(32, b0 + rng.randint(1, 8)), "cap": 2 * _log(rng, 64, 4096), "ncol": rng.randint(1, 32)}


# ---- inputs -------------------------------------------------------------------------------------------------------------
def _context():
    """One context on a stream of its own (the stage schedules are captured, which the default stream does not allow)."""
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
        _ctx.stream = torch.cuda.Stream()
        _ctx.use_stream(_ctx.stream.cuda_stream)
    return _ctx


def _rng(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _trit_tables():
    """65536 equally likely bytes of five (then of four) independent trits with P(-1, 0, +1) = (0.3, 0.4, 0.3)."""
    global _tables
    if _tables is None:
        p = torch.tensor([0.3, 0.4, 0.3], dtype=torch.float64)
        out = []
        for n in (5, 4):
            joint = p
            for _ in range(n - 1):
                joint = (joint[:, None] * p[None, :]).reshape(-1)
            u = (torch.arange(65536, dtype=torch.float64) + 0.5) / 65536
            code = torch.searchsorted(joint.cumsum(0), u).clamp_(max=joint.numel() - 1)
            out.append(((code * 256 + joint.numel() - 1) // joint.numel()).to(torch.uint8).cuda())
        _tables = out
    return _tables


def _blocks(g, n):
    """n random PTQ1_0 blocks (26 bytes of trits, fp16 scale |N(0, 0.02)|) as a byte tensor."""
    five, four = _trit_tables()
    out = torch.empty((n, BLOCK_BYTES), dtype=torch.uint8, device="cuda")
    step = 1 << 22
    for i in range(0, n, step):
        k = min(step, n - i)
        r = torch.randint(0, 65536, (k, 26), generator=g, device="cuda", dtype=torch.int32)
        out[i:i + k, :24] = five[r[:, :24]]
        out[i:i + k, 24:26] = four[r[:, 24:]]
        s = (torch.randn(k, generator=g, device="cuda") * 0.02).abs().to(torch.float16)
        out[i:i + k, 26:] = s.view(torch.uint8).view(k, 2)
    return out.view(-1)


class _State:
    """Device memory under library handles, all of it given back with the state."""

    def __init__(self, case):
        self.case, self.ctx, self.keep, self.model = case, _context(), [], None

    def wrap(self, t):
        b = self.ctx.wrap(t.data_ptr(), t.numel() * t.element_size())
        self.keep.append((b, t))
        return b

    def empty(self, n, dtype=torch.float32):
        t = torch.zeros(n, dtype=dtype, device="cuda")
        return t, self.wrap(t)

    def __del__(self):
        try:
            if self.model is not None:
                self.model.close()
            for b, _ in self.keep:
                b.free()
        except Exception:
            pass


class _DeviceModel(Model):
    """Model over weights that are in device memory already: each tensor registered by name where it lies."""

    def __init__(self, state, hp, g):
        self.ctx, self.hp, self.head_rows = state.ctx, hp, None
        L = self.ctx.lib
        fields = {f[0] for f in lib.HParamsC._fields_}
        hc = lib.HParamsC(**{k: (float(v) if k in ("rms_eps", "rope_base") else int(v)) for k, v in hp.asdict().items() if k in fields})
        self.h = C.c_void_p()
        self._ok(L.bn_model_create(self.ctx.h, C.byref(hc), C.byref(self.h)))
        b0, b1 = hp.block_begin, hp.block_end or hp.n_layer
        names = {}
        for name, spec in synth.tensor_shapes(hp).items():
            if name.startswith("blk."):
                here = b0 <= int(name.split(".")[1]) < b1
            else:
                here = b0 == 0 if name == "token_embd.weight" else b1 == hp.n_layer
            if here:
                names[name] = spec
        blocks = {n: s[1] * s[2] // 128 for n, s in names.items() if s[0] == "ptq"}
        ptq = _blocks(g, sum(blocks.values()))
        weights, off = state.wrap(ptq), 0
        for name, n in blocks.items():
            self._ok(L.bn_model_set_tensor(self.h, name.encode(), weights.h, off, n * BLOCK_BYTES))
            off += n * BLOCK_BYTES
        for name, spec in names.items():
            if spec[0] == "ptq":
                continue
            t = torch.randn(spec[1], generator=g, device="cuda")
            if name.endswith("norm.weight"):
                t = 1.0 + 0.1 * t
            elif name.endswith(("ssm_alpha.weight", "ssm_beta.weight")):
                t = 0.02 * t
            elif name.endswith("ssm_a"):
                t = -0.5 * (0.5 * t).exp()
            elif name.endswith("ssm_conv1d.weight"):
                t = 0.5 * t
            self._ok(L.bn_model_set_tensor(self.h, name.encode(), state.wrap(t.contiguous()).h, 0, t.numel() * 4))
        signs = torch.randint(0, 2, (hp.hidden + hp.ffn,), generator=g, device="cuda", dtype=torch.int32) * 2 - 1
        torch.cuda.synchronize()
        self._ok(L.bn_model_set_signs(self.h, state.wrap(signs).h, 0, signs.numel()))
        self._ok(L.bn_model_finalize(self.h))

    def _ok(self, rc):
        if rc != 0:
            raise lib.BonsaiError("%d: %s" % (rc, self.ctx.lib.bn_last_error().decode()))

    def close(self):
        if self.h is not None:
            self.ctx.lib.bn_model_destroy(self.h)
            self.h = None


def _tokens(g, n):
    return torch.randint(0, synth.HParams.vocab, (n,), generator=g, device="cuda", dtype=torch.int32)


def _prepare_gemv(s, g, M, K):
    s.w = s.wrap(_blocks(g, M * K // 128))
    s.x = s.wrap(torch.randn(K, generator=g, device="cuda"))
    s.pack = s.wrap(torch.empty(s.ctx.act_pack_bytes(K), dtype=torch.uint8, device="cuda"))
    s.out_t, s.out = s.empty(M)


def _prepare_gemm(s, g, M, K, ncol, tiled, hat):
    s.w = s.wrap(_blocks(g, M * K // 128))
    torch.cuda.synchronize()
    if tiled:
        native, s.w = s.w, s.ctx.gemm_repack(s.w, M, K)
        s.ctx.sync()
        s.keep = [k for k in s.keep if k[0] is not native] + [(s.w, None)]
        native.free()
    s.x = s.wrap(torch.randn(ncol * K, generator=g, device="cuda"))
    s.signs = s.wrap(torch.randint(0, 2, (K,), generator=g, device="cuda", dtype=torch.int32) * 2 - 1) if hat else None
    s.image = s.wrap(torch.empty(s.ctx.gemm_image_bytes(K, ncol), dtype=torch.uint8, device="cuda"))
    s.out_t, s.out = s.empty(ncol * M)
    s.out_t = s.out_t.view(ncol, M)


def _prepare_attn(s, g, keys, cap, n_head, n_kv, k_mode, v_mode):
    s.dims = lib.AttnDimsC(n_head=n_head, n_kv=n_kv, head_dim=HEAD_DIM, n_rot=64, cap=cap, k_mode=k_mode, v_mode=v_mode, rms_eps=1e-6, rope_base=1e7)
    kvb, scb = s.ctx.attn_sizes(s.dims)
    s.kv, s.scratch = s.empty(kvb, torch.uint8)[1], s.empty(scb, torch.uint8)[1]
    rows = min(keys, 4096)
    k, v = (torch.randn((rows, n_kv * HEAD_DIM), generator=g, device="cuda") for _ in range(2))
    s.k, s.v = s.wrap(k), s.wrap(v)
    s.qg = s.wrap(torch.randn((n_head, 2 * HEAD_DIM), generator=g, device="cuda"))
    s.qn, s.kn = (s.wrap(1.0 + 0.1 * torch.randn(HEAD_DIM, generator=g, device="cuda")) for _ in range(2))
    s.pre_t, s.pre = s.empty(n_head * HEAD_DIM)
    s.out_t, s.out = s.empty(n_head * HEAD_DIM)
    torch.cuda.synchronize()
    for p in range(0, keys, rows):
        s.ctx.attn_insert(s.dims, s.kv, s.k, s.v, min(rows, keys - p), p, s.qg, s.qn, s.kn, s.scratch)


def _prepare_decode(s, g, layers, cap, pos, steps):
    s.model = _DeviceModel(s, synth.HParams(n_layer=layers, cap=cap), g)
    prompt = _tokens(g, 16).tolist()
    if pos > 16:                     # the earlier context as the benchmark has it: a cache marked as filled
        s.model.fill_kv(0, pos - 16)
    for i, t in enumerate(prompt):
        s.first = s.model.token(t, pos - 16 + i)


def _prepare_prefill(s, g, layers, cap, pos, tokens, block):
    s.model = _DeviceModel(s, synth.HParams(n_layer=layers, cap=cap, batch_cols=block), g)
    if pos:
        s.model.fill_kv(0, pos)
    ids = _tokens(g, tokens).tolist()
    s.blocks = [(ids[i:i + block], pos + i) for i in range(0, tokens, block)]


def _prepare_stage(s, g, layers, b0, b1, cap, ncol):
    hp = synth.HParams(n_layer=layers, cap=cap, n_streams=ncol, batch_cols=ncol, block_begin=b0, block_end=b1)
    s.model = _DeviceModel(s, hp, g)
    s.pos = [cap - 1 - (i * 37) % (cap // 4) for i in range(ncol)]      # conversations of different lengths
    for i, p in enumerate(s.pos):
        s.model.fill_kv(i, p)
    s.first, s.last = b0 == 0, b1 == layers
    s.inp = s.wrap(_tokens(g, ncol) if s.first else torch.randn(ncol * hp.hidden, generator=g, device="cuda"))
    s.out_t, s.out = s.empty(ncol, torch.int32) if s.last else s.empty(ncol * hp.hidden)
    s.model.stage_prepare(0, ncol)


def prepare(case, seed):
    p = {k: v for k, v in case.items() if k not in ("name", "kind")}
    s = _State(case)
    {"gemv": _prepare_gemv, "gemm": _prepare_gemm, "attn": _prepare_attn, "decode": _prepare_decode,
     "prefill": _prepare_prefill, "stage": _prepare_stage}[case["kind"]](s, _rng(seed), **p)
    torch.cuda.synchronize()
    return s


# ---- one pass -----------------------------------------------------------------------------------------------------------
def run(s):
    c, ctx = s.case, s.ctx
    kind = c["kind"]
    if kind == "gemv":
        ctx.act_quant_q81(s.x, c["K"], s.pack)
        ctx.gemv_q81(s.w, c["M"], c["K"], s.pack, s.out)
        return s.out_t
    if kind == "gemm":
        ctx.gemm_act_quant(s.x, c["K"], c["ncol"], s.image, signs=s.signs, hat_block=c["hat"])
        ctx.gemm_q81(s.w, c["M"], c["K"], s.image, c["ncol"], s.out, tiled=c["tiled"])
        return s.out_t
    if kind == "attn":
        last = c["keys"] - 1
        ctx.attn_insert(s.dims, s.kv, s.k, s.v, 1, last, s.qg, s.qn, s.kn, s.scratch)
        ctx.attn_attend(s.dims, s.kv, last, s.scratch, s.pre, s.out)
        return s.pre_t, s.out_t
    if kind == "decode":
        if c["steps"] == 1:
            s.model.token(s.first, c["pos"], want_next=False)
            return s.model.logits()
        picks = s.model.decode(s.first, c["pos"], c["steps"])
        return torch.tensor(picks, dtype=torch.int32), s.model.logits()
    if kind == "prefill":
        for ids, pos in s.blocks[:-1]:
            s.model.prefill(ids, pos, want_next=False)
        ids, pos = s.blocks[-1]
        return s.model.prefill(ids, pos), s.model.logits()
    s.model.stage_batch(0, None, s.pos, s.inp, s.out)
    return (s.out_t, s.model.logits(c["ncol"] - 1)) if s.last else s.out_t


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------
def _kv_bytes(n_kv, k_mode, v_mode):
    """bytes of one position's keys and values in one layer"""
    n = n_kv * HEAD_DIM
    return sum(n * 2 if m else n + n // 16 for m in (k_mode, v_mode))


def _pass(hp, b0, b1, cols, keys, state_cols, head_cols):
    """Bytes and flops of blocks [b0, b1) for `cols` columns that attend to `keys` positions each: weights once, every
    sequence's recurrent state read and written, its keys and values read."""
    weights = f32 = 0
    for name, spec in synth.tensor_shapes(hp).items():
        if name.startswith("blk.") and b0 <= int(name.split(".")[1]) < b1:
            if spec[0] == "ptq":
                weights += spec[1] * spec[2]
            else:
                f32 += math.prod(spec[1]) * 4
    n_attn = sum(hp.is_attn(b) for b in range(b0, b1))
    n_gdn = b1 - b0 - n_attn
    state = (hp.gdn_heads * hp.gdn_dim * hp.gdn_dim + 3 * hp.qkv_dim) * 4 * n_gdn
    kv = sum(keys) if state_cols > 1 or cols == 1 else max(keys)        # one sequence's columns share its cache
    flops = 2.0 * weights * cols + n_gdn * cols * 8.0 * hp.gdn_heads * hp.gdn_dim ** 2 + n_attn * 4.0 * hp.n_head * HEAD_DIM * sum(keys)
    nbytes = weights / 128 * BLOCK_BYTES + f32 + 2 * state * state_cols + n_attn * kv * _kv_bytes(hp.n_kv, hp.k_mode, hp.v_mode)
    if head_cols:
        nbytes += hp.vocab * hp.hidden / 128 * BLOCK_BYTES + hp.vocab * 4 * head_cols
        flops += 2.0 * hp.vocab * hp.hidden * head_cols
    return nbytes, flops


def work(case):
    c = case
    kind = c["kind"]
    if kind in ("gemv", "gemm"):
        n = c.get("ncol", 1)
        return {"bytes": c["M"] * c["K"] / 128 * BLOCK_BYTES + 4 * n * (c["K"] + c["M"]), "flops": 2.0 * c["M"] * c["K"] * n}
    if kind == "attn":
        q = c["n_head"] * HEAD_DIM
        return {"bytes": c["keys"] * _kv_bytes(c["n_kv"], c["k_mode"], c["v_mode"]) + 4 * q * 4, "flops": 4.0 * q * c["keys"]}
    hp = synth.HParams(n_layer=c["layers"])
    if kind == "decode":
        b, f = _pass(hp, 0, c["layers"], 1, [c["pos"] + (c["steps"] - 1) / 2 + 1], 1, 1)
        return {"bytes": b * c["steps"], "flops": f * c["steps"]}
    if kind == "prefill":
        total = [0.0, 0.0]
        for i in range(0, c["tokens"], c["block"]):
            n = min(c["block"], c["tokens"] - i)
            b, f = _pass(hp, 0, c["layers"], n, [c["pos"] + i + j + 1 for j in range(n)], 1, 1 if i + n == c["tokens"] else 0)
            total[0] += b
            total[1] += f
        return {"bytes": total[0], "flops": total[1]}
    n = c["ncol"]
    keys = [c["cap"] - (i * 37) % (c["cap"] // 4) for i in range(n)]
    b, f = _pass(hp, c["b0"], c["b1"], n, keys, n, n if c["b1"] == c["layers"] else 0)
    return {"bytes": b + 2 * 4 * n * hp.hidden, "flops": f}


def tolerance(case):
    # Single operations: fp32 sums whose order is open (int8 codes and integer dots are exact on the way). Model passes:
    # the library's own contract - every schedule of a pass gives the same floats and the same greedy ids.
    return {"rel": 1e-5} if case["kind"] in ("gemv", "gemm", "attn") else "exact"
