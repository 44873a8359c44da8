"""The work a user of this library has it do, as measurable cases over its public C entry points.

A decoder model's linear layers reach the library in four situations, and every case is one of
them at a size of the benchmark's projections (hidden 5120, 10240 wide attention input, MLP
17408, a 1024-row key/value projection, an int8 output head):

  proj1    one token through one projection: staging and GEMV (x_gemv_w4a8)
  mlp1     one token through a whole MLP: RMSNorm + staging, gate|up fan-out, SiLU * up +
           staging, down-projection with the residual
  decode   a batch of 8..64 tokens through one projection, or a few that share their input:
           chunk staging and the batched GEMM, with a scale per (token, K32) block (the
           reference's arithmetic) or per token
  head     the output head in the int8 tier, one token or a decode batch
  prefill  a prompt chunk of 128..4096 tokens: staging and the GEMM, with a scale per block
           (packed sequences keep their segments), per token (fp32 or bf16 out), or with
           4-bit activations

Weights come in the tiers the loader makes: one FP16 scale per 32 ("k32"), 64 ("k64") or 16
("k16") reduction elements, symmetric or with zero points.
"""
import ctypes as C
import importlib

import torch

pkg = importlib.import_module("knivesysl-xe_b200")


# ------------------------------------------------------------------------------- cases
def listed():
    return [
        # key or value projection of one token: the smallest call, two launches and their latency
        {"name": "proj1_kv", "kind": "proj1", "M": 1024, "K": 5120, "tier": "k32", "zp": True},
        # single-stream decoding: the MLP of one layer for one token, weights as the loader packs them
        {"name": "mlp1", "kind": "mlp1", "H": 5120, "I": 17408, "tier": "k64", "zp": True},
        # eight concurrent streams, fused gate|up, per-token scales (the benchmark's headline)
        {"name": "gate_up_8", "kind": "decode", "M": 17408, "K": 5120, "count": 2, "T": 8, "tier": "k64",
         "zp": False, "act": "token"},
        # the same batch through the down-projection in the reference's arithmetic
        {"name": "down_8", "kind": "decode", "M": 5120, "K": 17408, "count": 1, "T": 8, "tier": "k32",
         "zp": True, "act": "block"},
        # a batch that is no power of two (24 streams, or 3 drafts for each of 8)
        {"name": "down_24", "kind": "decode", "M": 5120, "K": 17408, "count": 1, "T": 24, "tier": "k32",
         "zp": False, "act": "token"},
        # a full decode batch in the reference's arithmetic
        {"name": "down_64", "kind": "decode", "M": 5120, "K": 17408, "count": 1, "T": 64, "tier": "k32",
         "zp": True, "act": "block"},
        # logits of a decode batch: the int8 output head
        {"name": "head_8", "kind": "head", "M": 65536, "K": 5120, "T": 8},
        # a short prompt through the attention input projection
        {"name": "prefill_136", "kind": "prefill", "M": 10240, "K": 5120, "T": 136, "tier": "k32", "zp": True,
         "act": "block", "segments": 1},
        # three prompts packed into one chunk, boundaries on any multiple of 8 tokens
        {"name": "prefill_1000", "kind": "prefill", "M": 5120, "K": 17408, "T": 1000, "tier": "k64", "zp": True,
         "act": "block", "segments": 3},
        # 4-bit activations: what the reference runs K64 weights at in prefill by default
        {"name": "prefill_1024_a4", "kind": "prefill", "M": 17408, "K": 5120, "T": 1024, "tier": "k64",
         "zp": True, "act": "int4", "segments": 1},
        # per-token scales with bf16 output
        {"name": "prefill_2048_bf16", "kind": "prefill", "M": 17408, "K": 5120, "T": 2048, "tier": "k64",
         "zp": False, "act": "token_bf16", "segments": 1},
        # the benchmark's packed prefill: four segments of 1024 in the reference's arithmetic
        {"name": "prefill_4096", "kind": "prefill", "M": 17408, "K": 5120, "T": 4096, "tier": "k64",
         "zp": False, "act": "block", "segments": 4},
    ]


def _log(rng, lo, hi, step):
    """A multiple of `step` in [lo, hi], spread evenly over the logarithm."""
    v = lo * (hi / lo) ** rng.random()
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choices(["proj1", "mlp1", "decode", "head", "prefill"], weights=[2, 1, 4, 1, 4])[0]
    zp = rng.random() < 0.5
    if kind == "proj1":
        tier = rng.choices(["k32", "k64", "k16"], weights=[3, 3, 1])[0]
        return {"kind": kind, "M": _log(rng, 256, 17408, 16), "K": _log(rng, 512, 17408, 64), "tier": tier, "zp": zp}
    if kind == "mlp1":
        return {"kind": kind, "H": _log(rng, 1024, 5120, 64), "I": _log(rng, 2048, 17408, 64),
                "tier": rng.choice(["k32", "k64"]), "zp": zp}
    if kind == "decode":
        tier = rng.choice(["k32", "k64"])
        count = rng.choice([1, 1, 2, 3])
        return {"kind": kind, "M": _log(rng, 512, 17408, 16), "K": _log(rng, 1024, 17408, 32 if tier == "k32" else 64),
                "count": count, "T": 8 * rng.randint(1, 8), "tier": tier, "zp": zp,
                "act": rng.choice(["token", "block"])}
    if kind == "head":
        return {"kind": kind, "M": _log(rng, 8192, 65536, 16), "K": _log(rng, 1024, 5120, 64),
                "T": rng.choice([1, 8, 8, 16, 32])}
    act = rng.choice(["block", "block", "token", "token_bf16", "int4"])
    tier = "k64" if act == "int4" else rng.choice(["k32", "k64"])
    T = _log(rng, 128, 4096, 8)
    # rows in whole blocks of 128 (what the per-token and 4-bit calls take) or, with block scales, of
    # 16; a chunk is never dearer than the largest listed one
    rows = 16 if act == "block" and rng.random() < 0.25 else 128
    M, K = _log(rng, 1024, 17408, rows), _log(rng, 1024, 17408, 64)
    limit = 2 ** 37 if rows == 128 else 2 ** 33
    while T * M * K > limit:
        if T >= 256:
            T = T // 16 * 8
        else:
            M, K = max(1024, M // 2 // rows * rows), max(1024, K // 2 // 64 * 64)
    return {"kind": kind, "M": M, "K": K, "T": T, "tier": tier, "zp": zp, "act": act,
            "segments": rng.randint(1, 4) if act == "block" else 1}


# ------------------------------------------------------------------------------ weights
_GROUP = {"k16": 16, "k32": 32, "k64": 64}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


class _Weight:
    """One packed W4 weight of N(0, 0.02) values: codes [M/16][K/32][16 rows][16 bytes], byte b of a
    row holding k = 2b and 2b + 1, and a scale word per (row, group): an FP16 scale whose low
    four mantissa bits hold the zero point."""

    def __init__(self, M, K, tier, zp, gen):
        grp = _GROUP[tier]
        self.codes = torch.empty(M // 16, K // 32, 16, 16, dtype=torch.uint8, device="cuda")
        self.scales = torch.empty(M // 16, K // grp, 16, dtype=torch.int16, device="cuda")
        for r0 in range(0, M, 2048):
            rows = min(2048, M - r0)
            w = torch.randn(rows, K // grp, grp, device="cuda", generator=gen) * 0.02
            if zp:      # asymmetric: the group's range on 16 levels, w ~= s (q - z)
                lo, hi = w.amin(2).clamp(max=0.0), w.amax(2).clamp(min=0.0)
                s = self._fp16_without_low_nibble((hi - lo) / 15.0)
                z = torch.round(-8.0 - lo / s.float()).clamp(-8, 7)
            else:
                s = self._fp16_without_low_nibble(w.abs().amax(2) / 7.0)
                z = torch.zeros_like(s, dtype=torch.float32)
            q = torch.round(w / s.float()[..., None] + z[..., None]).clamp(-8, 7).to(torch.int32) & 15
            word = (s.view(torch.int16) & ~15) | (z.to(torch.int16) & 15)
            q = q.reshape(rows // 16, 16, K // 32, 16, 2)
            packed = (q[..., 0] | (q[..., 1] << 4)).to(torch.uint8)
            self.codes[r0 // 16:(r0 + rows) // 16] = packed.transpose(1, 2)
            self.scales[r0 // 16:(r0 + rows) // 16] = word.reshape(rows // 16, 16, K // grp).transpose(1, 2)
        r = self.rec = pkg.TqWeight()
        r.M, r.K, r.Mt, r.Kt = M, K, M // 16, K // 32
        r.d_s4, r.d_s4_scale, r.s4_ready = self.codes.data_ptr(), self.scales.data_ptr(), 1
        r.s4_k16, r.s4_k64 = int(tier == "k16"), int(tier == "k64")
        self.ref = C.byref(r)

    @staticmethod
    def _fp16_without_low_nibble(s):
        bits = s.to(torch.float16).view(torch.int16).to(torch.int32)
        return ((bits + 8) & 0xFFF0).to(torch.int16).view(torch.float16)


class _Weight8:
    """One packed W8 weight: codes [M/16][K/32][16 rows][32 bytes], an FP16 scale per (row, K32)."""

    def __init__(self, M, K, gen):
        self.codes = torch.empty(M // 16, K // 32, 16, 32, dtype=torch.int8, device="cuda")
        self.scales = torch.empty(M // 16, K // 32, 16, dtype=torch.float16, device="cuda")
        for r0 in range(0, M, 4096):
            rows = min(4096, M - r0)
            w = torch.randn(rows // 16, 16, K // 32, 32, device="cuda", generator=gen) * 0.02
            s = (w.abs().amax(3) / 127.0).to(torch.float16)
            q = torch.round(w / s.float()[..., None]).clamp(-127, 127).to(torch.int8)
            self.codes[r0 // 16:(r0 + rows) // 16] = q.transpose(1, 2)
            self.scales[r0 // 16:(r0 + rows) // 16] = s.transpose(1, 2)
        r = self.rec = pkg.TqWeight()
        r.M, r.K, r.Mt, r.Kt = M, K, M // 16, K // 32
        r.d_s8, r.d_s8_scale, r.s8_ready = self.codes.data_ptr(), self.scales.data_ptr(), 1
        self.ref = C.byref(r)


def _activations(T, K, gen, wide):
    """Token rows in front of a projection: the MLP's SiLU(g) * u where K is the wide side, else
    normalised hidden rows with 1% outlier channels."""
    if wide:
        g, u = (torch.randn(T, K, device="cuda", generator=gen) for _ in range(2))
        return (torch.nn.functional.silu(g) * u).contiguous()
    x = torch.randn(T, K, device="cuda", generator=gen)
    x[:, torch.randperm(K, device="cuda", generator=gen)[:max(1, K // 100)]] *= 20.0
    return x


def _f32(*shape):
    return torch.empty(*shape, dtype=torch.float32, device="cuda")


def _i32(*shape):
    return torch.empty(*shape, dtype=torch.int32, device="cuda")


# ------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    lib = pkg.load()
    assert lib.tq_set_device(torch.cuda.current_device()) == 0
    gen = _generator(seed)
    s = {"case": case, "lib": lib}
    kind = case["kind"]
    if kind == "mlp1":
        H, I = case["H"], case["I"]
        s["gate"], s["up"] = (_Weight(I, H, case["tier"], case["zp"], gen) for _ in range(2))
        s["down"] = _Weight(H, I, case["tier"], case["zp"], gen)
        s["pair"] = pkg.weight_array([s["gate"], s["up"]])
        s["x"] = torch.randn(H, device="cuda", generator=gen)
        s["norm"] = (torch.randn(H, device="cuda", generator=gen) * 0.1).to(torch.bfloat16)
        s["xn"], s["g"], s["u"], s["h"], s["y"] = _f32(H), _f32(I), _f32(I), _f32(I), _f32(H)
        s["gu"] = (C.c_void_p * 2)(s["g"].data_ptr(), s["u"].data_ptr())
    else:
        M, K, T = case["M"], case["K"], case.get("T", 1)
        n = case.get("count", 1)
        if kind == "head":
            s["w"] = [_Weight8(M, K, gen)]
        else:
            s["w"] = [_Weight(M, K, case["tier"], case["zp"], gen) for _ in range(n)]
        s["ws"] = pkg.weight_array(s["w"])
        s["x"] = _activations(T, K, gen, K > M)
        bf16 = case.get("act") == "token_bf16"
        s["y"] = [torch.empty(T, M, dtype=torch.bfloat16 if bf16 else torch.float32, device="cuda") for _ in range(n)]
        s["ys"] = (C.c_void_p * n)(*[y.data_ptr() for y in s["y"]])
        nblk = K // 32 * T
        s["aq"] = torch.empty(nblk, 32, dtype=torch.int8, device="cuda")
        s["as"], s["asum"], s["as_tok"] = _f32(nblk), _i32(nblk), _f32(T)
        if case.get("segments", 1) > 1:
            k = case["segments"]
            cuts = [T * i // k // 8 * 8 for i in range(k)] + [T]
            s["offsets"] = (C.c_int * (k + 1))(*cuts)
    torch.cuda.synchronize()      # the library has a stream of its own
    return s


# ---------------------------------------------------------------------------------- run
def _ok(rc):
    if rc != 0:
        raise RuntimeError(f"projection call returned {rc}")


def run(s):
    case, lib = s["case"], s["lib"]
    kind, act = case["kind"], case.get("act")
    if kind == "mlp1":
        H, I = case["H"], case["I"]
        lib.qwn_x_rmsnorm_quant(s["xn"].data_ptr(), s["x"].data_ptr(), s["norm"].data_ptr(), H, 1e-6)
        _ok(lib.qwn_x_gemv_w4a8_fanout(s["pair"], s["gu"], 2))
        lib.qwn_x_silu_mul_quant(s["h"].data_ptr(), s["g"].data_ptr(), s["u"].data_ptr(), I)
        _ok(lib.qwn_x_gemv_w4a8_prepared(s["down"].ref, s["y"].data_ptr(), s["x"].data_ptr()))
        return [s["xn"], s["g"], s["u"], s["h"], s["y"]]
    K, T = case["K"], case.get("T", 1)
    x, w, y = s["x"].data_ptr(), s["w"][0].ref, s["ys"][0]
    if kind == "proj1":
        _ok(lib.qwn_x_gemv_w4a8(w, x, y))
        return s["y"]
    if kind == "head" and T == 1:
        _ok(lib.qwn_x_gemv_w8a8(w, x, y))
        return s["y"]
    aq, as_, asum, as_tok = (s[k].data_ptr() for k in ("aq", "as", "asum", "as_tok"))
    if act == "int4":
        lib.qwn_x_quantize_act_chunk_s4(x, K, T, aq, as_, asum)
        _ok(lib.qwn_x_gemm_w4a4(w, aq, as_, asum, y, T))
    elif act in ("token", "token_bf16"):
        lib.qwn_x_quantize_act_chunk_pertoken(x, K, T, aq, as_, asum, as_tok)
        if kind == "prefill":
            _ok(lib.qwn_x_gemm_w4a8_pertoken(w, aq, as_tok, asum, y, T, int(act == "token_bf16")))
        else:
            _ok(lib.qwn_x_gemm_w4a8_fanout_pertoken(s["ws"], s["ys"], case["count"], aq, as_tok, asum, T))
    else:
        lib.qwn_x_quantize_act_chunk(x, K, T, aq, as_, asum)
        if kind == "head":
            _ok(lib.qwn_x_gemm_w8a8(w, aq, as_, y, T))
        elif kind == "prefill":
            _ok(lib.qwn_x_gemm_w4a8(w, aq, as_, asum, y, T, s.get("offsets"),
                                    case["segments"] if "offsets" in s else 0))
        else:
            _ok(lib.qwn_x_gemm_w4a8_fanout(s["ws"], s["ys"], case["count"], aq, as_, asum, T, None, 0))
    return s["y"]


# ---------------------------------------------------------------------- work, tolerance
def _weight_bytes(M, K, tier):
    return M * K + M * (K // 32) * 2 if tier == "k8" else M * K // 2 + M * (K // _GROUP[tier]) * 2


def work(case):
    """fp32 rows in, weights in, results out, each once; two operations per multiply-add."""
    if case["kind"] == "mlp1":
        H, I, tier = case["H"], case["I"], case["tier"]
        weights = 2 * _weight_bytes(I, H, tier) + _weight_bytes(H, I, tier)
        # x and its norm weights in; the normalised row, gate, up, hidden and the result out
        return {"bytes": weights + 4 * H + 2 * H + 4 * (2 * H + 3 * I), "flops": 6 * H * I}
    M, K, T, n = case["M"], case["K"], case.get("T", 1), case.get("count", 1)
    tier = "k8" if case["kind"] == "head" else case["tier"]
    out = 2 if case.get("act") == "token_bf16" else 4
    return {"bytes": n * _weight_bytes(M, K, tier) + 4 * T * K + out * n * T * M, "flops": 2 * n * T * M * K}


def tolerance(case):
    """The integer dots are exact, so results differ between correct implementations by the order and
    contraction of the fp32 sums over the K groups. In mlp1 such a difference can move a value
    across a rounding boundary of the second quantisation, one step of 1/127 of its block's
    maximum; bf16 outputs can round to the other neighbour."""
    if case.get("act") == "token_bf16":
        return {"rel": 2e-4, "max": 1.6e-2}
    if case["kind"] == "mlp1":
        return {"rel": 6e-4}
    return {"rel": 2e-6, "max": 2e-5}


# ------------------------------------------------------------------------------- exact
def _dequantised(w):
    """Rows of a packed weight in 64 bits, a block of rows at a time: (first row, values)."""
    M, K = w.rec.M, w.rec.K
    for r0 in range(0, M, 1024):
        rows = min(1024, M - r0)
        t = slice(r0 // 16, (r0 + rows) // 16)
        if isinstance(w, _Weight8):
            s, z = w.scales[t].double(), 0.0
            q = w.codes[t].double()
        else:
            word = w.scales[t].to(torch.int32)
            s = (word & 0xFFF0).to(torch.int16).view(torch.float16).double()
            z = (((word & 15) ^ 8) - 8).double().transpose(1, 2).reshape(rows, -1, 1)
            c = w.codes[t].to(torch.int32)
            q = ((torch.stack((c & 15, c >> 4), -1) ^ 8) - 8).double()
        q = q.reshape(rows // 16, K // 32, 16, 32).transpose(1, 2).reshape(rows, K)
        s = s.transpose(1, 2).reshape(rows, -1, 1)
        yield r0, ((q.reshape(rows, s.shape[1], -1) - z) * s).reshape(rows, K)


def _quantised(x, block, levels):
    """Rows as their codes stand for them: one scale, the largest magnitude / levels, per block. The
    scale and the code are what fp32 gives (they are data to the sums), the product is exact."""
    v = x.float().reshape(x.shape[0], -1, block)
    top = v.abs().amax(2, keepdim=True)
    s = torch.where(top > 0, top / levels, torch.ones_like(top))
    return (torch.round(v / s).clamp(-levels, levels).double() * s.double()).reshape(x.shape)


def _project(w, xq):
    y = torch.empty(xq.shape[0], w.rec.M, dtype=torch.float64, device="cuda")
    for r0, v in _dequantised(w):
        y[:, r0:r0 + v.shape[0]] = xq @ v.T
    return y


def exact(case, seed):
    s = prepare(case, seed)
    if case["kind"] == "mlp1":
        x = s["x"].double()
        xn = x / torch.sqrt((x * x).mean() + 1e-6) * (1.0 + s["norm"].double())
        g, u = (_project(w, _quantised(xn[None], 32, 127))[0] for w in (s["gate"], s["up"]))
        h = g / (1.0 + torch.exp(-g)) * u
        return [xn, g, u, h, _project(s["down"], _quantised(h[None], 32, 127))[0] + x]
    act = case.get("act", "block")
    block, levels = (64, 7) if act == "int4" else ((case["K"], 127) if act.startswith("token") else (32, 127))
    xq = _quantised(s["x"], block, levels)
    return [_project(w, xq) for w in s["w"]]
