"""What this library is used for, as calls that can be timed and checked.

Every case goes through the C interface of lib/libefm_b200.so (include/efm_b200.h) as an engine calls it: weights, cache slots, sampling
parameters and captured steps are in hand before the call, token ids, pixels and embeddings come with it.  Four kinds:

  text     one request of the text tower: prompt behind a fixed prefix, then sampled tokens.  Token ids in; tokens, last logits and the slot's cache out.
  encode   one or more images through the vision encoder: pixel rows in, embeddings out, both on the device.
  act      one action chunk: camera images, prompt, robot state and noise in, actions out, all on the host.
  layered  a layered decoder: one request (prompt, then tokens on the captured step), or steps of many live requests over the paged
           cache with a portion of another prompt beside them.

Weights are random with the spread of trained ones: matrices keep unit scale, sublayers add a fraction of the residual stream, and the
output table leans towards a successor for every token, so that the next token is as clear as a trained model makes it and rounding
never picks another one.  Routers of experts read channels with well separated values for the same reason.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

DEV = "cuda"
BF16 = torch.bfloat16
LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "edge-fm-x_b200", "lib", "libefm_b200.so")
P, I32, F32 = C.c_void_p, C.c_int32, C.c_float
HOST, DEVICE, EFM_BF16, EFM_F16, EFM_I8 = 0, 1, 2, 1, 6


# ---- the interface ---------------------------------------------------------------------------------------------------------
def struct(name, **fields):
    """ctypes structure from `name_of_type="field field ..."` groups given in order: i = int32, f = float."""
    out = []
    for kind, names in fields.items():
        out += [(n, {"i": I32, "f": F32}[kind[0]]) for n in names.split()]
    return type(name, (C.Structure,), {"_fields_": out})


class ModelDesc(C.Structure):
    _fields_ = [(n, I32) for n in ("struct_size", "num_layers", "hidden", "q_heads", "kv_heads", "head_dim", "intermediate", "vocab")] + \
        [("rms_eps", F32), ("rope_theta", F32), ("tied_lm_head", I32), ("use_mrope", I32), ("mrope_section", I32 * 3),
         ("max_prefill_tokens", I32), ("max_response_tokens", I32)]


class Sampling(C.Structure):
    _fields_ = [("temperature", F32), ("top_p", F32), ("top_k", I32), ("reserved", C.c_uint32), ("seed", C.c_uint64)]


class VitDesc(C.Structure):
    _fields_ = [(n, I32) for n in ("struct_size", "depth", "hidden", "heads", "intermediate", "out_hidden", "patch", "temporal_patch",
                                   "in_channels", "merge", "window", "n_fullatt")] + \
        [("fullatt", I32 * 8), ("rms_eps", F32), ("rope_theta", F32), ("max_patches", I32)]


VlaDesc = struct("VlaDesc", i="struct_size image_size patch vit_layers vit_hidden vit_heads vit_mlp shuffle n_images hidden layers q_heads "
                 "kv_heads head_dim mlp vocab lang_tokens expert_hidden expert_mlp state_dim action_dim chunk steps",
                 f="rope_theta rms_eps ln_eps")
DecoderDesc = struct("DecoderDesc", i="struct_size num_layers vocab width side_dim", f="norm_eps", i2="compute_dtype max_step_tokens "
                     "max_response_tokens cache_pages state_slots max_slots norm_layout", f2="embed_scale", i3="loop_start loop_stop loop_times",
                     f3="residual_mult", i4="tied_head", f4="logit_scale logit_softcap", i5="conv_taps depth_average")


class DecoderLayer(C.Structure):
    _fields_ = struct("", i="mixer heads kv_heads dim vdim window distance_bias", f="scale", i2="decay_rank ff keep_first qk_norm head_temp "
                      "qkv_bias rot_kind rot_dims", f2="rot_base", i3="q_rank kv_rank sink out_gate experts expert_ff expert_top expert_groups "
                      "expert_groups_kept", f3="rot_factor rot_original rot_fast rot_slow", i4="ff_act expert_glu", f4="expert_limit",
                      i5="expert_score expert_weight_input shared_ff", f5="shared_limit", i6="linear_heads linear_dim linear_vdim",
                      f6="mix_scale linear_scale")._fields_ + \
        [("linear_decay", P), ("linear_norm", I32), ("linear_tau", F32), ("score_weights", I32), ("out_bias", I32), ("expert_scale", F32),
         ("shared_gate", I32)]


class StepEntry(C.Structure):
    _fields_ = [("slot", I32), ("n_tokens", I32), ("kv_offset", I32), ("n_want", I32), ("rng_step", C.c_uint32), ("reserved", C.c_uint32),
                ("tokens", P), ("want", P)]


SIGNATURES = {
    "efm_b200_create": [P, I32, I32, I32, P], "efm_b200_destroy": [P], "efm_b200_set_weight": [P, C.c_char_p, P, P, I32, I32, I32],
    "efm_b200_set_decode_weight": [P, C.c_char_p, P, P, I32, I32, I32], "efm_b200_finalize_weights": [P], "efm_b200_alloc_kv_slot": [P, I32, I32],
    "efm_b200_set_sampling": [P, P], "efm_b200_prefill": [P, I32, P, I32, I32, P, I32, I32, I32, P, I32], "efm_b200_set_prefill_graph": [P, I32],
    "efm_b200_set_prefill_attention": [P, I32], "efm_b200_decode_begin": [P, I32, I32, P, I32], "efm_b200_decode_steps": [P, I32, I32],
    "efm_b200_capture_decode": [P, I32], "efm_b200_kv_layer_ptr": [P, I32, I32, P, P], "efm_b200_read_tokens": [P, P, I32, I32], "efm_b200_read_logits": [P, P, I32], "efm_b200_synchronize": [P],
    "efm_b200_vit_create": [P, P, P], "efm_b200_vit_destroy": [P], "efm_b200_vit_set_weight": [P, C.c_char_p, P, P, I32, I32, I32],
    "efm_b200_vit_finalize_weights": [P], "efm_b200_vit_encode": [P, P, I32, P, I32, P, I32],
    "efm_b200_vla_create": [P, I32, P], "efm_b200_vla_destroy": [P], "efm_b200_vla_set_weight": [P, C.c_char_p, P, P, I32, I32, I32],
    "efm_b200_vla_finalize_weights": [P], "efm_b200_vla_chunk": [P, P, P, P, P, I32, P],
    "efm_b200_decoder_create": [P, P, I32, P], "efm_b200_decoder_map_slot": [P, I32, P, I32, I32], "efm_b200_decoder_pin_prefix": [P, I32, I32],
    "efm_b200_decoder_step": [P, P, I32, P, P],
}
_lib = None


def lib():
    global _lib
    if _lib is None:
        _lib = C.CDLL(LIB)
        for name, args in SIGNATURES.items():
            fn = getattr(_lib, name)
            fn.restype, fn.argtypes = I32, args
        _lib.efm_b200_last_error.restype, _lib.efm_b200_last_error.argtypes = C.c_char_p, [P]
        _lib.efm_b200_vla_last_error.restype, _lib.efm_b200_vla_last_error.argtypes = C.c_char_p, [P]
    return _lib


def i32(values):
    return np.ascontiguousarray(values, dtype=np.int32)


def at(array):
    """Address of an array's or tensor's values (None: no pointer)."""
    return None if array is None else array.data_ptr() if isinstance(array, torch.Tensor) else array.ctypes.data


class Handle:
    """A context (`of` "") or a policy ("vla_"); every call raises on a status other than 0."""

    def __init__(self, create, *args, of=""):
        self.h, self.of = P(), of
        self.status("create", getattr(lib(), create)(*args, C.byref(self.h)))

    def status(self, what, st):
        if st != 0:
            text = lib().efm_b200_vla_last_error(self.h) if self.of else lib().efm_b200_last_error(self.h)
            raise RuntimeError("%s: status %d: %s" % (what, st, (text or b"").decode()))

    def __call__(self, name, *args):
        self.status(name, getattr(lib(), "efm_b200_" + name)(self.h, *args))

    def weight(self, name, t, call=None, on=None):
        torch.cuda.current_stream().synchronize()
        code = {BF16: EFM_BF16, torch.float16: EFM_F16, torch.int8: EFM_I8}[t.dtype]
        shape = (C.c_int64 * t.dim())(*t.shape)
        self.status(name, getattr(lib(), "efm_b200_" + (call or self.of + "set_weight"))(on or self.h, name.encode(), t.data_ptr(), shape, t.dim(), code, DEVICE))

    def __del__(self):
        if self.h:
            getattr(lib(), "efm_b200_%sdestroy" % self.of)(self.h)
            self.h = P()


def generator(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1_000_003 * int(seed) + salt)


def matrix(g, rows, cols, gain=1.0):
    return torch.randn(rows, cols, generator=g, device=DEV, dtype=BF16).mul_(gain * cols ** -0.5)


def vector(g, n, std=0.1, mean=0.0):
    return torch.randn(n, generator=g, device=DEV, dtype=BF16).mul_(std).add_(mean)


def ids(g, n, vocab):
    return torch.randint(0, vocab, (n,), generator=g, device=DEV).cpu().numpy().astype(np.int32)


# the token that the output table leans to behind token t: t * STEP + 1, a permutation as no vocabulary here is a multiple of STEP
STEP = 7919


def successor(t, vocab):
    return (t * STEP + 1) % vocab


def leaning_head(g, embed, share=0.5):
    V, W = embed.shape
    head = matrix(g, V, W, math.sqrt(1 - share * share))
    t = torch.arange(V, device=DEV)
    head[successor(t, V)] += embed * (share * W ** -0.5)
    return head


def rms(x, w=None, eps=1e-6):
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return x if w is None else x * w.double()


def lin(x, w, b=None):
    y = x @ w.double().T
    return y if b is None else y + b.double()


def attend(q, k, v, scale, visible, sink=None):
    """q [T, H, D], k [S, G, D], v [S, G, Dv], visible [T, S] -> [T, H * Dv]; sink [H]: exp(sink) more in the denominators."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        s = s.masked_fill(~visible, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].double().expand(T, 1)], 1)
        p = torch.softmax(s, -1)
        out.append(p[:, :k.shape[0]] @ v[:, h * G // H])
    return torch.stack(out, 1).reshape(T, -1)


def turn(x, angle, pairs=False):
    """x [T, H, D], angle [T, n]: channel i turns with i + n (pairs: 2 i with 2 i + 1), channels >= 2 n pass."""
    n = angle.shape[1]
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    if pairs:
        u, v = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
        turned = torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    else:
        u, v = x[..., :n], x[..., n:2 * n]
        turned = torch.cat([u * c - v * s, v * c + u * s], -1)
    return torch.cat([turned, x[..., 2 * n:]], -1)


def angles(pos, dims, base):
    return pos.double()[:, None] * base ** (-torch.arange(0, dims, 2, device=DEV, dtype=torch.float64) / dims)


def causal(T, window=0, keep=0):
    i, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None]
    see = j <= i
    return see if not window else see & ((i - j < window) | (j < keep))


# ---- text: the Qwen2.5 / Qwen2.5-VL text tower -----------------------------------------------------------------------------
# layers, hidden, query heads, key heads, head dim, feed-forward, vocabulary, M-RoPE
TEXT = {
    "0.5B": (24, 896, 14, 2, 64, 4864, 151936, False),
    "1.5B": (28, 1536, 12, 2, 128, 8960, 151936, False),
    "VL-3B": (36, 2048, 16, 2, 128, 11008, 151936, True),
    "VL-7B": (28, 3584, 28, 4, 128, 18944, 152064, True),
}
SECTION = (16, 24, 24)
LINEARS = ("self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj", "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj")


def text(name=None, *, model="0.5B", prefix=0, prompt=64, rows=0, columns=0, tokens=1, temperature=0.0, top_p=1.0, int8=False, int4=False):
    """rows x columns merged image tokens stand in front of the prompt; int8: INT8 prefill attention; int4: INT4 decode weights."""
    case = dict(kind="text", model=model, prefix=prefix, prompt=prompt, rows=rows, columns=columns, tokens=tokens, temperature=temperature,
                top_p=top_p, int8=int8, int4=int4)
    return case if name is None else dict(case, name=name)


def text_weights(model, seed):
    """(name, tensor) in the checkpoint's names."""
    L, W, H, G, D, F, V, _ = TEXT[model]
    g = generator(seed)
    add = 2.0 / math.sqrt(2 * L)                 # what the sublayers add together stays below the embedding
    embed = torch.randn(V, W, generator=g, device=DEV, dtype=BF16)
    yield "model.embed_tokens.weight", embed
    yield "lm_head.weight", leaning_head(g, embed)
    yield "model.norm.weight", vector(g, W, mean=1.0)
    for i in range(L):
        p = "model.layers.%d." % i
        yield p + "input_layernorm.weight", vector(g, W, mean=1.0)
        yield p + "post_attention_layernorm.weight", vector(g, W, mean=1.0)
        for n, r, k, gain in (("q", H * D, W, 1.4), ("k", G * D, W, 1.4), ("v", G * D, W, 1.0)):
            yield p + "self_attn.%s_proj.weight" % n, matrix(g, r, k, gain)
            yield p + "self_attn.%s_proj.bias" % n, vector(g, r)
        yield p + "self_attn.o_proj.weight", matrix(g, W, H * D, add)
        yield p + "mlp.gate_proj.weight", matrix(g, F, W)
        yield p + "mlp.up_proj.weight", matrix(g, F, W)
        yield p + "mlp.down_proj.weight", matrix(g, W, F, add)


def int4_of(w):
    """(values in [-8, 7] [N, K], scale per row and 128 columns as stored, [K / 128, N])."""
    N, K = w.shape
    x = w.float().view(N, K // 128, 128)
    s = (x.abs().amax(2) / 7.0).clamp_min(1e-8).half()
    return (x / s.float()[:, :, None]).round_().clamp_(-8, 7).to(torch.int8).view(N, K), s.T.contiguous()


def text_inputs(case, seed):
    """Ids of the prefix and of the request (an image's rows as ids from the vocabulary's end on), embeddings, M-RoPE positions of both
    and of the first sampled token."""
    V, W = TEXT[case["model"]][6], TEXT[case["model"]][1]
    g, n_img = generator(seed, 1), case["rows"] * case["columns"]
    prefix, words = ids(g, case["prefix"], V), ids(g, case["prompt"], V)
    request = np.concatenate([np.arange(V, V + n_img, dtype=np.int32), words])
    embeds = torch.randn(n_img, W, generator=g, device=DEV, dtype=BF16) if n_img else None
    start = case["prefix"] + max(case["rows"], case["columns"])
    place = np.arange(start, start + len(words))
    r, c = np.meshgrid(np.arange(case["rows"]), np.arange(case["columns"]), indexing="ij")
    image = case["prefix"] + np.stack([np.zeros(n_img, np.int64), r.reshape(-1), c.reshape(-1)])
    pos = i32(np.concatenate([image, np.stack([place] * 3)], 1))
    return prefix, request, embeds, pos, int(place[-1]) + 1


class CacheLayer:
    """K and V of one layer of a slot, bf16 [2, tokens, key heads * head dim], as a tensor that keeps the context."""

    def __init__(self, ctx, layer, shape):
        base = P()
        ctx("kv_layer_ptr", 0, layer, C.byref(base), None)
        self.ctx, self.__cuda_array_interface__ = ctx, dict(shape=shape, typestr="<i2", data=(base.value, False), version=2)


class Text:
    def __init__(self, case, seed):
        L, W, H, G, D, F, V, mrope = TEXT[case["model"]]
        self.case, self.V, self.mrope = case, V, mrope
        self.prefix, self.request, self.embeds, self.pos, first = text_inputs(case, seed)
        n = len(self.prefix) + len(self.request)
        desc = ModelDesc(C.sizeof(ModelDesc), L, W, H, G, D, F, V, 1e-6, 1e6, 0, int(mrope), SECTION, 2048, case["tokens"])
        self.ctx = c = Handle("efm_b200_create", C.byref(desc), 0, 0, 1)
        for name, t in text_weights(case["model"], seed):
            c.weight(name, t)
            linear = name[:-7]
            if case["int4"] and (linear == "lm_head" or linear.endswith(LINEARS)) and t.dim() == 2:
                q, s = int4_of(t)
                u = q.view(torch.uint8) + 8
                c.weight(linear + ".qweight", (u[0::2] | (u[1::2] << 4)).view(torch.int8), "set_decode_weight")
                c.weight(linear + ".scaling_factors", s, "set_decode_weight")
        c("finalize_weights")
        room = n + case["tokens"] - 1            # the last token is not fed back
        c("alloc_kv_slot", 0, room)
        c("set_sampling", C.byref(Sampling(case["temperature"], case["top_p"], 0, 0, seed)))
        if case["int8"]:
            c("set_prefill_attention", 1)
        c("set_prefill_graph", 1)
        if len(self.prefix):                     # the fixed prefix and the decode step's graph belong to an engine's start
            pos = i32([np.arange(len(self.prefix))] * 3)
            c("prefill", 0, at(self.prefix), len(self.prefix), 0, None, 0, -1, HOST, at(pos) if mrope else None, 0)
        c("capture_decode", 0)
        c("synchronize")
        self.tokens = np.empty(case["tokens"], np.int32)
        self.logits = torch.empty(V, dtype=torch.float32, pin_memory=True)
        self.first = i32([first] * 3)
        self.cache = [torch.as_tensor(CacheLayer(c, i, (2, room, G * D)), device=DEV).view(BF16) for i in range(L)]

    def run(self):
        c, k, n0, n = self.ctx, self.case["tokens"], len(self.prefix), len(self.request)
        n_img = 0 if self.embeds is None else self.embeds.shape[0]
        c("prefill", 0, at(self.request), n, n0, at(self.embeds), n_img, self.V if n_img else -1, DEVICE, at(self.pos) if self.mrope else None, 1)
        if k > 1:
            c("decode_begin", 0, n0 + n, at(self.first), 1)
            c("decode_steps", k - 1, 1)
        c("read_tokens", at(self.tokens), 0, k)
        c("read_logits", at(self.logits), self.V)
        return {"tokens": self.tokens, "logits": self.logits, "cache": self.cache}


def text_exact(case, seed):
    L, W, H, G, D, F, V, mrope = TEXT[case["model"]]
    w = dict(text_weights(case["model"], seed))
    prefix, request, embeds, pos, first = text_inputs(case, seed)
    n_img, k = case["rows"] * case["columns"], case["tokens"]
    chain = [successor(int(request[-1]), V)]
    while len(chain) < k:
        chain.append(successor(chain[-1], V))
    words = torch.tensor(np.concatenate([prefix, request[n_img:], chain[:k - 1]]).astype(np.int64), device=DEV)
    x = w["model.embed_tokens.weight"][words].double()
    if n_img:
        x = torch.cat([x[:len(prefix)], embeds.double(), x[len(prefix):]])
    T, n = x.shape[0], len(prefix) + len(request)
    if mrope:
        more = np.arange(first, first + k - 1)
        place = np.concatenate([np.stack([np.arange(len(prefix))] * 3), pos, np.stack([more] * 3)], 1)
        section = np.repeat(np.arange(3), SECTION)
        a = torch.tensor(place[section].T, device=DEV).double() * 1e6 ** (-torch.arange(0, D, 2, device=DEV, dtype=torch.float64) / D)
    else:
        a = angles(torch.arange(T, device=DEV), D, 1e6)

    def product(x, name):                        # rows of decode steps read the INT4 weights where there are any
        y = lin(x[:n] if case["int4"] else x, w[name + ".weight"], w.get(name + ".bias"))
        if case["int4"] and T > n:
            q, s = int4_of(w[name + ".weight"])
            full = (q.double().view(q.shape[0], -1, 128) * s.T.double()[:, :, None]).view(q.shape)
            y = torch.cat([y, lin(x[n:], full, w.get(name + ".bias"))])
        return y

    see, cache = causal(T), []
    for i in range(L):
        p = "model.layers.%d." % i
        h = rms(x, w[p + "input_layernorm.weight"])
        q, kk, v = (product(h, p + "self_attn.%s_proj" % m).view(T, -1, D) for m in "qkv")
        kk = turn(kk, a)
        cache.append(torch.stack([kk, v]).flatten(2).cpu())
        x = x + product(attend(turn(q, a), kk, v, D ** -0.5, see), p + "self_attn.o_proj")
        h = rms(x, w[p + "post_attention_layernorm.weight"])
        z = product(h, p + "mlp.gate_proj")
        x = x + product(z * torch.sigmoid(z) * product(h, p + "mlp.up_proj"), p + "mlp.down_proj")
    h = rms(x, w["model.norm.weight"])
    if k == 1:
        logits = lin(h[-1:], w["lm_head.weight"])
    else:
        logits = torch.cat([lin(h[n - 1:n], w["lm_head.weight"]), product(h, "lm_head")[n:]])
    return {"tokens": logits.argmax(1).int().cpu().numpy(), "logits": logits[-1].cpu(), "cache": cache}


def text_work(case):
    L, W, H, G, D, F, V, _ = TEXT[case["model"]]
    layer = W * (2 * H + 2 * G) * D + 3 * W * F
    n0, n, k = case["prefix"], case["rows"] * case["columns"] + case["prompt"], case["tokens"]
    cache = 4 * L * G * D                        # bytes of a position
    one = (L * layer + W * V) * (0.5 + 2 / 128 if case["int4"] else 2)
    steps = sum(one + (n0 + n + s) * cache for s in range(k - 1))
    pairs = n * n0 + n * (n + 1) / 2 + sum(n0 + n + s for s in range(1, k))
    return {"bytes": 2 * (L * layer + W * V) + n * W * 2 + (n0 + n) * cache + steps + 4 * V,
            "flops": 2 * L * layer * (n + k - 1) + 2 * W * V * k + 4 * L * H * D * pairs}


# ---- encode: the Qwen2.5-VL vision encoder ---------------------------------------------------------------------------------
VIT = dict(depth=32, hidden=1280, heads=16, ffn=3420, full=(7, 15, 23, 31))


def encode(name=None, *, height=32, width=32, images=1, out=2048):
    """Patch grid (14-pixel patches) of every image, width of the produced embeddings."""
    case = dict(kind="encode", height=height, width=width, images=images, out=out)
    return case if name is None else dict(case, name=name)


def encode_weights(case, seed):
    g, W, F = generator(seed), VIT["hidden"], VIT["ffn"]
    yield "visual.patch_embed.proj.weight", matrix(g, W, 1176).view(W, 3, 2, 14, 14)
    for i in range(VIT["depth"]):
        p = "visual.blocks.%d." % i
        for n in ("norm1", "norm2"):
            yield p + n + ".weight", vector(g, W, mean=1.0)
        for n, r, k, gain in (("attn.qkv", 3 * W, W, 1.2), ("attn.proj", W, W, 0.3), ("mlp.gate_proj", F, W, 1.0), ("mlp.up_proj", F, W, 1.0),
                              ("mlp.down_proj", W, F, 0.3)):
            yield p + n + ".weight", matrix(g, r, k, gain)
            yield p + n + ".bias", vector(g, r)
    yield "visual.merger.ln_q.weight", vector(g, W, mean=1.0)
    for n, r in (("0", 4 * W), ("2", case["out"])):
        yield "visual.merger.mlp.%s.weight" % n, matrix(g, r, 4 * W)
        yield "visual.merger.mlp.%s.bias" % n, vector(g, r)


def encode_pixels(case, seed):
    """RGB uniform in [0, 1], normalised, in the image processor's row order."""
    n = case["images"] * case["height"] * case["width"]
    x = torch.rand(n, 3, 392, generator=generator(seed, 1), device=DEV)
    mean, std = (torch.tensor(v, device=DEV)[None, :, None] for v in ((0.48, 0.46, 0.41), (0.27, 0.26, 0.28)))
    return ((x - mean) / std).view(n, 1176).to(BF16)


class Encode:
    def __init__(self, case, seed):
        n = case["images"] * case["height"] * case["width"]
        desc = ModelDesc(C.sizeof(ModelDesc), 1, 128, 2, 1, 64, 64, 64, 1e-6, 1e6, 1, 0, (0, 0, 0), 16, 1)     # the text context it shares a stream with
        self.ctx = Handle("efm_b200_create", C.byref(desc), 0, 0, 1)
        full = VIT["full"]
        vit = VitDesc(C.sizeof(VitDesc), VIT["depth"], VIT["hidden"], VIT["heads"], VIT["ffn"], case["out"], 14, 2, 3, 2, 112, len(full),
                      full + (0,) * (8 - len(full)), 1e-6, 1e4, n)
        self.vit = P()
        self.ctx("vit_create", C.byref(vit), C.byref(self.vit))
        for name, t in encode_weights(case, seed):
            self.ctx.weight(name, t, "vit_set_weight", self.vit)
        self.ctx.status("vit_finalize_weights", lib().efm_b200_vit_finalize_weights(self.vit))
        self.pixels = encode_pixels(case, seed)
        self.grids = i32([(1, case["height"], case["width"])] * case["images"])
        self.out = torch.empty(n // 4, case["out"], dtype=BF16, device=DEV)
        torch.cuda.current_stream().synchronize()

    def run(self):
        self.ctx.status("vit_encode", lib().efm_b200_vit_encode(self.vit, at(self.pixels), DEVICE, at(self.grids), len(self.grids), at(self.out), DEVICE))
        self.ctx("synchronize")                  # the embeddings are on another stream than torch's
        return self.out

    def __del__(self):
        if getattr(self, "vit", None):
            lib().efm_b200_vit_destroy(self.vit)
            self.vit = None


def encode_exact(case, seed):
    w = {k[7:]: v for k, v in encode_weights(case, seed)}
    h, wd, H, D = case["height"], case["width"], VIT["heads"], VIT["hidden"] // VIT["heads"]
    n = h * wd
    pixels = encode_pixels(case, seed)
    # patch row / column of an input row: 2 x 2 blocks of patches, blocks in rows
    b, e = torch.arange(n, device=DEV) // 4, torch.arange(n, device=DEV) % 4
    row, col = b // (wd // 2) * 2 + e // 2, b % (wd // 2) * 2 + e % 2
    a = torch.cat([angles(row, D // 2, 1e4), angles(col, D // 2, 1e4)], 1)
    window = row // 8 * 10_000 + col // 8
    same, everything = window[:, None] == window[None], torch.ones(n, n, dtype=torch.bool, device=DEV)
    out = []
    for img in range(case["images"]):
        x = lin(pixels[img * n:(img + 1) * n].double(), w["patch_embed.proj.weight"].view(-1, 1176))
        for i in range(VIT["depth"]):
            p = "blocks.%d." % i
            q, k, v = lin(rms(x, w[p + "norm1.weight"]), w[p + "attn.qkv.weight"], w[p + "attn.qkv.bias"]).view(n, 3, H, D).unbind(1)
            y = attend(turn(q, a), turn(k, a), v, D ** -0.5, everything if i in VIT["full"] else same)
            x = x + lin(y, w[p + "attn.proj.weight"], w[p + "attn.proj.bias"])
            y = rms(x, w[p + "norm2.weight"])
            z, u = (lin(y, w[p + "mlp.%s_proj.weight" % m], w[p + "mlp.%s_proj.bias" % m]) for m in ("gate", "up"))
            x = x + lin(z * torch.sigmoid(z) * u, w[p + "mlp.down_proj.weight"], w[p + "mlp.down_proj.bias"])
        y = lin(rms(x, w["merger.ln_q.weight"]).view(n // 4, -1), w["merger.mlp.0.weight"], w["merger.mlp.0.bias"])
        out.append(lin(0.5 * y * (1 + torch.erf(y / math.sqrt(2))), w["merger.mlp.2.weight"], w["merger.mlp.2.bias"]))
    return torch.cat(out)


def encode_work(case):
    W, F, L, full = VIT["hidden"], VIT["ffn"], VIT["depth"], len(VIT["full"])
    h, w = case["height"], case["width"]
    n = case["images"] * h * w

    def spans(x):                                # sizes of the 8-patch windows along a side
        return [min(8, x - i) for i in range(0, x, 8)]
    inside = sum((r * c) ** 2 for r in spans(h) for c in spans(w)) * case["images"]
    weights = L * (4 * W * W + 3 * W * F) + W * 1176 + 16 * W * W + 4 * W * case["out"]
    pairs = full * case["images"] * (h * w) ** 2 + (L - full) * inside
    return {"bytes": 2 * weights + 2 * n * 1176 + 2 * n // 4 * case["out"],
            "flops": 2 * n * (L * (4 * W * W + 3 * W * F) + W * 1176) + 2 * (n // 4) * (16 * W * W + 4 * W * case["out"]) + 4 * W * pairs}


# ---- act: the SmolVLA-shaped action chunk ----------------------------------------------------------------------------------
VLA = dict(patch=16, vit_layers=12, vit_hidden=768, vit_heads=12, vit_mlp=3072, shuffle=4, hidden=960, layers=16, q_heads=15, kv_heads=5, head_dim=64,
           mlp=2560, vocab=49152, expert_hidden=720, expert_mlp=2048, state_dim=32, action_dim=32)


def act(name=None, *, images=3, size=512, words=48, chunk=50, steps=10):
    case = dict(kind="act", images=images, size=size, words=words, chunk=chunk, steps=steps)
    return case if name is None else dict(case, name=name)


def act_weights(case, seed):
    m, g = VLA, generator(seed)
    Hv, H, E, QD, KD = m["vit_hidden"], m["hidden"], m["expert_hidden"], m["q_heads"] * 64, m["kv_heads"] * 64

    def dense(name, r, k, bias=True):
        yield name + ".weight", matrix(g, r, k, 0.5)
        if bias:
            yield name + ".bias", vector(g, r, 0.02)
    yield from dense("vit.patch", Hv, 3 * m["patch"] ** 2)
    yield "vit.pos", vector(g, (case["size"] // m["patch"]) ** 2 * Hv, 0.02).view(-1, Hv)
    for i in range(m["vit_layers"]):
        p = "vit.%d." % i
        for n in ("ln1", "ln2"):
            yield p + n + ".weight", vector(g, Hv, 0.02, 1.0)
            yield p + n + ".bias", vector(g, Hv, 0.02)
        for n, r, k in [(c, Hv, Hv) for c in "qkvo"] + [("fc1", m["vit_mlp"], Hv), ("fc2", Hv, m["vit_mlp"])]:
            yield from dense(p + n, r, k)
    yield "vit.post_ln.weight", vector(g, Hv, 0.02, 1.0)
    yield "vit.post_ln.bias", vector(g, Hv, 0.02)
    yield from dense("connector", H, Hv * m["shuffle"] ** 2, False)
    yield "embed", vector(g, m["vocab"] * H, 0.02).view(-1, H)
    yield from dense("state_proj", H, m["state_dim"])
    for tower, W, F in (("vlm", H, m["mlp"]), ("expert", E, m["expert_mlp"])):
        for i in range(m["layers"]):
            p, kin = "%s.%d." % (tower, i), KD if tower == "expert" and i % 2 else W
            yield p + "norm1", vector(g, W, 0.02, 1.0)
            yield p + "norm2", vector(g, W, 0.02, 1.0)
            for n, r, k in (("q", QD, W), ("k", KD, kin), ("v", KD, kin), ("o", W, QD), ("gate", F, W), ("up", F, W), ("down", W, F)):
                yield from dense(p + n, r, k, False)
    yield "expert.norm", vector(g, E, 0.02, 1.0)
    for n, r, k in (("action_in", E, m["action_dim"]), ("time_in", E, 2 * E), ("time_out", E, E), ("action_out", m["action_dim"], E)):
        yield from dense(n, r, k)


def act_inputs(case, seed):
    g = torch.Generator().manual_seed(int(seed) + 4242)
    images = torch.rand(case["images"], 3, case["size"], case["size"], generator=g) * 2 - 1
    words = torch.randint(0, VLA["vocab"], (case["words"],), generator=g, dtype=torch.int32)
    state = torch.rand(VLA["state_dim"], generator=g) * 2 - 1
    return images, words, state, torch.randn(case["chunk"], VLA["action_dim"], generator=g)


class Act:
    def __init__(self, case, seed):
        sizes = dict(VLA, image_size=case["size"], n_images=case["images"], lang_tokens=case["words"], chunk=case["chunk"], steps=case["steps"])
        desc = VlaDesc(struct_size=C.sizeof(VlaDesc), rope_theta=1e5, rms_eps=1e-5, ln_eps=1e-6, **sizes)
        self.pol = Handle("efm_b200_vla_create", C.byref(desc), 0, of="vla_")
        for name, t in act_weights(case, seed):
            self.pol.weight(name, t)
        self.pol("vla_finalize_weights")
        self.inputs = [t.pin_memory() for t in act_inputs(case, seed)]
        self.out = torch.empty(case["chunk"], VLA["action_dim"], pin_memory=True)

    def run(self):
        self.pol("vla_chunk", *(at(t) for t in self.inputs), HOST, at(self.out))
        return self.out


def act_exact(case, seed):
    m, w = VLA, dict(act_weights(case, seed))
    images, words, state, noise = (t.to(DEV) for t in act_inputs(case, seed))
    L, D, H = m["layers"], 64, m["hidden"]
    side, Hv, n_img, s = case["size"] // m["patch"], m["vit_hidden"], case["images"], m["shuffle"]

    def dense(x, name):
        return lin(x, w[name + ".weight"], w.get(name + ".bias"))

    def norm(x, name):
        x = x - x.mean(-1, keepdim=True)
        return rms(x, w[name + ".weight"], 1e-6) + w[name + ".bias"].double()

    def glu(x, p):
        z = dense(x, p + "gate")
        return dense(z * torch.sigmoid(z) * dense(x, p + "up"), p + "down")
    tokens = []
    for img in images.double():
        x = img.view(3, side, 16, side, 16).permute(1, 3, 0, 2, 4).reshape(side * side, -1)
        x = dense(x, "vit.patch") + w["vit.pos"].double()
        everything = torch.ones(side * side, side * side, dtype=torch.bool, device=DEV)
        for i in range(m["vit_layers"]):
            p = "vit.%d." % i
            h = norm(x, p + "ln1")
            q, k, v = (dense(h, p + c).view(-1, m["vit_heads"], 64) for c in "qkv")
            x = x + dense(attend(q, k, v, 0.125, everything), p + "o")
            x = x + dense(torch.nn.functional.gelu(dense(norm(x, p + "ln2"), p + "fc1"), approximate="tanh"), p + "fc2")
        x = norm(x, "vit.post_ln").view(side // s, s, side // s, s, Hv).permute(0, 2, 1, 3, 4).reshape(-1, s * s * Hv)
        tokens.append(dense(x, "connector"))
    x = torch.cat([torch.cat(tokens) * math.sqrt(H), w["embed"][words.long()].double() * math.sqrt(H), dense(state.double()[None], "state_proj")])
    N, n = x.shape[0], case["chunk"]
    see = torch.ones(N, N, dtype=torch.bool, device=DEV)
    see[:N - 1, N - 1] = False
    a, cache = angles(torch.arange(N + n, device=DEV), D, 1e5), []
    for i in range(L):
        p = "vlm.%d." % i
        h = rms(x, w[p + "norm1"], 1e-5)
        q, k, v = (dense(h, p + c).view(N, -1, D) for c in "qkv")
        q, k = turn(q, a[:N]), turn(k, a[:N])
        cache.append((k, v))
        x = x + dense(attend(q, k, v, 0.125, see), p + "o")
        x = x + glu(rms(x, w[p + "norm2"], 1e-5), p)
    period = 4e-3 * (4.0 / 4e-3) ** torch.linspace(0, 1, m["expert_hidden"] // 2, dtype=torch.float64, device=DEV)
    over = torch.ones(n, N, dtype=torch.bool, device=DEV)
    y = noise.double()
    for t in range(case["steps"]):
        angle = 2 * math.pi / period * (1.0 - t / case["steps"])
        time = torch.cat([angle.sin(), angle.cos()]).expand(n, -1)
        z = dense(torch.cat([dense(y, "action_in"), time], 1), "time_in")
        x = dense(z * torch.sigmoid(z), "time_out")
        for i in range(L):
            p, (k, v) = "expert.%d." % i, cache[i]
            h = rms(x, w[p + "norm1"], 1e-5)
            q = dense(h, p + "q").view(n, -1, D)
            if i % 2 == 0:
                own_k, own_v = (dense(h, p + c).view(n, -1, D) for c in "kv")
                o = attend(turn(q, a[N:]), torch.cat([k, turn(own_k, a[N:])]), torch.cat([v, own_v]), 0.125, torch.cat([over, causal(n)], 1))
            else:
                k, v = (dense(c.reshape(N, -1), p + b).view(N, -1, D) for c, b in ((k, "k"), (v, "v")))
                o = attend(turn(q, a[:n]), k, v, 0.125, over)
            x = x + dense(o, p + "o")
            x = x + glu(rms(x, w[p + "norm2"], 1e-5), p)
        y = y - dense(rms(x, w["expert.norm"], 1e-5), "action_out") / case["steps"]
    return y.cpu()


def act_work(case):
    m = VLA
    Hv, H, E, QD, KD, L, n = m["vit_hidden"], m["hidden"], m["expert_hidden"], m["q_heads"] * 64, m["kv_heads"] * 64, m["layers"], case["chunk"]
    patches = (case["size"] // m["patch"]) ** 2
    rows, tokens = case["images"] * patches, case["images"] * patches // m["shuffle"] ** 2
    N = tokens + case["words"] + 1
    tower = m["vit_layers"] * (4 * Hv * Hv + 2 * Hv * m["vit_mlp"]) + 3 * m["patch"] ** 2 * Hv
    backbone = L * (H * (2 * QD + 2 * KD) + 3 * H * m["mlp"])
    expert = L * (2 * E * QD + 3 * E * m["expert_mlp"]) + L // 2 * 2 * E * KD + 3 * E * E + 2 * E * m["action_dim"]
    bridge = L // 2 * 2 * KD * KD
    connector = H * Hv * m["shuffle"] ** 2
    flops = 2 * rows * tower + 4 * m["vit_layers"] * rows * patches * Hv + 2 * tokens * connector + N * 2 * (backbone + bridge) + 4 * L * N * N * QD
    flops += case["steps"] * (2 * n * expert + 4 * QD * n * (L * N + L // 2 * (n + 1) / 2))
    return {"bytes": 2 * (tower + backbone + bridge + connector) + 2 * expert * case["steps"] + 12 * case["images"] * case["size"] ** 2, "flops": flops}


# ---- layered: decoders listed layer by layer -------------------------------------------------------------------------------
# Folizen: windowed attention with a feed-forward and the generalised delta rule in turn, a token input behind every layer.
# Temuvik: latent attention and windowed attention that keeps the first tokens in turn, routed experts everywhere.
# width: heads, key heads (128 channels), feed-forward
LAYERED = {1024: (8, 2, 4096), 2048: (16, 4, 8192)}
SIDE, RANK, KEEP, VOCAB = 64, 64, 16, 32768
EXPERTS, TOP, GROUPS, GROUPS_KEPT, KV_RANK, ROT = 32, 4, 4, 2, 512, 64


def layered(name=None, *, design="Folizen", width=2048, layers=8, window=1024, prompt=512, tokens=32, live=0, portion=0):
    """live = 0: one request, `tokens` tokens behind a prompt.  live > 0: `tokens` steps of as many requests, whose contexts run up to
    `prompt` tokens, with `portion` tokens of one more request's prompt in each step."""
    case = dict(kind="layered", design=design, width=width, layers=layers, window=window, prompt=prompt, tokens=tokens, live=live, portion=portion)
    return case if name is None else dict(case, name=name)


def layered_weights(case, seed):
    W, (H, G, F) = case["width"], LAYERED[case["width"]]
    g, folizen = generator(seed), case["design"] == "Folizen"
    embed = torch.randn(VOCAB, W, generator=g, device=DEV, dtype=BF16)
    if not folizen:                              # routers read the last channels, which only the embedding writes
        code = torch.linspace(-1.6, 1.6, EXPERTS, device=DEV)
        embed[:, -EXPERTS:] = code[torch.rand(VOCAB, EXPERTS, generator=g, device=DEV).argsort(1)].to(BF16)
    yield "embed", embed
    yield "head", leaning_head(g, embed)
    yield "final.norm", vector(g, W, mean=1.0)
    if folizen:
        yield "side.embed", torch.randn(VOCAB, SIDE * case["layers"], generator=g, device=DEV, dtype=BF16)

    def added():                                 # weight of a sublayer's normalised output
        t = vector(g, W, 0.03, 0.2)
        if not folizen:
            t[-EXPERTS:] = 0
        return t

    def into():
        t = vector(g, W, mean=1.0)
        t[-EXPERTS:] = 1
        return t
    for i in range(case["layers"]):
        p = "l%d." % i
        if folizen:
            yield p + "norm1", added()
            if i % 2 == 0:
                for n, r in (("q", H * 128), ("k", G * 128), ("v", G * 128)):
                    yield p + "mix." + n, matrix(g, r, W)
                yield p + "mix.q.norm", vector(g, 128, mean=1.4)
                yield p + "mix.k.norm", vector(g, 128, mean=1.4)
                yield p + "mix.temp", vector(g, H, mean=1.0)
                yield p + "mix.o", matrix(g, W, H * 128)
                yield p + "norm2", added()
                yield p + "mlp.up", matrix(g, F, W)
                yield p + "mlp.act", torch.tensor([0.7, -0.4, 0.5, 0.2], device=DEV, dtype=BF16)
                yield p + "mlp.down", matrix(g, W, F)
            else:
                for n in "rkvga":
                    yield p + "mix." + n, matrix(g, W, W, 0.35 if n == "k" else 1.0)
                yield p + "mix.w1", matrix(g, RANK, W)
                yield p + "mix.w2", matrix(g, W, RANK)
                for n in ("a.b", "w0"):
                    yield p + "mix." + n, vector(g, W, 0.3)
                yield p + "mix.norm", vector(g, W, mean=1.0)
                yield p + "mix.o", matrix(g, W, W)
            yield p + "side.gate", matrix(g, SIDE, W)
            yield p + "side.proj", matrix(g, W, SIDE)
            yield p + "side.norm", added()
            continue
        yield p + "norm1", into()
        yield p + "norm1b", added()
        if i % 2 == 0:
            for n, r, k in (("dq", 3 * W // 8, W), ("uq", H * (128 + ROT), 3 * W // 8), ("dkv", KV_RANK + ROT, W), ("uk", H * 128, KV_RANK),
                            ("uv", H * 128, KV_RANK), ("g", H * 128, W), ("o", W, H * 128)):
                yield p + "mix." + n, matrix(g, r, k, 1.4 if n in ("uq", "uk") else 1.0)
            yield p + "mix.dq.norm", vector(g, 3 * W // 8, mean=1.0)
            yield p + "mix.dkv.norm", vector(g, KV_RANK, mean=1.0)
            yield p + "mix.sink", vector(g, H, 0.5)
        else:
            for n, r in (("q", H * 128), ("k", G * 128), ("v", G * 128)):
                yield p + "mix." + n, matrix(g, r, W)
                yield p + "mix." + n + ".b", vector(g, r)
            yield p + "mix.o", matrix(g, W, H * 128)
        yield p + "norm2", into()
        yield p + "norm2b", added()
        router = torch.zeros(EXPERTS, W, device=DEV, dtype=BF16)
        place = torch.rand(EXPERTS, generator=g, device=DEV).argsort()
        router[torch.arange(EXPERTS, device=DEV), W - EXPERTS + place] = 1.0
        yield p + "mlp.router", router
        for e in range(EXPERTS):
            for n in ("gate", "up"):
                yield p + "mlp.e%d.%s" % (e, n), matrix(g, F // TOP, W)
            yield p + "mlp.e%d.down" % e, matrix(g, W, F // TOP)


def layered_lengths(case):
    """Contexts of the live requests: from a short one to `prompt` tokens, evenly."""
    return [max(1, case["prompt"] * (i + 1) // case["live"]) for i in range(case["live"])]


def layered_inputs(case, seed):
    g = generator(seed, 1)
    if not case["live"]:
        return [ids(g, case["prompt"], VOCAB)], None
    return [ids(g, n + 1, VOCAB) for n in layered_lengths(case)], ids(g, case["portion"] * case["tokens"], VOCAB)


class Layered:
    def __init__(self, case, seed):
        W, (H, G, F) = case["width"], LAYERED[case["width"]]
        folizen, k = case["design"] == "Folizen", case["tokens"]
        layers = (DecoderLayer * case["layers"])()
        for i, l in enumerate(layers):
            l.heads, l.dim, l.vdim, l.window, l.scale = H, 128, 128, case["window"], 128 ** -0.5
            if folizen and i % 2 == 0:
                l.mixer, l.kv_heads, l.distance_bias, l.head_temp, l.ff = 0, G, 1, 1, F
            elif folizen:
                l.mixer, l.heads, l.dim, l.vdim, l.window, l.scale, l.decay_rank = 1, W // 64, 64, 0, 0, 0.0, RANK
            else:
                l.rot_base, l.experts, l.expert_ff, l.expert_top, l.expert_groups, l.expert_groups_kept = 1e5, EXPERTS, F // TOP, TOP, GROUPS, GROUPS_KEPT
                if i % 2 == 0:
                    l.mixer, l.q_rank, l.kv_rank, l.sink, l.out_gate, l.rot_kind, l.rot_dims, l.scale = 2, 3 * W // 8, KV_RANK, 1, 1, 2, ROT, (128 + ROT) ** -0.5
                else:
                    l.mixer, l.kv_heads, l.keep_first, l.qk_norm, l.qkv_bias, l.rot_kind, l.rot_dims = 0, G, KEEP, 1, 1, 1, 128
        self.case, self.folizen = case, folizen
        self.prompts, self.other = layered_inputs(case, seed)
        room = [len(p) + k for p in self.prompts] + ([len(self.other) + 1] if case["live"] else [])
        pages = [(n + 63) // 64 for n in room]
        n_states = 2 * len(room) if folizen else 0
        desc = DecoderDesc(struct_size=C.sizeof(DecoderDesc), num_layers=len(layers), vocab=VOCAB, width=W, side_dim=SIDE if folizen else 0, norm_eps=1e-5,
                           compute_dtype=EFM_BF16, max_step_tokens=2048, max_response_tokens=max(k, 1), cache_pages=sum(pages), state_slots=n_states,
                           max_slots=len(room), norm_layout=0 if folizen else 1, embed_scale=1.0, logit_scale=1.0)
        self.ctx = c = Handle("efm_b200_decoder_create", C.byref(desc), layers, 0)
        for name, t in layered_weights(case, seed):
            c.weight(name, t)
        c("finalize_weights")
        first = 0
        for s, n in enumerate(pages):
            c("decoder_map_slot", s, at(i32(range(first, first + n))), n, s if folizen else -1)
            first += n
        c("set_sampling", C.byref(Sampling(0.0, 1.0, 0, 0, 0)))
        if case["live"]:
            for s, p in enumerate(self.prompts):                 # what the requests hold before these steps
                self.step([(s, p[:-1], 0, False)], None, None)
                c("decoder_pin_prefix", s, len(room) + s if folizen else -1)
            self.logits = np.empty((case["live"], VOCAB), np.float32)
            self.sampled = np.empty((k, case["live"]), np.int32)
        else:
            c("set_prefill_graph", 1)
            c("capture_decode", 0)
            self.logits = torch.empty(VOCAB, dtype=torch.float32, pin_memory=True)
            self.tokens = np.empty(k, np.int32)
        c("synchronize")

    def step(self, entries, logits, sampled):
        """entries: (slot, tokens, position of the first, whether the last one's logits are wanted)."""
        batch, held = (StepEntry * len(entries))(), []
        for e, (slot, tokens, offset, wanted) in zip(batch, entries):
            last = i32([len(tokens) - 1])
            held.append((tokens, last))
            e.slot, e.n_tokens, e.kv_offset, e.n_want, e.tokens, e.want = slot, len(tokens), offset, int(wanted), at(tokens), at(last)
        self.ctx("decoder_step", batch, len(entries), at(logits), at(sampled))

    def run(self):
        case, c, k = self.case, self.ctx, self.case["tokens"]
        if not case["live"]:
            n = len(self.prompts[0])
            c("prefill", 0, at(self.prompts[0]), n, 0, None, 0, -1, HOST, None, 1)
            if k > 1:
                c("decode_begin", 0, n, None, 1)
                c("decode_steps", k - 1, 1)
            c("read_tokens", at(self.tokens), 0, k)
            c("read_logits", at(self.logits), VOCAB)
            return {"tokens": self.tokens, "logits": self.logits}
        now = [p[-1:] for p in self.prompts]
        for t in range(k):
            entries = [(s, now[s], len(p) - 1 + t, True) for s, p in enumerate(self.prompts)]
            if case["portion"]:
                m = case["portion"]
                entries.append((case["live"], self.other[t * m:(t + 1) * m], t * m, False))
            self.step(entries, self.logits if t == k - 1 else None, self.sampled[t])
            now = [self.sampled[t, s:s + 1] for s in range(case["live"])]
        return {"tokens": self.sampled, "logits": self.logits}


def delta_rule(r, k, v, w, a):
    """r, k, v, w, a [T, H, D]: S = diag(w) S - (a u)(u^T S) + k v^T with u = k / |k|, o = S^T r."""
    S = torch.zeros(r.shape[1], r.shape[2], r.shape[2], dtype=r.dtype, device=DEV)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au, out = a * u, torch.empty_like(v)
    for t in range(r.shape[0]):
        S = torch.baddbmm(w[t][:, :, None] * S, torch.stack([k[t], -au[t]], 2), torch.stack([v[t], (u[t][:, None] @ S)[:, 0]], 1))
        out[t] = (r[t][:, None] @ S)[:, 0]
    return out


def layered_forward(case, w, tokens):
    """Logits of the places behind the last `case["tokens"]` tokens."""
    W, (H, G, F), T = case["width"], LAYERED[case["width"]], len(tokens)
    tokens = torch.tensor(np.asarray(tokens, np.int64), device=DEV)
    x = w["embed"][tokens].double()
    pos = torch.arange(T, device=DEV)
    for i in range(case["layers"]):
        p = "l%d." % i

        def get(name):
            return w[p + name]

        def added(y, name):
            return rms(y, get(name), 1e-5)
        if case["design"] == "Folizen":
            if i % 2 == 0:
                q = rms(lin(x, get("mix.q")).view(T, H, 128), get("mix.q.norm"), 1e-5) * get("mix.temp").double()[None, :, None]
                k = rms(lin(x, get("mix.k")).view(T, G, 128), get("mix.k.norm"), 1e-5)
                v = lin(x, get("mix.v")).view(T, G, 128)
                see, far = causal(T, case["window"]), (pos[:, None] - pos[None]).double()
                y = []
                for h in range(H):
                    s = q[:, h] @ k[:, h * G // H].T * 128 ** -0.5 - 2.0 ** (-8.0 * (h + 1) / H) * far
                    y.append(torch.softmax(s.masked_fill(~see, float("-inf")), -1) @ v[:, h * G // H])
                x = x + added(lin(torch.stack(y, 1).reshape(T, -1), get("mix.o")), "norm1")
                z, c = lin(x, get("mlp.up")), get("mlp.act").double()
                z = c[0] * rms(z, None, 1e-5) + c[1] * rms(z ** 2, None, 1e-5) + c[2] * rms(z ** 3, None, 1e-5) + c[3]
                x = x + added(lin(z, get("mlp.down")), "norm2")
            else:
                r, k, v = (lin(x, get("mix." + n)).view(T, -1, 64) for n in "rkv")
                z = lin(torch.tanh(lin(x, get("mix.w1"))), get("mix.w2"), get("mix.w0"))
                decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(z)).view(T, -1, 64)
                a = torch.sigmoid(lin(x, get("mix.a"), get("mix.a.b"))).view(T, -1, 64)
                o = rms(delta_rule(r, k, v, decay, a), None, 1e-5).reshape(T, W) * get("mix.norm").double()
                x = x + added(lin(o * torch.sigmoid(lin(x, get("mix.g"))), get("mix.o")), "norm1")
            e = w["side.embed"][tokens][:, i * SIDE:(i + 1) * SIDE].double()
            z = torch.nn.functional.gelu(lin(x, get("side.gate")), approximate="tanh") * e
            x = x + added(lin(z, get("side.proj")), "side.norm")
            continue
        h = rms(x, get("norm1"), 1e-5)
        if i % 2 == 0:
            a = angles(pos, ROT, 1e5)
            q = lin(rms(lin(h, get("mix.dq")), get("mix.dq.norm"), 1e-5), get("mix.uq")).view(T, H, 128 + ROT)
            down = lin(h, get("mix.dkv"))
            c = rms(down[:, :KV_RANK], get("mix.dkv.norm"), 1e-5)
            kr = turn(down[:, None, KV_RANK:], a, True).expand(T, H, ROT)
            k = torch.cat([lin(c, get("mix.uk")).view(T, H, 128), kr], -1)
            q = torch.cat([q[..., :128], turn(q[..., 128:], a, True)], -1)
            y = attend(q, k, lin(c, get("mix.uv")).view(T, H, 128), (128 + ROT) ** -0.5, causal(T, case["window"]), get("mix.sink"))
            y = y * torch.sigmoid(lin(h, get("mix.g")))
        else:
            a = angles(pos, 128, 1e5)
            q, k = (rms(turn(lin(h, get("mix." + n), get("mix.%s.b" % n)).view(T, -1, 128), a), None, 1e-5) for n in "qk")
            v = lin(h, get("mix.v"), get("mix.v.b")).view(T, G, 128)
            y = attend(q, k, v, 128 ** -0.5, causal(T, case["window"], KEEP))
        x = x + added(lin(y, get("mix.o")), "norm1b")
        h = rms(x, get("norm2"), 1e-5)
        s = torch.softmax(lin(h, get("mlp.router")), -1)
        best = s.view(T, GROUPS, -1).amax(-1)
        shut = best < best.topk(GROUPS_KEPT, -1).values[:, -1:]
        chosen = s.masked_fill(shut.repeat_interleave(EXPERTS // GROUPS, 1), -1).topk(TOP, -1).indices
        y = torch.zeros_like(x)
        for e in range(EXPERTS):
            rows = (chosen == e).any(1).nonzero()[:, 0]
            z = lin(h[rows], get("mlp.e%d.gate" % e))
            y[rows] += s[rows, e, None] * lin(z * torch.sigmoid(z) * lin(h[rows], get("mlp.e%d.up" % e)), get("mlp.e%d.down" % e))
        x = x + added(y, "norm2b")
    return lin(rms(x[-case["tokens"]:], w["final.norm"], 1e-5), w["head"])


def layered_exact(case, seed):
    w, k = dict(layered_weights(case, seed)), case["tokens"]
    tokens, logits = [], []
    for p in layered_inputs(case, seed)[0]:
        chain = [int(p[-1])]
        while len(chain) < k:
            chain.append(successor(chain[-1], VOCAB))
        z = layered_forward(case, w, np.concatenate([p, chain[1:]]))
        tokens.append(z.argmax(1).int().cpu())
        logits.append(z[-1].cpu())
    if not case["live"]:
        return {"tokens": tokens[0].numpy(), "logits": logits[0]}
    return {"tokens": torch.stack(tokens, 1).contiguous().numpy(), "logits": torch.stack(logits).numpy()}


def layered_work(case):
    W, (H, G, F), L, k = case["width"], LAYERED[case["width"]], case["layers"], case["tokens"]
    att = W * (2 * H + 2 * G) * 128
    if case["design"] == "Folizen":
        kinds = [(att + 2 * W * F + 2 * W * SIDE, 0, G * 256, H * 128), (6 * W * W + 2 * W * RANK + 2 * W * SIDE, 0, 0, 0)]
    else:
        lat = W * (3 * W // 8 + KV_RANK + ROT + 2 * H * 128) + 3 * W // 8 * H * (128 + ROT) + KV_RANK * H * 256
        one = 3 * W * F // TOP
        kinds = [(lat + W * EXPERTS, one, KV_RANK + ROT, H * (256 + ROT) / 2), (att + W * EXPERTS, one, G * 256, H * 128)]
    kinds = [kinds[i % 2] for i in range(L)]
    state = 0 if case["design"] != "Folizen" else L // 2 * W * 64 * 4 * 2

    def reads(rows):                             # bytes of the weights that `rows` rows use, each once
        return 2 * (sum(m + min(EXPERTS, rows * TOP) * e for m, e, _, _ in kinds) + W * VOCAB)

    def row(seen):                               # operations of a row that sees so many keys
        seen = min(seen, case["window"])
        return 2 * sum(m + TOP * e + 2 * a * seen for m, e, _, a in kinds) + (14 * L // 2 * W * 64 if state else 0)

    def cache(seen):
        return 2 * sum(c for _, _, c, _ in kinds) * min(seen, case["window"]) + state
    if not case["live"]:
        n = case["prompt"]
        return {"bytes": reads(n) + cache(n) + sum(reads(1) + cache(n + t) for t in range(1, k)),
                "flops": sum(row(i + 1) for i in range(n + k - 1)) + 2 * W * VOCAB * k}
    lengths, m = layered_lengths(case), case["portion"]
    return {"bytes": sum(reads(case["live"] + m) + sum(cache(n + t) for n in lengths) + (cache((t + 1) * m) if m else 0) for t in range(k)),
            "flops": sum(sum(row(n + t) for n in lengths) + sum(row(t * m + i + 1) for i in range(m)) + 2 * W * VOCAB * case["live"] for t in range(k))}


# ---- the cases -------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # a one-line command behind a resident system prompt: time to the first token of the smallest model
        text("first_token_0p5b", model="0.5B", prefix=128, prompt=17),
        # a short answer of the smallest model: every step is latency
        text("generate_0p5b", model="0.5B", prefix=128, prompt=64, tokens=64),
        # a sampled answer behind a longer context
        text("generate_1p5b_top_p", model="1.5B", prefix=512, prompt=256, tokens=64, temperature=0.7, top_p=0.9),
        # a document of odd length, longer than one prefill pass takes
        text("prompt_1p5b_long", model="1.5B", prompt=3001),
        # time to the first token of a large image with INT8 prefill attention
        text("image_prompt_7b", model="VL-7B", rows=26, columns=46, prompt=128, int8=True),
        # a long answer of the largest model: bytes of the weights
        text("generate_7b", model="VL-7B", prompt=333, tokens=32),
        # the same model decoding on INT4 weights
        text("generate_7b_int4", model="VL-7B", prompt=100, tokens=32, int4=True),
        # a 448 x 448 and a 1288 x 728 image through the vision encoder
        encode("encode_448", height=32, width=32, out=2048),
        encode("encode_1288x728", height=52, width=92, out=3584),
        # one control tick of a three-camera robot policy
        act("action_chunk"),
        # one request of a layered decoder with recurrent layers: a long prompt, then tokens on the captured step
        layered("request_delta_rule", design="Folizen", width=2048, prompt=2000, tokens=32),
        # serving a layered decoder with routed experts: sixteen live requests and a prompt in portions
        layered("serve_experts", design="Temuvik", width=2048, prompt=1500, tokens=8, live=16, portion=200),
    ]


def draw(rng):
    def spread(low, high):                       # evenly over the logarithm
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    kind = rng.choice(("text", "text", "text", "encode", "act", "layered"))
    if kind == "text":
        model = rng.choice(tuple(TEXT))
        image = TEXT[model][7] and rng.random() < 0.5
        int4 = rng.random() < 0.25
        sampled = rng.random() < 0.3
        return text(model=model, prefix=0 if image or rng.random() < 0.5 else spread(16, 600), prompt=spread(5, 1000 if model == "VL-7B" else 3000),
                    rows=rng.randint(4, 24) if image else 0, columns=rng.randint(4, 32) if image else 0, tokens=spread(1, 48),
                    temperature=0.7 if sampled else 0.0, top_p=0.9 if sampled else 1.0, int8=rng.random() < 0.3,
                    int4=int4 and model != "0.5B")           # INT4 groups: inputs in multiples of 128
    if kind == "encode":
        return encode(height=2 * rng.randint(4, 26), width=2 * rng.randint(4, 30), images=rng.choice((1, 1, 2)), out=rng.choice((2048, 3584)))
    if kind == "act":
        return act(images=rng.randint(1, 3), size=64 * rng.randint(4, 8), words=rng.randint(8, 64), chunk=rng.randint(10, 50), steps=rng.randint(4, 10))
    live = rng.choice((0, 0, rng.randint(2, 16)))
    return layered(design=rng.choice(("Folizen", "Temuvik")), width=rng.choice(tuple(LAYERED)), layers=2 * rng.randint(1, 4), window=rng.choice((256, 1024)),
                   prompt=spread(20, 2000), tokens=rng.randint(2, 8) if live else spread(2, 32), live=live, portion=rng.choice((0, spread(7, 200))) if live else 0)


KINDS = {"text": (Text, text_exact, text_work), "encode": (Encode, encode_exact, encode_work), "act": (Act, act_exact, act_work),
         "layered": (Layered, layered_exact, layered_work)}


def prepare(case, seed):
    return KINDS[case["kind"]][0](case, seed)


def run(state):
    return state.run()


def exact(case, seed):
    return KINDS[case["kind"]][1](case, seed)


def work(case):
    return KINDS[case["kind"]][2](case)


def tolerance(case):
    """bf16 operands (INT8 scores with int8) through every layer: 0.002 to 0.008 from the 64-bit values at the start of the last layer,
    four times the middle of that between two such computations; tokens are clear and stay."""
    return {"rel": 0.02, "max": 0.3, "differ": 0.0}
