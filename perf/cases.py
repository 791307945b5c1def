"""What is measured: the layers, blocks and calls that training and inference with this framework consist of.

``listed`` names them at the sizes of the framework's own workloads (the PPO, ACT, vision-language-action and world-model
configurations, the language-model head); ``draw`` gives other sizes of the same ranges, odd ones among them.  Each training
case is one forward and backward pass of a layer or block, replayed through ``GraphedStep`` as the trainers replay theirs;
inference cases are launched eagerly under ``no_grad``, as the deployment code does.

Weights and inputs are functions of the seed alone and are exactly representable in bf16, so that the 64-bit results of
``exact`` refer to the numbers the kernels see.
"""
import math
import zlib

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

DEV = "cuda"


# ------------------------------------------------------------------------------------------------ inputs and weights
def _gen(seed, name):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (1 << 62))


def _randn(seed, name, *shape, scale=1.0):
    return (torch.randn(*shape, generator=_gen(seed, name), device=DEV) * scale).to(torch.bfloat16)


def _rand(seed, name, *shape):
    return torch.rand(*shape, generator=_gen(seed, name), device=DEV)


def _weight(seed, name, shape):
    """Value of the parameter ``name`` in the layout that files hold, on the grid of bf16, fp32."""
    leaf = name.rsplit(".", 1)[-1]
    r = torch.randn(*shape, generator=_gen(seed, "w:" + name), device=DEV)
    if leaf == "gamma":
        r = 1.0 + 0.1 * r
    elif leaf in ("bias", "beta"):
        r = 0.1 * r
    elif leaf == "log_std":
        r = 0.1 * r - 0.5
    elif leaf == "queries":
        r = 0.5 * r
    elif len(shape) == 4:                                   # convolution [OC, IC, KH, KW]
        r = r * math.sqrt(2.0 / (shape[1] * shape[2] * shape[3]))
    else:                                                   # dense [IN, OUT], embedding [ROWS, DIM]
        r = r / math.sqrt(shape[0]) if name != "wte.weight" else r * 0.5
    return r.to(torch.bfloat16).float()


def _load(module, seed, prefix=""):
    module.to(DEV)
    for n, p in module.named_params():
        p.load_file_(_weight(seed, prefix + n, tuple(p.file_view().shape)))
    return module


def _grads(params):
    return {n: p.grad for n, p in params}


def _graphed(fn, inputs):
    """A captured step: two eager calls and the capturing one, as in the first three steps of a training run."""
    from noeira_b200.utils.graphs import GraphedStep
    step = GraphedStep(fn, inputs)
    for _ in range(3):
        step(*inputs)
    return step


def _train_state(module, inputs, forward, backward):
    """State of a forward + backward pass of ``module``; gradients are cleared at the start of each pass."""
    from noeira_b200 import nn
    params = list(module.named_params())
    opt = nn.AdamW(params, lr=1e-4)

    def fn(*xs):
        opt.zero_grad()
        y = forward(*xs)
        return y, backward(*xs)

    return {"step": _graphed(fn, inputs), "inputs": inputs, "grads": _grads(params), "opt": opt, "module": module}


def _train_pass(st):
    y, dx = st["step"](*st["inputs"])
    return {"y": y, "dx": dx, "grads": st["grads"]}


class _W64:
    """64-bit leaves of the same weights, made on first use."""

    def __init__(self, seed, prefix=""):
        self.seed, self.prefix, self.leaf = seed, prefix, {}

    def __call__(self, name, *shape):
        if name not in self.leaf:
            self.leaf[name] = _weight(self.seed, self.prefix + name, shape).double().requires_grad_(True)
        return self.leaf[name]

    def grads(self):
        """Gradients in the layout of ``Param.grad`` (convolutions: [KH·KW·IC padded to 8, OC])."""
        out = {}
        for n, w in self.leaf.items():
            g = w.grad
            if g.dim() == 4:
                oc, ic, kh, kw = g.shape
                g = F.pad(g.permute(2, 3, 1, 0), (0, 0, 0, -ic % 8)).reshape(kh * kw * (ic + -ic % 8), oc)
            out[n] = g
        return out


def _linear64(x, W, name, i, o, bias=True):
    y = x @ W(name + ".weight", i, o)
    return y + W(name + ".bias", o) if bias else y


def _norm64(x, W, name, d, eps, rms):
    if rms:
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * W(name + ".gamma", d)
    return F.layer_norm(x, (d,), W(name + ".gamma", d), W(name + ".beta", d), eps)


def _head64(q, k, v, allow, bias):
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if bias is not None:
        s = s + bias
    if allow is not None:
        s = s.masked_fill(~allow, float("-inf"))
    return torch.softmax(s, -1) @ v


def _attention64(q, k, v, allow=None, bias=None):
    """q [B, Sq, H, D], k / v [B, Sk, Hkv, D]: head by head and recomputed in the backward, to fit long sequences."""
    B, Sq, H, _ = q.shape
    rep = H // k.shape[2]
    per = max(1, min(B, int(2e9 // (Sq * k.shape[1] * 8))))
    rows = []
    for b in range(0, B, per):
        heads = [checkpoint(_head64, q[b:b + per, :, h], k[b:b + per, :, h // rep], v[b:b + per, :, h // rep], allow, bias,
                            use_reentrant=False) for h in range(H)]
        rows.append(torch.stack(heads, 2))
    return torch.cat(rows, 0)


def _rope64(x, theta, pos0=0):
    S, D = x.shape[1], x.shape[-1]
    inv = theta ** (-torch.arange(D // 2, dtype=torch.float64, device=x.device) * 2 / D)
    a = (pos0 + torch.arange(S, dtype=torch.float64, device=x.device))[:, None] * inv
    sn, cs = a.sin()[None, :, None], a.cos()[None, :, None]
    x1, x2 = x[..., : D // 2], x[..., D // 2:]
    return torch.cat([x1 * cs - x2 * sn, x2 * cs + x1 * sn], -1)


def _leaf64(x):
    return x.double().requires_grad_(True)


# ------------------------------------------------------------------------------------------------ actor-critic update
# The minibatch step of PPO: forward, data gradients and parameter gradients of the 256-wide actor and critic, one group.
def _policy_inputs(c, seed):
    M = c["rows"]
    x = torch.zeros(M, 64, device=DEV, dtype=torch.bfloat16)      # the environments' observation rows: 128-byte pitch
    x[:, : c["obs"]] = _randn(seed, "obs", M, c["obs"])
    ap = (c["act"] + 7) // 8 * 8
    dmu = torch.zeros(M, ap, device=DEV, dtype=torch.bfloat16)
    dmu[:, : c["act"]] = _randn(seed, "dmu", M, c["act"], scale=1.0 / M)
    dv = torch.zeros(M, 8, device=DEV, dtype=torch.bfloat16)
    dv[:, :1] = _randn(seed, "dv", M, 1, scale=1.0 / M)
    return x, dmu, dv


def _policy_prepare(c, seed):
    from noeira_b200 import nn
    from noeira_b200.agents.ppo import make_actor, make_critic
    from noeira_b200.ops.mlp import Mlp3Pass, mlp3_backward_group, mlp3_forward_group, mlp3_param_grads
    from noeira_b200.ops.streams import Branch
    actor = _load(make_actor(c["obs"], c["act"], 256), seed, "actor.")
    critic = _load(make_critic(c["obs"], 256), seed, "critic.")
    pa, pc = list(actor.named_params("actor.")), list(critic.named_params("critic."))
    opts = [nn.Adam(pa, lr=3e-4), nn.Adam(pc, lr=1e-3)]
    (a1, a2, a3), (c1, c2, c3) = actor.mods, critic.mods
    dev = torch.device(DEV, torch.cuda.current_device())
    passes = [Mlp3Pass(a1, a2, a3.lin, c["rows"], dev), Mlp3Pass(c1, c2, c3, c["rows"], dev)]
    branches = [[Branch(torch.cuda.Stream(), 4 + 3 * i + j) for j in range(3)] for i in range(2)]

    def fn(x, dmu, dv):
        for o in opts:
            o.zero_grad()
        mu, v = mlp3_forward_group(passes, [x, x])
        mlp3_backward_group(passes, [x, x], [dmu, dv])
        mlp3_param_grads(passes[0], x, dmu, branches[0])
        mlp3_param_grads(passes[1], x, dv, branches[1])
        for row in branches:
            for b in row:
                b.join()
        return mu, v

    inputs = _policy_inputs(c, seed)
    grads = {n: p.grad for n, p in pa + pc if not n.endswith("log_std")}
    return {"step": _graphed(fn, inputs), "inputs": inputs, "grads": grads, "keep": (actor, critic, opts)}


def _policy_run(st):
    mu, v = st["step"](*st["inputs"])
    return {"mu": mu, "v": v, "grads": st["grads"]}


def _policy_exact(c, seed):
    x, dmu, dv = _policy_inputs(c, seed)
    W, x = _W64(seed), x[:, : c["obs"]].double()
    outs = {}
    for net, width, dy, key in (("actor.", c["act"], dmu, "mu"), ("critic.", 1, dv, "v")):
        h = torch.tanh(_linear64(x, W, net + "0", c["obs"], 256))
        h = torch.tanh(_linear64(h, W, net + "1", 256, 256))
        y = _linear64(h, W, net + "2", 256, width)
        y.backward(dy[:, :width].double())
        outs[key] = y.detach()
    return {**outs, "grads": W.grads()}


def _policy_work(c):
    M, o, a = c["rows"], c["obs"], c["act"]
    w = 2 * (o * 256 + 256 * 256) + 256 * (a + 1)
    return {"bytes": M * (2 * (o + a + 1) + 4 * (a + 1)) + 6 * w, "flops": 6.0 * M * w - 4.0 * M * o * 256}


# ------------------------------------------------------------------------------------------------ batched physics
# Two control steps of the planar-chain environments from a given state, as a planner's rollout restores and steps them.
def _physics_prepare(c, seed):
    from noeira_b200.envs import PlanarChainEnv
    env = PlanarChainEnv(c["envs"], seed=int(seed) % 65521, model_seed=0)
    env.reset_batch()
    acts = _rand(seed, "act", 42, c["envs"], 6) * 2 - 1
    for t in range(40):                                        # bodies on the ground, joints near their limits
        env.step_batch(acts[t])
    e = env.engine
    saved = [t.clone() for t in (e.qpos, e.qvel, e.warm, e.step_count, e.ep_return)]
    return {"env": env, "saved": saved, "acts": acts[40:].contiguous()}


def _physics_run(st):
    env, e = st["env"], st["env"].engine
    for dst, src in zip((e.qpos, e.qvel, e.warm, e.step_count, e.ep_return), st["saved"]):
        dst.copy_(src)
    for a in st["acts"]:
        obs, reward, done, term = env.step_batch(a, auto_reset=False)
    return {"obs": obs, "reward": reward, "done": done, "qpos": e.qpos, "qvel": e.qvel}


def _physics_exact(c, seed):
    return None                                                # a 64-bit simulation of thousands of environments takes minutes


def _physics_work(c):
    # per environment and step: state, action, observation and multipliers in and out; about 6 k operations per substep for
    # kinematics, mass matrix, bias and factorisation of 9 degrees of freedom, 20 rows x 8 sweeps of the solver
    return {"bytes": 2.0 * c["envs"] * 4 * (2 * 18 + 2 * 48 + 6 + 17 + 5), "flops": 2.0 * c["envs"] * 5 * (6e3 + 20 * 20 * 18 + 8 * 20 * 40)}


# ------------------------------------------------------------------------------------------------ transformer blocks
# Pre-norm blocks: the vision tower and the language prefix of the vision-language-action model in inference, the world
# model's dynamics block and decoder blocks in training.
def _block_make(c):
    from noeira_b200 import nn
    return nn.TransformerBlock(c["dim"], c["heads"], c["ff"], kv_heads=c["kv"], head_dim=c["hd"], norm=c["norm"], ffn=c["ffn"],
                               mask=c["mask"], frame=c["frame"], rope_theta=c["rope"], bias=c["bias"], eps=c["eps"])


def _block_bias(c):
    """The prefix mask: nobody but the last (state) token sees the last token."""
    if not c["prefix"]:
        return None
    m = torch.zeros(c["seq"], c["seq"], device=DEV)
    m[: c["seq"] - 1, c["seq"] - 1] = float("-inf")
    return m


def _block_prepare(c, seed):
    m = _load(_block_make(c), seed)
    x = _randn(seed, "x", c["batch"], c["seq"], c["dim"])
    if c["train"]:
        dy = _randn(seed, "dy", c["batch"], c["seq"], c["dim"], scale=1e-3)
        return _train_state(m, (x, dy), lambda x, dy: m.forward(x), lambda x, dy: m.vjp(dy))
    for p in m.params():
        p.shadow                                               # the bf16 weights that inference reads
    return {"m": m, "x": x, "bias": _block_bias(c)}


def _block_run(st):
    if "step" in st:
        return _train_pass(st)
    with torch.no_grad():
        y = st["m"].forward(st["x"], bias=st["bias"])
        st["m"].release_buffers()
    return y


def _block64(x, W, c):
    B, S, D = x.shape
    H, KV, hd, rms = c["heads"], c["kv"], c["hd"], c["norm"] == "rms"
    qkv = _linear64(_norm64(x, W, "norm1", D, c["eps"], rms), W, "attn.qkv", D, (H + 2 * KV) * hd, c["bias"]).reshape(B, S, H + 2 * KV, hd)
    q, k, v = qkv[:, :, :H], qkv[:, :, H:H + KV], qkv[:, :, H + KV:]
    if c["rope"]:
        q, k = _rope64(q, c["rope"]), _rope64(k, c["rope"])
    i, j = torch.arange(S, device=x.device)[:, None], torch.arange(S, device=x.device)[None]
    allow = None
    if c["mask"]:
        f = c["frame"] if c["mask"] == "block_causal" else 1
        allow = (j // f) <= (i // f)
    o = _attention64(q, k, v, allow, _block_bias(c))
    x = x + _linear64(o.reshape(B, S, H * hd), W, "attn.out", H * hd, D, c["bias"])
    h = _norm64(x, W, "norm2", D, c["eps"], rms)
    if c["ffn"] == "swiglu":
        g, u = _linear64(h, W, "ffn.0", D, 2 * c["ff"], c["bias"]).chunk(2, -1)
        h = F.silu(g) * u
    else:
        h = F.gelu(_linear64(h, W, "ffn.0", D, c["ff"], c["bias"]), approximate="tanh")
    return x + _linear64(h, W, "ffn.1", c["ff"], D, c["bias"])


def _block_exact(c, seed):
    W, x = _W64(seed), _leaf64(_randn(seed, "x", c["batch"], c["seq"], c["dim"]))
    if not c["train"]:
        with torch.no_grad():
            return _block64(x, W, c)
    y = _block64(x, W, c)
    y.backward(_randn(seed, "dy", c["batch"], c["seq"], c["dim"], scale=1e-3).double())
    return {"y": y.detach(), "dx": x.grad, "grads": W.grads()}


def _block_work(c):
    T, D = c["batch"] * c["seq"], c["dim"]
    w = D * (c["heads"] + 2 * c["kv"]) * c["hd"] + c["heads"] * c["hd"] * D + D * c["ff"] * (3 if c["ffn"] == "swiglu" else 2)
    share = 1.0 if not c["mask"] else 0.5 * (1 + (c["frame"] if c["mask"] == "block_causal" else 1) / c["seq"])
    att = 4.0 * T * c["seq"] * c["heads"] * c["hd"] * share
    if c["train"]:
        return {"bytes": 8.0 * T * D + 6.0 * w, "flops": 6.0 * T * w + 3.5 * att}
    return {"bytes": 4.0 * T * D + 2.0 * w, "flops": 2.0 * T * w + att}


_VIT = dict(kind="block", dim=768, heads=12, kv=12, hd=64, ff=3072, norm="layer", ffn="gelu", mask=None, frame=0, rope=None, bias=True,
            eps=1e-6, prefix=False, train=False)
_PREFIX = dict(kind="block", dim=960, heads=15, kv=5, hd=64, ff=2560, norm="rms", ffn="swiglu", mask=None, frame=0, rope=1e5, bias=False,
               eps=1e-5, prefix=True, train=False)
_WORLD = dict(kind="block", dim=2048, heads=16, kv=4, hd=128, ff=5632, norm="rms", ffn="swiglu", mask="block_causal", frame=257, rope=None,
              bias=False, eps=1e-5, prefix=False, train=True)
_DECODER = dict(kind="block", dim=384, heads=6, kv=6, hd=64, ff=1536, norm="layer", ffn="gelu", mask="causal", frame=0, rope=None, bias=True,
                eps=1e-5, prefix=False, train=True)


# ------------------------------------------------------------------------------------------------ action expert layer
# One layer of the action expert: a chunk of action tokens over the cached prefix keys and values (self: prefix and
# causal suffix; cross: prefix only), forward and backward in fine-tuning.
def _expert_inputs(c, seed):
    x = _randn(seed, "x", c["batch"], c["chunk"], 720)
    pk, pv = (_randn(seed, n, c["batch"], c["prefix"], 5, 64) for n in ("pk", "pv"))
    return x, pk, pv, _randn(seed, "dy", c["batch"], c["chunk"], 720, scale=1e-3)


def _expert_prepare(c, seed):
    from noeira_b200.models.vla import ExpertLayer, VLAConfig
    m = _load(ExpertLayer(VLAConfig(), cross=c["cross"]), seed)
    P = c["prefix"]
    return _train_state(m, _expert_inputs(c, seed), lambda x, pk, pv, dy: m.forward(x, pk, pv, P), lambda x, pk, pv, dy: m.vjp(dy))


def _expert_exact(c, seed):
    x, pk, pv, dy = (t.double() for t in _expert_inputs(c, seed))
    x.requires_grad_(True)
    W, (B, S, D), P = _W64(seed), x.shape, c["prefix"]
    h = _norm64(x, W, "input_layernorm", D, 1e-5, True)
    q = _rope64(_linear64(h, W, "self_attn.q_proj", D, 960, False).reshape(B, S, 15, 64), 1e5, P)
    if c["cross"]:
        k = _linear64(pk.reshape(B, P, 320), W, "self_attn.k_proj", 320, 320, False).reshape(B, P, 5, 64)
        v = _linear64(pv.reshape(B, P, 320), W, "self_attn.v_proj", 320, 320, False).reshape(B, P, 5, 64)
        allow = None
    else:
        k = torch.cat([pk, _rope64(_linear64(h, W, "self_attn.k_proj", D, 320, False).reshape(B, S, 5, 64), 1e5, P)], 1)
        v = torch.cat([pv, _linear64(h, W, "self_attn.v_proj", D, 320, False).reshape(B, S, 5, 64)], 1)
        allow = torch.arange(P + S, device=x.device)[None] <= torch.arange(S, device=x.device)[:, None] + P
    o = _attention64(q, k, v, allow)
    r = x + _linear64(o.reshape(B, S, 960), W, "self_attn.o_proj", 960, D, False)
    g, u = _linear64(_norm64(r, W, "post_attention_layernorm", D, 1e-5, True), W, "mlp.0", D, 4096, False).chunk(2, -1)
    y = r + _linear64(F.silu(g) * u, W, "mlp.1", 2048, D, False)
    y.backward(dy)
    return {"y": y.detach(), "dx": x.grad, "grads": W.grads()}


def _expert_work(c):
    T, B, P = c["batch"] * c["chunk"], c["batch"], c["prefix"]
    w = 720 * 960 * 2 + 720 * 2048 * 3
    kv = (2.0 * 6 / 3 * B * P * 2 * 320 * 320) if c["cross"] else 6.0 * T * 2 * 720 * 320
    n = w + 2 * 320 * (320 if c["cross"] else 720)
    att = 4.0 * T * (P if c["cross"] else P + c["chunk"] / 2) * 960
    return {"bytes": 8.0 * T * 720 + 4.0 * B * P * 320 + 6.0 * n, "flops": 6.0 * T * w + kv + 3.5 * att}


# ------------------------------------------------------------------------------------------------ DETR encoder layer
# A post-norm encoder layer of ACT over the camera tokens of a batch, positions added to queries and keys.
def _detr_inputs(c, seed):
    D = c["dim"]
    return (_randn(seed, "x", c["batch"], c["tokens"], D), _randn(seed, "pos", 1, c["tokens"], D, scale=0.5),
            _randn(seed, "dy", c["batch"], c["tokens"], D, scale=1e-3))


def _detr_prepare(c, seed):
    from noeira_b200.models.act import DETREncoderLayer
    m = _load(DETREncoderLayer(c["dim"], c["heads"], c["ff"], p=0.0), seed)
    st = _train_state(m, _detr_inputs(c, seed), lambda x, pos, dy: m.forward(x, pos), lambda x, pos, dy: m.vjp(dy))
    del st["grads"]["attn.k.bias"]                             # softmax ignores it: zero, and rounding on top
    return st


def _mha64(W, name, xq, xk, xv, D, H):
    B, Sq, Sk = xq.shape[0], xq.shape[1], xk.shape[1]
    q = _linear64(xq, W, name + ".q", D, D).reshape(B, Sq, H, D // H)
    k = _linear64(xk, W, name + ".k", D, D).reshape(B, Sk, H, D // H)
    v = _linear64(xv, W, name + ".v", D, D).reshape(B, Sk, H, D // H)
    return _linear64(_attention64(q, k, v).reshape(B, Sq, D), W, name + ".o", D, D)


def _ffn64(W, name, x, D, ff):
    return _linear64(torch.relu(_linear64(x, W, name + ".f1", D, ff)), W, name + ".f2", ff, D)


def _encoder64(W, pre, x, pos, D, H, ff):
    xp = x + pos
    n1 = _norm64(x + _mha64(W, pre + "attn", xp, xp, x, D, H), W, pre + "n1", D, 1e-5, False)
    return _norm64(n1 + _ffn64(W, pre + "ffn", n1, D, ff), W, pre + "out", D, 1e-5, False)


def _detr_exact(c, seed):
    x, pos, dy = (t.double() for t in _detr_inputs(c, seed))
    x = x.requires_grad_(True)
    pos = pos.expand(c["batch"], -1, -1).contiguous().requires_grad_(True)
    W = _W64(seed)
    y = _encoder64(W, "", x, pos, c["dim"], c["heads"], c["ff"])
    y.backward(dy)
    grads = W.grads()
    del grads["attn.k.bias"]
    return {"y": y.detach(), "dx": [x.grad, pos.grad], "grads": grads}


def _detr_work(c):
    T, D = c["batch"] * c["tokens"], c["dim"]
    w = 4 * D * D + 2 * D * c["ff"]
    return {"bytes": 8.0 * T * D + 6.0 * w, "flops": 6.0 * T * w + 3.5 * 4.0 * T * c["tokens"] * D}


# ------------------------------------------------------------------------------------------------ ResNet block
# A residual block of the ACT backbone: two 3x3 convolutions with batch statistics, ReLU and the shortcut.
def _conv64(x, W, name, oc, ic, k, stride, pad):
    return F.conv2d(x, W(name + ".weight", oc, ic, k, k), None, stride, pad)


def _bn64(x, W, name, c, training=True):
    g, b = W(name + ".gamma", c).view(1, c, 1, 1), W(name + ".beta", c).view(1, c, 1, 1)
    mean, var = (x.mean((0, 2, 3), keepdim=True), x.var((0, 2, 3), unbiased=False, keepdim=True)) if training else (0.0, torch.ones_like(g))
    return (x - mean) * torch.rsqrt(var + 1e-5) * g + b


def _resblock64(x, W, pre, ic, oc, stride, training=True):
    idt = x
    if stride != 1 or ic != oc:
        idt = _bn64(_conv64(x, W, pre + "downsample.0", oc, ic, 1, stride, 0), W, pre + "downsample.1", oc, training)
    h = torch.relu(_bn64(_conv64(x, W, pre + "conv1", oc, ic, 3, stride, 1), W, pre + "bn1", oc, training))
    return torch.relu(_bn64(_conv64(h, W, pre + "conv2", oc, oc, 3, 1, 1), W, pre + "bn2", oc, training) + idt)


def _res_inputs(c, seed):
    s = c["stride"]
    oh, ow = (c["h"] - 1) // s + 1, (c["w"] - 1) // s + 1
    x = torch.relu(_randn(seed, "x", c["images"], c["h"], c["w"], c["ic"]))          # what a ReLU in front leaves
    # gradients of about one magnitude, as an L1 loss has them: a ReLU that another rounding opens or shuts then moves an element
    # of dx by less than the spread of dx
    u = _rand(seed, "dy", c["images"], oh, ow, c["oc"]) - 0.5
    return x, ((0.8 + 0.4 * u.abs()) * u.sign() * 1e-3).to(torch.bfloat16)


def _res_prepare(c, seed):
    from noeira_b200 import nn
    m = _load(nn.BasicBlock(c["ic"], c["oc"], c["stride"]), seed)
    st = _train_state(m, _res_inputs(c, seed), lambda x, dy: m.forward(x), lambda x, dy: m.vjp(dy))
    return {**st, "stats": {n: s.data for n, s in m.named_states()}}


def _res_run(st):
    return {**_train_pass(st), "stats": st["stats"]}


def _res_exact(c, seed):
    x, dy = _res_inputs(c, seed)
    x, W = _leaf64(x), _W64(seed)
    y = _resblock64(x.permute(0, 3, 1, 2), W, "", c["ic"], c["oc"], c["stride"]).permute(0, 2, 3, 1)
    y.backward(dy.double())
    return {"y": y.detach(), "dx": x.grad, "grads": W.grads(), "stats": None}


def _res_work(c):
    s = c["stride"]
    pix_in, pix = c["images"] * c["h"] * c["w"], c["images"] * ((c["h"] - 1) // s + 1) * ((c["w"] - 1) // s + 1)
    w = 9 * c["ic"] * c["oc"] + 9 * c["oc"] ** 2 + (c["ic"] * c["oc"] if (s != 1 or c["ic"] != c["oc"]) else 0)
    return {"bytes": 4.0 * pix_in * c["ic"] + 4.0 * pix * c["oc"] + 6.0 * w, "flops": 6.0 * pix * w}


# ------------------------------------------------------------------------------------------------ ResNet stem
# Camera frames to features: normalisation of the bytes, 7x7 / 2 convolution, batch norm, ReLU, 3x3 / 2 max pooling.
def _stem_inputs(c, seed):
    img = torch.randint(0, 256, (c["images"], 3, c["h"], c["w"]), dtype=torch.uint8, generator=_gen(seed, "img"), device=DEV)
    half = lambda n: (n - 1) // 2 + 1
    return img, _randn(seed, "dy", c["images"], half(half(c["h"])), half(half(c["w"])), 64, scale=1e-3)


def _stem_prepare(c, seed):
    from noeira_b200 import nn

    class Stem(nn.Module):
        def __init__(self):
            super().__init__()
            self.conv1 = self.add_child("conv1", nn.Conv2D(3, 64, 7, 2, 3, bias=False, need_input_grad=False))
            self.bn1 = self.add_child("bn1", nn.BatchNorm2D(64, relu=True))
            self.pool = nn.MaxPool2D(3, 2, 1)

        def forward(self, img):
            return self.pool.forward(self.bn1.forward(self.conv1.forward(nn.normalize_images(img))))

        def vjp(self, dy):
            return self.conv1.vjp(self.bn1.vjp(self.pool.vjp(dy)))

    m = _load(Stem(), seed)
    st = _train_state(m, _stem_inputs(c, seed), lambda img, dy: m.forward(img), lambda img, dy: m.vjp(dy))
    return {**st, "stats": {n: s.data for n, s in m.named_states()}}


def _images64(img):
    mean, std = (torch.tensor(v, dtype=torch.float64, device=DEV).view(1, 3, 1, 1) for v in ((0.485, 0.456, 0.406), (0.229, 0.224, 0.225)))
    return (img.double() / 255 - mean) / std


def _stem_exact(c, seed):
    img, dy = _stem_inputs(c, seed)
    W = _W64(seed)
    h = torch.relu(_bn64(_conv64(_images64(img), W, "conv1", 64, 3, 7, 2, 3), W, "bn1", 64))
    y = F.max_pool2d(h, 3, 2, 1).permute(0, 2, 3, 1)
    y.backward(dy.double())
    return {"y": y.detach(), "dx": None, "grads": W.grads(), "stats": None}


def _stem_work(c):
    pix = c["images"] * ((c["h"] - 1) // 2 + 1) * ((c["w"] - 1) // 2 + 1)
    return {"bytes": 3.0 * c["images"] * c["h"] * c["w"] + 4.0 * pix / 4 * 64 + 6.0 * 147 * 64, "flops": 4.0 * pix * 147 * 64}


# ------------------------------------------------------------------------------------------------ optimizer step
# AdamW over all parameters of a model, with or without clipping by the global gradient norm.
def _adamw_values(c, seed):
    n, d = c["layers"], c["dim"]
    for i in range(n):
        for leaf, shape in ((f"{i}.weight", (d, 4 * d)), (f"{i}.bias", (4 * d,))):
            g = torch.randn(*shape, generator=_gen(seed, "g" + leaf), device=DEV) * 1e-2
            m = torch.randn(*shape, generator=_gen(seed, "m" + leaf), device=DEV) * 1e-2
            v = torch.rand(*shape, generator=_gen(seed, "v" + leaf), device=DEV) * 1e-4
            yield leaf, _weight(seed, leaf, shape), g, m, v


def _adamw_prepare(c, seed):
    from noeira_b200 import nn
    m = nn.Sequential(*[nn.Linear(c["dim"], 4 * c["dim"], init=nn.Zero()) for _ in range(c["layers"])]).to(DEV)
    ps = dict(m.named_params())
    opt = nn.AdamW(ps.items(), lr=1e-4, weight_decay=1e-2)
    opt.max_grad_norm = c["clip"]
    opt.load_scalars({"t": 10.0, "b1t": 0.9 ** 10, "b2t": 0.999 ** 10})
    for n, w, g, mm, vv in _adamw_values(c, seed):
        ps[n].set_(w)
        ps[n].grad.copy_(g)
        ps[n].m.copy_(mm)
        ps[n].v.copy_(vv)
    opt.arena.refresh_shadow()
    return {"opt": opt, "module": m}


def _adamw_run(st):
    opt = st["opt"]
    if opt.max_grad_norm > 0:
        opt.clip()
    opt.step()
    a = opt.arena
    return {"val": a.val, "m": a.m, "v": a.v, "shadow": a.shadow}


def _adamw_exact(c, seed):
    vals = [(n, w.double(), g.double(), m.double(), v.double()) for n, w, g, m, v in _adamw_values(c, seed)]
    scale = 1.0
    if c["clip"] > 0:
        norm = math.sqrt(sum(float(g.pow(2).sum()) for _, _, g, _, _ in vals))
        scale = c["clip"] / (norm + 1e-6) if norm > c["clip"] else 1.0
    val, ms, vs = [], [], []
    for n, w, g, m, v in vals:
        g = g * scale
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        if n.endswith("weight"):
            w = w * (1 - 1e-4 * 1e-2)
        w = w - 1e-4 * (m / (1 - 0.9 ** 11)) / ((v / (1 - 0.999 ** 11)).sqrt() + 1e-8)
        val, ms, vs = val + [w.reshape(-1)], ms + [m.reshape(-1)], vs + [v.reshape(-1)]
    val = torch.cat(val)
    return {"val": val, "m": torch.cat(ms), "v": torch.cat(vs), "shadow": val}


def _adamw_work(c):
    n = c["layers"] * (4 * c["dim"] ** 2 + 4 * c["dim"])
    return {"bytes": 30.0 * n + (4.0 * n if c["clip"] else 0.0), "flops": 15.0 * n}


# ------------------------------------------------------------------------------------------------ token embedding and head
# The vocabulary ends of a language model: embedding, final norm, output projection, cross-entropy, and back.
def _head_inputs(c, seed):
    ids = (c["vocab"] * _rand(seed, "ids", c["rows"]) ** 3).long().clamp_(max=c["vocab"] - 1)       # frequent and rare tokens
    tgt = (c["vocab"] * _rand(seed, "tgt", c["rows"]) ** 3).long().clamp_(max=c["vocab"] - 1)
    return ids, tgt


def _head_prepare(c, seed):
    from noeira_b200 import nn

    class Ends(nn.Module):
        def __init__(self):
            super().__init__()
            self.wte = self.add_child("wte", nn.Embedding(c["vocab"], c["dim"]))
            self.ln = self.add_child("ln_f", nn.LayerNorm(c["dim"]))
            self.head = self.add_child("head", nn.Linear(c["dim"], c["vocab"], bias=False, init=nn.Zero()))
            self.loss = torch.zeros(1, device=DEV)

        def forward(self, ids):
            self.logits = self.head.forward(self.ln.forward(self.wte.forward(ids)))
            return self.logits

        def vjp(self, tgt):
            self.loss.zero_()
            d = nn.cross_entropy(self.logits, tgt, self.loss)
            dh = self.ln.vjp(self.head.vjp(d))
            self.wte.vjp(dh)
            return dh

    m = _load(Ends(), seed)
    st = _train_state(m, _head_inputs(c, seed), lambda ids, tgt: m.forward(ids), lambda ids, tgt: m.vjp(tgt))
    return {**st, "loss": m.loss}


def _head_run(st):
    dlogits, dh = st["step"](*st["inputs"])                      # the loss leaves the gradient in the logits' memory
    return {"dlogits": dlogits, "dh": dh, "loss": st["loss"], "grads": st["grads"]}


def _head_exact(c, seed):
    ids, tgt = _head_inputs(c, seed)
    W = _W64(seed)
    x = W("wte.weight", c["vocab"], c["dim"])[ids]
    x.retain_grad()
    logits = _norm64(x, W, "ln_f", c["dim"], 1e-5, False) @ W("head.weight", c["dim"], c["vocab"])
    logits.retain_grad()
    loss = F.cross_entropy(logits, tgt)
    loss.backward()
    return {"dlogits": logits.grad, "dh": x.grad, "loss": loss.detach().reshape(1), "grads": W.grads()}


def _head_work(c):
    M, D, V = c["rows"], c["dim"], c["vocab"]
    return {"bytes": 16.0 * M + 2.0 * M * V + 4.0 * M * D + 2 * 6.0 * D * V, "flops": 6.0 * M * D * V}


# ------------------------------------------------------------------------------------------------ policy query
# One query of the deployed ACT policy: camera frames and joint state to an action chunk, the whole network.
def _act_cfg(c):
    return dict(height=c["h"], width=c["w"], n_cam=c["cams"], enc_layers=4, dec_layers=7, chunk=c["chunk"])


def _act_inputs(c, seed):
    img = torch.randint(0, 256, (c["batch"], c["cams"], 3, c["h"], c["w"]), dtype=torch.uint8, generator=_gen(seed, "img"), device=DEV)
    return _randn(seed, "qpos", c["batch"], 6).float(), img


def _act_prepare(c, seed):
    from noeira_b200.models.act import ACTConfig, ACTModel
    m = _load(ACTModel(ACTConfig(**_act_cfg(c))), seed)
    m.eval()
    for p in m.params():
        p.shadow
    return {"m": m, "inputs": _act_inputs(c, seed)}


def _act_run(st):
    with torch.no_grad():
        return st["m"].infer(*st["inputs"])


def _sin64(n, d):
    pos, i = torch.arange(n, dtype=torch.float64, device=DEV)[:, None], torch.arange(d, dtype=torch.float64, device=DEV)[None]
    a = pos / 10000.0 ** (2 * torch.div(i, 2, rounding_mode="floor") / d)
    out = torch.zeros(n, d, dtype=torch.float64, device=DEV)
    out[:, 0::2], out[:, 1::2] = a[:, 0::2].sin(), a[:, 1::2].cos()
    return out


def _act_exact(c, seed):
    with torch.no_grad():
        qpos, img = _act_inputs(c, seed)
        W, B, D, H, ff, K = _W64(seed), c["batch"], 512, 8, 3200, c["chunk"]
        h = _images64(img.reshape(B * c["cams"], 3, c["h"], c["w"]))
        h = F.max_pool2d(torch.relu(_bn64(_conv64(h, W, "feat.0.conv1", 64, 3, 7, 2, 3), W, "feat.0.bn1", 64, False)), 3, 2, 1)
        ic = 64
        for li, (oc, s) in enumerate(((64, 1), (128, 2), (256, 2), (512, 2)), 1):
            for bi in range(2):
                h = _resblock64(h, W, f"feat.0.layer{li}.{bi}.", ic, oc, s if bi == 0 else 1, False)
                ic = oc
        oh, ow = h.shape[2:]
        src = _linear64(h.permute(0, 2, 3, 1).reshape(B, c["cams"] * oh * ow, 512), W, "src.0", 512, D)
        lat = W("lattok.bias", D).expand(B, 1, D)
        mem = torch.cat([lat, _linear64(qpos.double(), W, "prop", 6, D)[:, None], src], 1)
        img_pos = torch.cat([_sin64(oh, 256)[:, None].expand(oh, ow, 256), _sin64(ow, 256)[None].expand(oh, ow, 256)], -1)
        pos = torch.cat([W("addpos.queries", 2, D), img_pos.reshape(oh * ow, D).repeat(c["cams"], 1)], 0)[None]
        for i in range(4):
            mem = _encoder64(W, f"memory.{i}.", mem, pos, D, H, ff)
        kmem, qpe = mem + pos, W("qpe.queries", K, D)[None]
        x = W("tgt0.queries", K, D).expand(B, K, D)
        for i in range(7):
            p, xq = f"hs.{i}.", x + qpe
            n1 = _norm64(x + _mha64(W, p + "self", xq, xq, x, D, H), W, p + "n1", D, 1e-5, False)
            n2 = _norm64(n1 + _mha64(W, p + "cross", n1 + qpe, kmem, mem, D, H), W, p + "n2", D, 1e-5, False)
            x = _norm64(n2 + _ffn64(W, p + "ffn", n2, D, ff), W, p + "out", D, 1e-5, False)
        return _linear64(_norm64(x, W, "hsn.0", D, 1e-5, False), W, "ahat.0", D, 6)


def _act_work(c):
    B, px = c["batch"], c["batch"] * c["cams"] * c["h"] * c["w"]
    conv = px / 4 * 147 * 64 + px / 16 * 4 * 9 * 64 * 64
    for ic, oc, s in ((64, 128, 64), (128, 256, 256), (256, 512, 1024)):
        conv += px / s * (9 * ic * oc + 3 * 9 * oc * oc + ic * oc)
    tok, K, D, ff = B * (c["cams"] * math.ceil(c["h"] / 32) * math.ceil(c["w"] / 32) + 2), B * c["chunk"], 512, 3200
    lin = tok * (4 * (4 * D * D + 2 * D * ff) + 7 * 2 * D * D + D * D) + K * 7 * (6 * D * D + 2 * D * ff)
    att = 4.0 * tok * tok / B * D * 4 + 7 * 4.0 * K * (tok / B + c["chunk"]) * D
    w = 11.2e6 + 4 * (4 * D * D + 2 * D * ff) + 7 * (8 * D * D + 2 * D * ff)
    return {"bytes": 3.0 * px + 2.0 * w, "flops": 2.0 * (conv + lin) + att}


# ------------------------------------------------------------------------------------------------ the cases
_KINDS = {
    "policy": (_policy_prepare, _policy_run, _policy_exact, _policy_work),
    "physics": (_physics_prepare, _physics_run, _physics_exact, _physics_work),
    "block": (_block_prepare, _block_run, _block_exact, _block_work),
    "expert": (_expert_prepare, _train_pass, _expert_exact, _expert_work),
    "detr": (_detr_prepare, _train_pass, _detr_exact, _detr_work),
    "resblock": (_res_prepare, _res_run, _res_exact, _res_work),
    "stem": (_stem_prepare, _res_run, _stem_exact, _stem_work),
    "adamw": (_adamw_prepare, _adamw_run, _adamw_exact, _adamw_work),
    "head": (_head_prepare, _head_run, _head_exact, _head_work),
    "act": (_act_prepare, _act_run, _act_exact, _act_work),
}

# measured: the error of the path against `exact`, times about four (bf16 chains; ReLU and max selections flip near ties)
_TOLERANCE = {
    "policy": {"rel": 1.5e-2},
    "physics": {"rel": 2e-2, "max": 0.9},
    "block": {"rel": 2e-2},
    "expert": {"rel": 2e-2},
    "detr": {"rel": 3e-2},
    "resblock": {"rel": 3e-2},
    "stem": {"rel": 3e-2},
    "adamw": {"rel": 1e-4, "max": 1e-2},
    "head": {"rel": 1.2e-2},
    "act": {"rel": 3e-2},
}


def listed():
    return [
        # minibatch of the PPO benchmark configuration: 4096 environments x 32 steps / 8
        dict(name="policy_update", kind="policy", rows=16384, obs=17, act=6),
        # its 4096 environments
        dict(name="physics_step", kind="physics", envs=4096),
        # two robots asking their policy for the next chunk: two 480 x 640 cameras each; latency and launches
        dict(name="act_query", kind="act", batch=2, cams=2, h=480, w=640, chunk=100),
        # ACT training at 8 samples per GPU: 2 cameras x 15 x 20 tokens + 2
        dict(name="detr_encoder", kind="detr", batch=8, tokens=602, dim=512, heads=8, ff=3200),
        # the backbone's first stage on the 16 camera frames of that batch
        dict(name="res_block", kind="resblock", images=16, h=120, w=160, ic=64, oc=64, stride=1),
        # and the step into its third stage
        dict(name="res_down", kind="resblock", images=16, h=60, w=80, ic=128, oc=256, stride=2),
        # the frames themselves
        dict(name="res_stem", kind="stem", images=16, h=480, w=640),
        # vision tower of the vision-language-action model on 24 images (three cameras, batch 8)
        dict(name="vit_block", batch=24, seq=1024, **_VIT),
        # its action expert in fine-tuning: 64 samples, chunks of 50 actions, prefix of 241 tokens
        dict(name="expert_layer", kind="expert", batch=64, chunk=50, prefix=241, cross=False),
        # world-model training: 64 frames of 257 tokens
        dict(name="world_block", batch=1, seq=16448, **_WORLD),
        # language-model head over a 49152-token vocabulary
        dict(name="token_head", kind="head", rows=4096, dim=384, vocab=49152),
        # one optimizer step of an 84 M-parameter model (ACT)
        dict(name="adamw_step", kind="adamw", layers=20, dim=1024, clip=0.0),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(sorted(_KINDS) + ["block", "block", "resblock"])
    if kind == "policy":
        return dict(kind=kind, rows=log(1024, 32768), obs=rng.randint(3, 64), act=rng.randint(1, 16))
    if kind == "physics":
        return dict(kind=kind, envs=log(64, 4096))
    if kind == "act":
        return dict(kind=kind, batch=rng.randint(2, 4), cams=rng.randint(1, 2), h=rng.randint(96, 480), w=rng.randint(128, 640),
                    chunk=rng.randint(20, 100))
    if kind == "detr":
        dim = rng.choice((256, 512))
        return dict(kind=kind, batch=rng.randint(1, 8), tokens=log(50, 602), dim=dim, heads=dim // 64,
                    ff=rng.choice((1024, 2048, 3200)))
    if kind == "resblock":
        ic = rng.choice((64, 128, 256, 512))
        down = ic < 512 and rng.random() < 0.4
        side = 160 * 64 // ic
        return dict(kind=kind, images=rng.randint(1, 16), h=rng.randint(max(side // 3, 7), side * 3 // 4), w=rng.randint(max(side // 2, 9), side),
                    ic=ic, oc=2 * ic if down else ic, stride=2 if down else 1)
    if kind == "stem":
        return dict(kind=kind, images=rng.randint(1, 16), h=rng.randint(96, 480), w=rng.randint(128, 640))
    if kind == "expert":
        return dict(kind=kind, batch=log(1, 64), chunk=rng.randint(10, 100), prefix=rng.randint(50, 300), cross=rng.random() < 0.5)
    if kind == "adamw":
        return dict(kind=kind, layers=rng.randint(1, 20), dim=rng.choice((64, 256, 720, 960, 1024)), clip=rng.choice((0.0, 1.0)))
    if kind == "head":
        return dict(kind=kind, rows=log(256, 4096), dim=rng.choice((192, 384, 512, 960)), vocab=rng.choice((512, 8192, 32000, 49152)))
    form = rng.choice(("vit", "prefix", "world", "decoder"))
    if form == "vit":
        return dict(batch=rng.randint(1, 24), seq=rng.choice((196, 256, 577, 1024)), **_VIT)
    if form == "prefix":
        return dict(batch=log(1, 64), seq=rng.randint(100, 300), **_PREFIX)
    if form == "world":
        return dict(batch=1, seq=257 * rng.randint(2, 40), **_WORLD)
    return dict(batch=rng.randint(1, 32), seq=rng.randint(64, 1024), **_DECODER)


def prepare(case, seed):
    return {"kind": case["kind"], "state": _KINDS[case["kind"]][0](case, seed)}


def run(state):
    return _KINDS[state["kind"]][1](state["state"])


def exact(case, seed):
    return _KINDS[case["kind"]][2](case, seed)


def work(case):
    return _KINDS[case["kind"]][3](case)


def tolerance(case):
    return dict(_TOLERANCE[case["kind"]])
