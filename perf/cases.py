"""Workloads of this framework, each driven through the public entry points as a user's program drives them.

Six kinds of program, over the range of sizes they are used at:

lm        a training step of the LSTM language model (`LstmLm`): dropout masks drawn on the device, token ids handed over in
          pinned host memory, forward + backward, and either the clipped SGD update ("update") or, as a data-parallel rank or a
          program with a trainer of its own does it, gradients into a cleared buffer ("grads").
layer     one LSTM layer over a whole sequence, forward and backward, through the sequence entry points of `Context`.
generate  text generation with a 2-layer LSTM language model: the prompt through the sequence entry point (prefill), then one
          token after another: lookup, fused LSTM steps, output projection, log-softmax (decode).
output    embedding lookup -> linear projection to the vocabulary -> PickNegLogSoftmax, backward through all of it, and the
          scatter-add into the embedding gradient.
nodes     the elementwise, softmax and normalisation nodes one by one, forward and backward, on Dim({D}, N) tensors.
tagger    a pass of the autobatched BiLSTM tagger (`Tagger`) over a mini-batch of ragged sentences, with the update or with
          gradients into a cleared buffer.

All values are float32, the only type of these entry points; ids are uint32.
"""
import ctypes as C
import math

import numpy as np
import torch

from dynet_b200 import capi, lm, tagger

KEEP = 0.8          # dropout 0.2, the rate of the language-model configuration


def listed():
    return [
        # a small language model (word-level text of one author, a test run): the step is a few hundred microseconds, launches count
        dict(name="lm small B16", kind="lm", V=2000, E=128, H=256, L=1, T=20, B=16, dropout=True, out="update"),
        # sizes that fit no tile, no dropout: a model whose widths were picked by hand
        dict(name="lm odd B30", kind="lm", V=5003, E=200, H=300, L=2, T=35, B=30, dropout=False, out="update"),
        # one rank's share of the language-model configuration on 8 GPUs; its gradients go to the sum over the ranks
        dict(name="lm share B64", kind="lm", V=10000, E=512, H=1024, L=2, T=35, B=64, dropout=True, out="grads"),
        # the language-model configuration on one GPU
        dict(name="lm full B512", kind="lm", V=10000, E=512, H=1024, L=2, T=35, B=512, dropout=True, out="update"),
        # the single-layer LSTM configuration: loss = sum of squares of all states
        dict(name="layer I128 H256 B32", kind="layer", I=128, H=256, B=32, T=50),
        # one interactive user: a prompt and eight tokens one at a time
        dict(name="generate B1", kind="generate", V=10000, E=512, H=1024, L=2, B=1, prompt=16, tokens=8),
        # the embedding + output softmax configuration
        dict(name="output V50000 N4096", kind="output", V=50000, E=512, N=4096),
        # the smallest calls: a hidden vector of a small model for a small batch
        dict(name="nodes D100 N16", kind="nodes", D=100, N=16),
        # the elementwise / normalisation sweep configuration
        dict(name="nodes D4096 N1024", kind="nodes", D=4096, N=1024),
        # the tagger as its example trains it (small mini-batches), one rank's share on 8 GPUs, and the whole configuration
        dict(name="tagger S16", kind="tagger", S=16, lo=5, hi=60, V=5000, E=128, H=256, TH=32, NT=45, out="update"),
        dict(name="tagger share S256", kind="tagger", S=256, lo=5, hi=100, V=20000, E=128, H=256, TH=32, NT=45, out="grads"),
        dict(name="tagger full S2048", kind="tagger", S=2048, lo=5, hi=100, V=20000, E=128, H=256, TH=32, NT=45, out="update"),
    ]


def draw(rng):
    def size(lo, hi, step=1):
        """Log-uniform in lo .. hi; every other time a multiple of `step`."""
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if rng.random() < 0.5 and step > 1:
            n = max(step, n // step * step)
        return max(lo, min(hi, n))

    kind = rng.choice(["lm", "layer", "generate", "output", "nodes", "nodes", "tagger"])
    if kind == "lm":
        return dict(kind=kind, V=size(500, 10000), E=size(32, 512, 32), H=size(64, 1024, 64), L=rng.choice([1, 2]), T=rng.randint(5, 35),
                    B=size(4, 512, 32), dropout=rng.random() < 0.5, out=rng.choice(["update", "grads"]))
    if kind == "layer":
        return dict(kind=kind, I=size(32, 1024, 32), H=size(64, 1024, 64), B=size(4, 512, 32), T=rng.randint(5, 50))
    if kind == "generate":
        return dict(kind=kind, V=size(500, 10000), E=size(32, 512, 32), H=size(64, 1024, 64), L=2, B=size(1, 64, 8), prompt=rng.randint(1, 35),
                    tokens=rng.randint(4, 16))
    if kind == "output":
        return dict(kind=kind, V=size(500, 50000), E=size(32, 512, 32), N=size(16, 4096, 32))
    if kind == "nodes":
        D = size(16, 8192, 64)
        return dict(kind=kind, D=D, N=size(1, min(4096, 4194304 // D), 8))
    return dict(kind="tagger", S=size(8, 1024, 8), lo=rng.randint(1, 10), hi=rng.randint(20, 100), V=size(500, 20000), E=size(32, 128, 32),
                H=size(64, 256, 64), TH=size(16, 128, 16), NT=rng.randint(5, 45), out=rng.choice(["update", "grads"]))


class _Program:
    """What a user's program holds; hands the driver's device memory back when it ends."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for close in getattr(self, "closers", ()):
            close()


def _tensor(t, dims, bd=1):
    return capi.DyTensor.of(t.data_ptr(), dims, bd)


def _zipf(r, n, V, s=1.1):
    cdf = np.cumsum(np.arange(1, V + 1, dtype=np.float64) ** (-s))
    return np.minimum(np.searchsorted(cdf / cdf[-1], r.random(n)), V - 1).astype(np.uint32)


def _glorot(gen, rows, cols):
    """Column-major [rows, cols] as a torch tensor [cols, rows]."""
    return (torch.rand(cols, rows, device="cuda", generator=gen) * 2 - 1) * math.sqrt(6.0 / (rows + cols))


def _device_ids(ids):
    return torch.from_numpy(ids.astype(np.uint32).view(np.int32)).cuda()


# ---- lm ------------------------------------------------------------------------------------------------------------------

def _prepare_lm(c, seed):
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        m = lm.LstmLm(c["V"], c["E"], c["H"], c["L"], c["T"], c["B"], seed=seed, dropout=c["dropout"], stream=stream.cuda_stream)
        tokens, _ = lm.synthetic_batch(dict(V=c["V"], E=c["E"], H=c["H"], L=c["L"], T=c["T"], B=c["B"]), seed=seed + 1000, dropout=0.0)
        pinned = torch.from_numpy(tokens.view(np.int32)).pin_memory()
        s = _Program(kind="lm", m=m, stream=stream, tokens=pinned, dropout=c["dropout"], update=c["out"] == "update", seed=seed, step=0,
                     closers=[m.close])
        # one step launch by launch (sizes the scratch memory), then the step as a graph, as the benchmark trains
        _run_lm(s)
        m.set_graph(True)
        _run_lm(s)
    return s


def _run_lm(s):
    m = s.m
    with torch.cuda.stream(s.stream):
        masks = m.draw_masks(KEEP, s.seed, s.step) if s.dropout else None
        s.step += 1
        if s.update:
            m.launch_forward_backward(s.tokens, masks)
            m.update()
            return {"loss": m.loss_dev, "params": m.params}
        m.grads.zero_()
        m.launch_forward_backward(s.tokens, masks)
        return {"loss": m.loss_dev, "grads": m.grads}


def _lm_params(c):
    return sum(r * k for r, k in lm.param_shapes(c["V"], c["E"], c["H"], c["L"]))


def _work_lm(c):
    per_token = 2.0 * c["V"] * c["H"] + sum(2.0 * 4 * c["H"] * ((c["E"] if l == 0 else c["H"]) + c["H"]) for l in range(c["L"]))
    return {"bytes": 8.0 * _lm_params(c) + 4.0 * (c["T"] + 1) * c["B"], "flops": 3.0 * per_token * c["T"] * c["B"]}


# ---- layer ---------------------------------------------------------------------------------------------------------------

def _prepare_layer(c, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    I, H, B, T = c["I"], c["H"], c["B"], c["T"]
    ctx = capi.Context(0, torch.cuda.current_stream().cuda_stream)
    x = torch.randn(T * B, I, device="cuda", generator=gen)
    Wx, Wh, b = _glorot(gen, 4 * H, I), _glorot(gen, 4 * H, H), torch.zeros(4 * H, device="cuda")
    zero = torch.zeros(B, H, device="cuda")
    gates, cs, hs = (torch.empty(T * B, n, device="cuda") for n in (4 * H, H, H))
    dh = torch.empty(T * B, H, device="cuda")
    acc = torch.zeros(T * B * (H + I) + 4 * H * (I + H + 1), device="cuda")   # everything that is accumulated into
    dc, dx, dWx, dWh, db = torch.split(acc, [T * B * H, T * B * I, 4 * H * I, 4 * H * H, 4 * H])
    w = ctx.wgrad_create(4 * H, I, H, T * B)
    s = _Program(kind="layer", ctx=ctx, w=w, acc=acc, hs=hs, dh=dh, dx=dx, dWx=dWx, dWh=dWh, db=db, G=4 * H, T=T,
                 keep=(x, Wx, Wh, b, zero, gates, cs, dc), closers=[lambda: ctx.wgrad_destroy(w)])
    s.at = capi.LstmGatesAttrs(0, 0.0, 1.0)
    s.tx, s.tz = _tensor(x, [I], T * B), _tensor(zero, [H], B)
    s.tWx, s.tWh, s.tb = _tensor(Wx, [4 * H, I]), _tensor(Wh, [4 * H, H]), _tensor(b, [4 * H])
    s.tg, s.tc, s.th = _tensor(gates, [4 * H], T * B), _tensor(cs, [H], T * B), _tensor(hs, [H], T * B)
    s.tdh, s.tdc, s.tdx, s.tdb = _tensor(dh, [H], T * B), _tensor(dc, [H], T * B), _tensor(dx, [I], T * B), _tensor(db, [4 * H])
    return s


def _run_layer(s):
    s.ctx.lstm_seq_fwd(s.tx, s.tz, s.tz, s.tWx, s.tWh, s.tb, None, None, s.at, s.tg, s.tc, s.th, s.w, s.T)
    s.acc.zero_()
    torch.mul(s.hs, 2.0, out=s.dh)                       # loss = sum of h^2
    s.ctx.lstm_seq_bwd(s.tx, s.tz, s.tz, s.tWx, s.tWh, None, None, s.at, s.tg, s.tc, s.th, s.tdh, s.tdc, s.tdx, None, None, s.tdb, s.w, s.T)
    s.ctx.wgrad_flush(s.w, s.dWx.data_ptr(), s.G, s.dWh.data_ptr(), s.G)
    return {"h": s.hs, "dx": s.dx, "dWx": s.dWx, "dWh": s.dWh, "db": s.db}


def _work_layer(c):
    I, H, n = c["I"], c["H"], c["T"] * c["B"]
    return {"bytes": 4.0 * (2 * 4 * H * (I + H + 1) + n * (2 * I + H)), "flops": 3.0 * 2.0 * 4 * H * (I + H) * n}


# ---- generate ------------------------------------------------------------------------------------------------------------

def _prepare_generate(c, seed):
    gen, r = torch.Generator("cuda").manual_seed(seed), np.random.Generator(np.random.PCG64(seed))
    V, E, H, L, B, P, S = (c[k] for k in ("V", "E", "H", "L", "B", "prompt", "tokens"))
    ctx = capi.Context(0, torch.cuda.current_stream().cuda_stream)
    ctx.param_cache(True)                                # the weights stay what they are while text is generated
    table = (torch.rand(V, E, device="cuda", generator=gen) * 2 - 1) * math.sqrt(3.0 / E)
    R, bias = _glorot(gen, V, H), torch.randn(V, device="cuda", generator=gen) * 0.1
    ids = _device_ids(_zipf(r, (P + S) * B, V))
    zero = torch.zeros(B, H, device="cuda")
    s = _Program(kind="generate", ctx=ctx, S=S, P=P, at=capi.LstmGatesAttrs(0, 0.0, 1.0), keep=[table, R, bias, ids, zero])
    xp = torch.empty(P * B, E, device="cuda")
    s.prompt = (_tensor(xp, [E], P * B), capi.LookupAttrs(table.data_ptr(), V, None, P * B, 1.0), ids.data_ptr())
    x = torch.empty(B, E, device="cuda")
    s.step_x, s.step_at = _tensor(x, [E], B), capi.LookupAttrs(table.data_ptr(), V, None, B, 1.0)
    s.step_ids = [ids.data_ptr() + 4 * (P + k) * B for k in range(S)]
    s.layers, s.states = [], []
    below, below_step = xp, [x, x]
    for l in range(L):
        I = E if l == 0 else H
        Wx, Wh, b = _glorot(gen, 4 * H, I), _glorot(gen, 4 * H, H), torch.randn(4 * H, device="cuda", generator=gen) * 0.1
        gp, cp, hp = (torch.empty(P * B, n, device="cuda") for n in (4 * H, H, H))
        g1 = torch.empty(B, 4 * H, device="cuda")
        c2, h2 = [torch.empty(B, H, device="cuda") for _ in range(2)], [torch.empty(B, H, device="cuda") for _ in range(2)]
        last = (_tensor(hp[(P - 1) * B:], [H], B), _tensor(cp[(P - 1) * B:], [H], B))
        s.layers.append(dict(W=(_tensor(Wx, [4 * H, I]), _tensor(Wh, [4 * H, H]), _tensor(b, [4 * H])), tz=_tensor(zero, [H], B),
                             xp=_tensor(below, [I], P * B), gp=_tensor(gp, [4 * H], P * B), cp=_tensor(cp, [H], P * B), hp=_tensor(hp, [H], P * B),
                             x=[_tensor(t, [I], B) for t in below_step], last=last, g=_tensor(g1, [4 * H], B),
                             c=[_tensor(t, [H], B) for t in c2], h=[_tensor(t, [H], B) for t in h2]))
        s.states += [c2[(S - 1) % 2], h2[(S - 1) % 2]]
        s.keep += [Wx, Wh, b, gp, cp, hp, g1, c2, h2]
        below, below_step = hp, h2
    logits, s.logp, s.aux = torch.empty(B, V, device="cuda"), torch.empty(S, B, V, device="cuda"), torch.empty(2 * B, device="cuda")
    s.keep += [xp, x, logits]
    s.tb, s.tR, s.param = _tensor(bias, [V]), _tensor(R, [V, H]), capi.AffineAttrs(1)   # 1: R is a parameter (its operand form is kept)
    s.tlogits, s.tlogp, s.dim0 = _tensor(logits, [V], B), [_tensor(s.logp[k], [V], B) for k in range(S)], capi.DimAttrs(0)
    return s


def _run_generate(s):
    ctx = s.ctx
    tx, at, ids = s.prompt
    ctx.fwd("lookup", [], tx, at, ids)
    for y in s.layers:
        Wx, Wh, b = y["W"]
        ctx.lstm_seq_fwd(y["xp"], y["tz"], y["tz"], Wx, Wh, b, None, None, s.at, y["gp"], y["cp"], y["hp"], None, s.P)
    for k in range(s.S):
        i = k % 2
        ctx.fwd("lookup", [], s.step_x, s.step_at, s.step_ids[k])
        for y in s.layers:
            Wx, Wh, b = y["W"]
            h, cc = y["last"] if k == 0 else (y["h"][1 - i], y["c"][1 - i])
            ctx.lstm_fwd_fused(y["x"][i], h, cc, Wx, Wh, b, None, None, s.at, y["g"], y["c"][i], y["h"][i])
        ctx.fwd("affine_transform", [s.tb, s.tR, s.layers[-1]["h"][i]], s.tlogits, s.param)
        ctx.fwd("log_softmax", [s.tlogits], s.tlogp[k], s.dim0, s.aux.data_ptr())
    return {"logp": s.logp, "states": s.states}


def _work_generate(c):
    V, E, H, L, B = (c[k] for k in ("V", "E", "H", "L", "B"))
    w = sum(4 * H * ((E if l == 0 else H) + H + 1) for l in range(L))
    head, n = V * (H + 1), c["prompt"] + c["tokens"]
    # the weights are read once for the prompt and once for every new token; log-probabilities are written once
    return {"bytes": 4.0 * (w * (1 + c["tokens"]) + head * c["tokens"] + n * B * E + c["tokens"] * B * V),
            "flops": 2.0 * B * (w * n + head * c["tokens"])}


# ---- output --------------------------------------------------------------------------------------------------------------

def _prepare_output(c, seed):
    gen, r = torch.Generator("cuda").manual_seed(seed), np.random.Generator(np.random.PCG64(seed))
    V, E, N = c["V"], c["E"], c["N"]
    ctx = capi.Context(0, torch.cuda.current_stream().cuda_stream)
    table = torch.randn(V, E, device="cuda", generator=gen) * 0.05
    W, b = _glorot(gen, V, E), torch.zeros(V, device="cuda")
    ids = _device_ids(_zipf(r, N, V))
    x, logits, loss, aux = torch.empty(N, E, device="cuda"), torch.empty(N, V, device="cuda"), torch.empty(N, device="cuda"), torch.zeros(3 * N, device="cuda")
    aux[2 * N:].view(torch.int32).copy_(_device_ids(_zipf(r, N, V)))                   # targets, on the device
    ones = torch.ones(N, device="cuda")
    acc = torch.zeros(N * E + V * (2 * E + 1), device="cuda")
    dx, dW, dtable, db = torch.split(acc, [N * E, V * E, V * E, V])
    s = _Program(kind="output", ctx=ctx, V=V, E=E, N=N, ids=ids, aux=aux, loss=loss, acc=acc, dx=dx, dW=dW, dtable=dtable, db=db,
                 keep=(table, W, b, x, logits, ones))
    s.look, s.pick = capi.LookupAttrs(table.data_ptr(), V, None, N, 1.0), capi.PickAttrs(None, N)
    s.tx, s.tlog, s.tloss, s.tones = _tensor(x, [E], N), _tensor(logits, [V], N), _tensor(loss, [1], N), _tensor(ones, [1], N)
    s.tW, s.tb, s.tdW, s.tdb, s.tdx = _tensor(W, [V, E]), _tensor(b, [V]), _tensor(dW, [V, E]), _tensor(db, [V]), _tensor(dx, [E], N)
    return s


def _run_output(s):
    ctx = s.ctx
    ctx.fwd("lookup", [], s.tx, s.look, s.ids.data_ptr())
    ctx.fwd("affine_transform", [s.tb, s.tW, s.tx], s.tlog)
    ctx.fwd("pickneglogsoftmax", [s.tlog], s.tloss, s.pick, s.aux.data_ptr())
    s.acc.zero_()
    ctx.softmax_output_bwd_fused(s.tlog, s.tx, s.tW, s.tones, s.aux.data_ptr(), s.tdW, s.tdb, s.tdx)
    ctx.lookup_accumulate_grads([], s.ids.data_ptr(), s.dx.data_ptr(), s.dtable.data_ptr(), s.E, s.V, n=s.N)
    return {"loss": s.loss, "dW": s.dW, "db": s.db, "dx": s.dx, "dtable": s.dtable}


def _work_output(c):
    V, E, N = c["V"], c["E"], c["N"]
    return {"bytes": 4.0 * (3 * V * E + 2 * V + 3 * N * E + 3 * N), "flops": 6.0 * V * E * N}


# ---- nodes ---------------------------------------------------------------------------------------------------------------

def _prepare_nodes(c, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    D, N = c["D"], c["N"]
    ctx = capi.Context(0, torch.cuda.current_stream().cuda_stream)
    x, x2, up = (torch.randn(N, D, device="cuda", generator=gen) for _ in range(3))
    gain, bias = torch.rand(D, device="cuda", generator=gen) + 0.5, torch.randn(D, device="cuda", generator=gen) * 0.1
    g1 = torch.rand(1, device="cuda", generator=gen) + 0.5
    col, mat = lambda t: _tensor(t, [D], N), lambda t: _tensor(t, [D, N])   # noqa: E731
    calls = [("tanh", [col(x)], None, [0]), ("logistic", [col(x)], None, [0]), ("rectify", [col(x)], None, [0]),
             ("elu", [col(x)], capi.EluAttrs(1.0, 1.0), [0]), ("cmult", [col(x), col(x2)], None, [0, 1]),
             ("softmax", [col(x)], capi.DimAttrs(0), [0]), ("softmax", [mat(x)], capi.DimAttrs(1), [0]),
             ("layer_norm", [col(x), _tensor(gain, [D]), _tensor(bias, [D])], None, [0, 1, 2]),
             ("weight_norm", [mat(x), _tensor(g1, [1])], None, [0, 1])]
    room = lambda n: (n + 3) // 4 * 4                                        # every gradient starts on 16 bytes  # noqa: E731
    sizes = [room(D if n == "layer_norm" and i else 1 if n == "weight_norm" and i else D * N) for n, _, _, bwd in calls for i in bwd]
    acc = torch.zeros(sum(sizes), device="cuda")
    grads, at = list(torch.split(acc, sizes)), 0
    s = _Program(kind="nodes", ctx=ctx, acc=acc, plan=[], outs=[], keep=(x, x2, up, gain, bias, g1))
    for name, xs, attrs, bwd in calls:
        y = torch.empty(N, D, device="cuda")
        shape = mat if xs[0].nd == 2 else col
        back = []
        for i in bwd:
            d, at = grads[at], at + 1
            small = D if name == "layer_norm" and i else 1 if name == "weight_norm" and i else 0
            back.append((i, _tensor(d, [small]) if small else shape(d)))
            s.outs.append(d)
        s.plan.append((name, xs, attrs, shape(y), shape(up), back))
        s.outs.append(y)
    return s


def _run_nodes(s):
    ctx = s.ctx
    s.acc.zero_()
    for name, xs, attrs, y, up, back in s.plan:
        ctx.fwd(name, xs, y, attrs)
        for i, d in back:
            ctx.bwd(name, xs, y, up, i, d, attrs)
    return s.outs


def _work_nodes(c):
    # forward 2 tensors in and out (cmult 3), backward 3 per full-size gradient: 49 in all
    return {"bytes": 4.0 * 49 * c["D"] * c["N"], "flops": 100.0 * c["D"] * c["N"]}


# ---- tagger --------------------------------------------------------------------------------------------------------------

def _prepare_tagger(c, seed):
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        lens, words, tags = tagger.synthetic_corpus(c["S"], c["V"], c["NT"], seed=seed + 2000, lo=c["lo"], hi=c["hi"])
        m = tagger.Tagger(c["V"], c["E"], c["H"], c["TH"], c["NT"], max_sentences=c["S"], max_tokens=int(lens.sum()), max_len=c["hi"],
                          seed=seed, stream=stream.cuda_stream)
    return _Program(kind="tagger", m=m, stream=stream, batch=(lens, words, tags), update=c["out"] == "update", closers=[m.close])


def _run_tagger(s):
    m = s.m
    with torch.cuda.stream(s.stream):
        if s.update:
            m.launch_forward_backward(*s.batch)
            m.update()
            return {"loss": m.loss_dev, "params": m.params}
        m.grads.zero_()
        m.launch_forward_backward(*s.batch)
        return {"loss": m.loss_dev, "grads": m.grads}


def _work_tagger(c):
    n = c["S"] * (c["lo"] + c["hi"]) / 2.0                                   # expected number of tokens
    E, H, TH, NT = c["E"], c["H"], c["TH"], c["NT"]
    params = sum(r * k for r, k in tagger.param_shapes(c["V"], E, H, TH, NT))
    return {"bytes": 8.0 * params + 8.0 * n, "flops": 3.0 * 2.0 * n * (2 * 4 * H * (E + H) + 2 * TH * H + NT * TH)}


# ---- the five functions --------------------------------------------------------------------------------------------------

_PREPARE = dict(lm=_prepare_lm, layer=_prepare_layer, generate=_prepare_generate, output=_prepare_output, nodes=_prepare_nodes,
                tagger=_prepare_tagger)
_RUN = dict(lm=_run_lm, layer=_run_layer, generate=_run_generate, output=_run_output, nodes=_run_nodes, tagger=_run_tagger)
_WORK = dict(lm=_work_lm, layer=_work_layer, generate=_work_generate, output=_work_output, nodes=_work_nodes, tagger=_work_tagger)


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    torch.cuda.synchronize()
    return s


def run(state):
    return _RUN[state.kind](state)


def work(case):
    return _WORK[case["kind"]](case)


def tolerance(case):
    # float32 with sums in an order of the implementation's choosing; where a recurrence passes on the rounding of up to 100
    # steps, five times that of one sum
    return {"rel": 5e-5 if case["kind"] in ("lm", "layer", "generate", "tagger") else 1e-5}
