"""The optimizer-step and codec workloads this package is timed on.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)` one more of the same ranges, `prepare`
what a training program holds before the call (parameters, gradients, an optimizer in mid-training), `run` one call
through the public classes (`optimizer.step()`, the functions of `came_b200.quant`), `work` the compulsory bytes and
operations of it and `tolerance` how far two correct implementations may be apart.

Parameter sets (`"set"`):

    decoder   a decoder-only transformer: embedding and head [vocab, hidden], per layer q, o [hidden, hidden], k, v
              [hidden, kv], gate, up [hidden, ffn], down [ffn, hidden] and two norm vectors
    gpt       the GPT-2 arrangement: token and position embeddings, fused qkv, biases, two LayerNorms per layer
    adapter   pairs of low-rank factors [rank, width], [width, rank]
    conv      3 x 3 and 1 x 1 convolution kernels over a pyramid of widths, each with a bias
    dense     one matrix and its bias
    odd       a token embedding, a head stored [hidden, vocab] and two feed-forward matrices whose sizes are no multiple of 8
    codec     one fp32 matrix through the blockwise and the tile codec, both directions
"""
import math

import torch

import came_b200
from came_b200 import quant
from came_b200.optim import bind_flat_views

LR, WD = 2e-4, 1e-2
CHUNK = 1 << 30          # elements of one flat buffer at most
ALIGN = 512              # bytes: what the allocator gives a tensor of its own


def listed():
    return [
        # the smallest call: a linear probe on top of frozen features
        dict(name="probe-fp32-came", set="dense", rows=1000, cols=768, cls="CAME", dtype="float32"),
        # low-rank fine-tuning: hundreds of small thin matrices, where launches and the host count
        dict(name="adapter-bf16-8bit", set="adapter", modules=264, rank=16, width=640, cls="CAME8bit", dtype="bfloat16"),
        # a small language model whose whole step is replayed as a CUDA graph
        dict(name="small-lm-graph-bf16-8bit", set="decoder", vocab=8000, hidden=512, kv=512, ffn=1408, layers=8, cls="CAME8bit",
             dtype="bfloat16", graph=True),
        # a mid-size language model; the trainer drops its gradients every step (zero_grad(set_to_none=True)), so that
        # they lie elsewhere in the next one
        dict(name="mid-lm-moved-grads-bf16-8bit", set="decoder", vocab=32000, hidden=1024, kv=256, ffn=2816, layers=12, cls="CAME8bit",
             dtype="bfloat16", moved=True),
        # one large square layer, plain CAME
        dict(name="square-fp32-came", set="dense", rows=4096, cols=4096, cls="CAME", dtype="float32"),
        # full fine-tuning of a convolutional network with loss scaling: tensors of more than two dimensions
        dict(name="conv-fp16-full", set="conv", width=320, levels=3, blocks=2, cls="CAME8bitFull", dtype="float16", grad_scale=1.0 / 1024),
        # a model whose vocabulary and widths suit no tile
        dict(name="odd-bf16-8bit", set="odd", vocab=50257, hidden=770, ffn=3083, cls="CAME8bit", dtype="bfloat16"),
        # pre-training of GPT-2 medium in fp32
        dict(name="gpt2m-fp32-camecuda", set="gpt", vocab=50257, hidden=1024, layers=24, cls="CAMECUDA", dtype="float32"),
        # a 1.3 B parameter model with the memory-saving class (flat layout)
        dict(name="llama1b-bf16-memory", set="decoder", vocab=32000, hidden=2048, kv=2048, ffn=5632, layers=22, cls="CAME8bitMemory",
             dtype="bfloat16"),
        # the same model, matrices only, fp16 with loss scaling
        dict(name="llama1b-fp16-2d", set="decoder", vocab=32000, hidden=2048, kv=2048, ffn=5632, layers=22, vectors=False, cls="CAME8bit2D",
             dtype="float16", grad_scale=1.0 / 1024),
        # the largest: all of Llama-7B on one GPU
        dict(name="llama7b-bf16-8bit", set="decoder", vocab=32000, hidden=4096, kv=4096, ffn=11008, layers=32, cls="CAME8bit",
             dtype="bfloat16"),
        # the codec on its own, encode and decode, both layouts (checkpoint conversion, state surgery)
        dict(name="codec-4096x11008", set="codec", rows=4096, cols=11008),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, step=64, odd=0.25):
    """A width of the range: mostly a multiple of `step`, sometimes whatever comes."""
    n = _log(rng, lo, hi)
    return n if rng.random() < odd else max(step, n // step * step)


def draw(rng):
    kind = rng.choice(["decoder", "decoder", "decoder", "gpt", "adapter", "conv", "dense", "odd", "codec"])
    if kind == "codec":
        return dict(set="codec", rows=_log(rng, 64, 8192), cols=_log(rng, 64, 11008))
    cls = rng.choice(["CAME8bit", "CAME8bit", "CAME8bit2D", "CAME8bitMemory", "CAME8bitFull", "CAMECUDA", "CAME"])
    dtype = rng.choice(["bfloat16", "bfloat16", "float16", "float32"])
    case = dict(set=kind, cls=cls, dtype=dtype)
    if kind == "decoder":
        hidden = _size(rng, 128, 4096)
        kv = hidden if rng.random() < 0.5 else max(64, hidden // 4)
        case.update(vocab=_size(rng, 1000, 64000, 64, 0.5), hidden=hidden, kv=kv, ffn=_size(rng, 2 * hidden, 4 * hidden, 64, 0.1))
        per_layer = hidden * (2 * hidden + 2 * kv + 3 * case["ffn"])
        most = max(1, (1_500_000_000 - 2 * case["vocab"] * hidden) // per_layer)
        case["layers"] = _log(rng, 1, min(32, most))
    elif kind == "gpt":
        hidden = _size(rng, 128, 1600)
        case.update(vocab=_size(rng, 1000, 50257, 64, 0.5), hidden=hidden, layers=_log(rng, 1, 24))
    elif kind == "adapter":
        case.update(modules=_log(rng, 8, 300), rank=rng.choice([4, 8, 16, 32, 64]), width=_size(rng, 256, 4096))
    elif kind == "conv":
        case.update(width=_size(rng, 32, 320, 32), levels=rng.randint(1, 3), blocks=rng.randint(1, 3))
    elif kind == "dense":
        case.update(rows=_log(rng, 64, 16384), cols=_size(rng, 64, 16384))
    else:
        case.update(vocab=_log(rng, 1000, 50257), hidden=_log(rng, 129, 1100), ffn=_log(rng, 500, 4400))
    if cls == "CAME8bit2D":
        if kind == "conv":
            case["cls"] = "CAME8bitFull"
        else:
            case["vectors"] = False
    if dtype == "float16" and rng.random() < 0.5:
        case["grad_scale"] = 1.0 / 1024
    if kind != "adapter" and rng.random() < 0.2:
        case["graph"] = True
    elif rng.random() < 0.25:
        case["moved"] = True
    return case


def _shapes(case):
    kind = case["set"]
    if kind == "decoder":
        h, kv, f = case["hidden"], case["kv"], case["ffn"]
        out = [(case["vocab"], h)]
        for _ in range(case["layers"]):
            out += [(h, h), (h, kv), (h, kv), (h, h), (h, f), (h, f), (f, h), (h,), (h,)]
        out += [(h,), (case["vocab"], h)]
    elif kind == "gpt":
        h = case["hidden"]
        out = [(case["vocab"], h), (1024, h)]
        for _ in range(case["layers"]):
            out += [(h,), (h,), (h, 3 * h), (3 * h,), (h, h), (h,), (h,), (h,), (h, 4 * h), (4 * h,), (4 * h, h), (h,)]
        out += [(h,), (h,)]
    elif kind == "adapter":
        out = []
        for i in range(case["modules"]):
            w = case["width"] * (1 + i % 2)
            out += [(case["rank"], w), (w, case["rank"])]
    elif kind == "conv":
        out, c_in = [], 4
        for level in range(case["levels"]):
            c = case["width"] << level
            out += [(c, c_in, 3, 3), (c,)]
            for _ in range(case["blocks"]):
                out += [(c, c, 3, 3), (c,), (c, c, 1, 1), (c,)]
            c_in = c
    elif kind == "dense":
        out = [(case["rows"], case["cols"]), (case["rows"],)]
    else:
        v, h, f = case["vocab"], case["hidden"], case["ffn"]
        out = [(v, h), (h, f), (f,), (f, h), (h,), (h, v)]
    return out if case.get("vectors", True) else [s for s in out if len(s) > 1]


def _flat(tensors):
    """Moves tensors of one dtype into flat buffers (every tensor on an allocation boundary); -> buffers, views."""
    esz = tensors[0].element_size()
    step = ALIGN // esz
    groups, size = [[]], 0
    for i, t in enumerate(tensors):
        n = -(-t.numel() // step) * step
        if size and size + n > CHUNK:
            groups.append([])
            size = 0
        groups[-1].append((i, size))
        size += n
    buffers, views = [], [None] * len(tensors)
    for group in groups:
        i, at = group[-1]
        buf = torch.zeros(at + -(-tensors[i].numel() // step) * step, dtype=tensors[0].dtype, device=tensors[0].device)
        for i, at in group:
            t = tensors[i]
            views[i] = buf[at: at + t.numel()].view(t.shape)
            views[i].copy_(t)
        buffers.append(buf)
    return buffers, views


def _fill_grads(params, sets, gen, scales, inv_scale):
    for grads in sets:
        for p, g, sc in zip(params, grads, scales):
            g.copy_(torch.randn(p.shape, generator=gen, device=p.device).mul_(sc * inv_scale))


class _Training:
    """A training program between backward() and step()."""

    def __init__(self, case, seed):
        dev = torch.device("cuda")
        gen = torch.Generator(device=dev).manual_seed(seed)
        host = torch.Generator().manual_seed(seed)
        dtype = getattr(torch, case["dtype"])
        shapes = _shapes(case)
        # weights N(0, 0.02^2); gradients N(0, 1) times a scale of the tensor's own, times the loss scale
        self.param_buffers, views = _flat([torch.empty(s, dtype=dtype, device=dev) for s in shapes])
        for v in views:
            v.copy_(torch.randn(v.shape, generator=gen, device=dev).mul_(0.02))
        self.params = [torch.nn.Parameter(v) for v in views]
        scales = [10.0 ** float(x) for x in torch.empty(len(shapes)).uniform_(-5, -2, generator=host)]
        gs = case.get("grad_scale", 1.0)
        self.sets = [[torch.empty_like(p) for p in self.params] for _ in range(2 if case.get("moved") else 1)]
        self.turn = 0
        kwargs = {} if case["cls"] == "CAME" else dict(eps=(1e-30, 1e-16), clip_threshold=1.0)
        self.opt = getattr(came_b200, case["cls"])(self.params, lr=LR, weight_decay=WD, betas=(0.9, 0.95, 0.995), **kwargs)
        if gs != 1.0:
            self.opt.param_groups[0]["grad_scale"] = gs
        _fill_grads(self.params, self.sets, gen, scales, 1.0 / gs)
        for p, g in zip(self.params, self.sets[0]):
            p.grad = g
        # optimizer states in flat buffers, one kind after the other, as sharded optimizers keep them
        self.opt.prime_for_cuda_graph()
        self.state_buffers = {}
        kept = {}
        for p in self.params:
            st = self.opt.state[p]
            for k, v in st.items():
                if torch.is_tensor(v) and not v._is_view():
                    kept.setdefault((k, v.dtype), []).append(st)
        for (k, dt), states in kept.items():
            buffers, moved = _flat([st[k] for st in states])
            self.state_buffers[f"{k}:{dt}"] = buffers
            for st, v in zip(states, moved):
                st[k] = v
        for p in self.params:
            if "factored_row_q" in self.opt.state[p]:
                bind_flat_views(self.opt.state[p])
        # one step of the past: no state is at its initial value
        self.opt.step()
        _fill_grads(self.params, self.sets, gen, scales, 1.0 / gs)
        self.graph = None
        if case.get("graph"):
            torch.cuda.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph):
                self.opt.step()
        self.outputs = {"params": self.param_buffers, **self.state_buffers}

    def step(self):
        if self.graph is not None:
            self.graph.replay()
        else:
            if len(self.sets) > 1:
                self.turn ^= 1
                for p, g in zip(self.params, self.sets[self.turn]):
                    p.grad = g
            self.opt.step()
        return self.outputs


def prepare(case, seed):
    if case["set"] == "codec":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(case["rows"], case["cols"], generator=gen, device="cuda")
        # momenta: magnitudes that vary from row to row
        x *= torch.randn(case["rows"], 1, generator=gen, device="cuda").exp_().mul_(1e-3)
        return x
    return _Training(case, seed)


def run(state):
    if isinstance(state, _Training):
        return state.step()
    q, a = quant.quantize_blockwise(state, signed=True)
    u, b = quant.quantize_blockwise(state, signed=False)
    t, c = quant.quantize_tile16(state)
    return [q, a, quant.dequantize_blockwise(q, a, signed=True), u, b, quant.dequantize_blockwise(u, b, signed=False),
            t, c, quant.dequantize_tile16(t, c)]


def work(case):
    if case["set"] == "codec":
        n = case["rows"] * case["cols"]
        # three encodes (4 bytes in, 1 out), three decodes (1 in, 4 out), an absmax per 256 elements
        return {"bytes": 6.0 * (5 * n + 4 * math.ceil(n / 256)), "flops": 6.0 * 4 * n}
    esz = 4 if case["dtype"] == "float32" else 2
    fp32 = case["cls"] in ("CAME", "CAMECUDA")
    msz = 4.0 if fp32 else 1.0 + 4.0 / 256      # a state value with its share of the absmax
    nbytes = flops = 0.0
    for s in _shapes(case):
        n = math.prod(s)
        nbytes += n * (3 * esz + 2 * msz)       # gradient read, parameter and momentum read and written
        if len(s) == 1:
            nbytes += n * 2 * msz               # second moment read and written
            flops += 15.0 * n
        else:                                   # second-moment and residual vectors
            nbytes += 4 * msz * (n / s[-1] + n / s[-2])
            flops += 20.0 * n
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["set"] == "codec":
        return "exact"
    fp32_states = case["cls"] in ("CAME", "CAMECUDA")
    if case["dtype"] == "float32":
        # 8-bit states: an entry on a rounding boundary moves by one code, which moves what is derived from it
        return {"rel": 1e-5, "max": 1e-3} if fp32_states else {"rel": 1e-3, "max": 2e-2, "differ": 0.01}
    # parameters in 16 bits: a value next to a rounding boundary moves by one spacing, twice where decay rounds too
    return {"rel": 1e-2, "max": 2e-2, "differ": 0.01}
