"""The work this framework is used for, as cases that can be timed: whole modules through ``DaceModule`` and the encoder
runner, from single requests to full batches.

Every case is one forward pass of a network in evaluation mode with weights and inputs drawn from a seed.  The modules
are written the way a user writes them (plain ``torch.nn``); the framework exports, imports, optimises and compiles
them in ``prepare``, as a program does once, and ``run`` is the call such a program makes for each batch.
"""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F

from daceml_b200.runner import BertEncoder
from daceml_b200.torch import DaceModule

DTYPES = {"fp16": torch.float16, "fp32": torch.float32}


# ---------------------------------------------------------------------------------------------
# modules
# ---------------------------------------------------------------------------------------------
class MLP(nn.Module):
    """Three linear layers with ReLU and a log-softmax over the classes."""

    def __init__(self, features, hidden1, hidden2, classes):
        super().__init__()
        self.fc1, self.fc2, self.fc3 = nn.Linear(features, hidden1), nn.Linear(hidden1, hidden2), nn.Linear(hidden2, classes)

    def forward(self, x):
        return F.log_softmax(self.fc3(F.relu(self.fc2(F.relu(self.fc1(x))))), dim=-1)


class LeNet(nn.Module):
    """32x32 images: two 3x3 convolutions with ReLU and 2x2 max pooling, three linear layers, log-softmax."""

    def __init__(self):
        super().__init__()
        self.conv1, self.conv2 = nn.Conv2d(1, 6, 3), nn.Conv2d(6, 16, 3)
        self.fc1, self.fc2, self.fc3 = nn.Linear(16 * 6 * 6, 120), nn.Linear(120, 84), nn.Linear(84, 10)

    def forward(self, x):
        x = F.max_pool2d(F.relu(self.conv1(x)), 2)
        x = F.max_pool2d(F.relu(self.conv2(x)), 2)
        x = x.view(-1, 16 * 6 * 6)
        return F.log_softmax(self.fc3(F.relu(self.fc2(F.relu(self.fc1(x))))), dim=1)


class EncoderLayer(nn.Module):
    """Post-LN transformer encoder layer (attention with 64-wide heads, erf GELU), as BERT's."""

    def __init__(self, hidden, ffn):
        super().__init__()
        self.heads = hidden // 64
        self.q, self.k, self.v, self.o = (nn.Linear(hidden, hidden) for _ in range(4))
        self.up, self.down = nn.Linear(hidden, ffn), nn.Linear(ffn, hidden)
        self.ln1, self.ln2 = nn.LayerNorm(hidden, eps=1e-12), nn.LayerNorm(hidden, eps=1e-12)

    def forward(self, x, mask=None):
        b, s, h = x.shape
        q, k, v = (p(x).view(b, s, self.heads, 64).transpose(1, 2) for p in (self.q, self.k, self.v))
        scores = torch.matmul(q, k.transpose(2, 3)) * 0.125
        if mask is not None:
            scores = scores + mask
        ctx = torch.matmul(torch.softmax(scores, dim=-1), v).transpose(1, 2).contiguous().reshape(b, s, h)
        x = self.ln1(self.o(ctx) + x)
        return self.ln2(self.down(F.gelu(self.up(x))) + x)


class Encoder(nn.Module):
    """Encoder layers over hidden states; with ``whole`` also token and position embeddings in front (token ids and a
    padding mask as inputs) and the pooler behind."""

    def __init__(self, layers, hidden, ffn, whole, vocab=1000, positions=512):
        super().__init__()
        self.whole = whole
        self.layers = nn.ModuleList([EncoderLayer(hidden, ffn) for _ in range(layers)])
        if whole:
            self.tok, self.pos = nn.Embedding(vocab, hidden), nn.Embedding(positions, hidden)
            self.norm = nn.LayerNorm(hidden, eps=1e-12)
            self.pooler = nn.Linear(hidden, hidden)

    def forward(self, x, mask=None):
        if not self.whole:
            for layer in self.layers:
                x = layer(x)
            return x
        h = self.norm(self.tok(x) + self.pos.weight[:x.shape[1]])
        bias = (1.0 - mask[:, None, None, :].to(h.dtype)) * -10000.0
        for layer in self.layers:
            h = layer(h, bias)
        return h, torch.tanh(self.pooler(h[:, 0]))


class MBConv(nn.Module):
    """Inverted-bottleneck block with squeeze-excite, batch normalisation folded into the convolutions."""

    def __init__(self, cin, mid, red):
        super().__init__()
        self.expand = nn.Conv2d(cin, mid, 1)
        self.depthwise = nn.Conv2d(mid, mid, 3, padding=1, groups=mid)
        self.se_reduce, self.se_expand = nn.Conv2d(mid, red, 1), nn.Conv2d(red, mid, 1)
        self.project = nn.Conv2d(mid, cin, 1)

    def forward(self, x):
        y = self.expand(x)
        y = y * torch.sigmoid(y)
        y = self.depthwise(y)
        y = y * torch.sigmoid(y)
        s = self.se_reduce(F.adaptive_avg_pool2d(y, 1))
        s = self.se_expand(s * torch.sigmoid(s))
        return self.project(torch.sigmoid(s) * y) + x


class BasicBlock(nn.Module):
    """Residual block of two 3x3 convolutions with batch normalisation; strided with a 1x1 shortcut when it down-samples."""

    def __init__(self, cin, cout, stride):
        super().__init__()
        self.conv1, self.bn1 = nn.Conv2d(cin, cout, 3, stride=stride, padding=1, bias=False), nn.BatchNorm2d(cout)
        self.conv2, self.bn2 = nn.Conv2d(cout, cout, 3, padding=1, bias=False), nn.BatchNorm2d(cout)
        self.down = None
        if stride != 1 or cin != cout:
            self.down = nn.Sequential(nn.Conv2d(cin, cout, 1, stride=stride, bias=False), nn.BatchNorm2d(cout))

    def forward(self, x):
        y = torch.relu(self.bn1(self.conv1(x)))
        y = self.bn2(self.conv2(y))
        return torch.relu(y + (x if self.down is None else self.down(x)))


# ---------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # one request to a small network: the time of the call itself
        dict(name="mlp request", kind="mlp", batch=1, features=784, hidden1=120, hidden2=32, classes=10, dtype="fp32", graph=False),
        # the same network over a full batch
        dict(name="mlp batch", kind="mlp", batch=4096, features=784, hidden1=120, hidden2=32, classes=10, dtype="fp32", graph=False),
        # a small convolutional network on a few images: eight short launches in a row
        dict(name="lenet images", kind="lenet", batch=8, dtype="fp32", graph=False),
        # a single strided convolution on a batch of small images, as a first layer has it
        dict(name="strided conv", kind="conv", batch=32, cin=3, cout=16, size=64, kernel=3, stride=2, pad=0, dtype="fp32", graph=False),
        # one text request to a whole encoder: ids and padding mask in, hidden states and pooled vector out, odd length
        dict(name="bert request", kind="encoder", layers=4, batch=1, seq=77, hidden=768, whole=True, dtype="fp16", graph=False),
        # a batch of short padded texts for classification
        dict(name="bert classify", kind="encoder", layers=2, batch=32, seq=128, hidden=768, whole=True, dtype="fp16", graph=False),
        # the BERT-large encoder layer over full-length samples, replayed as a CUDA graph
        dict(name="bert-large layer", kind="encoder", layers=1, batch=8, seq=512, hidden=1024, whole=False, dtype="fp16", graph=True),
        # a base-size encoder layer in full precision
        dict(name="bert-base fp32", kind="encoder", layers=1, batch=8, seq=512, hidden=768, whole=False, dtype="fp32", graph=False),
        # the 24-layer BERT-large encoder on one GPU's share of a large batch
        dict(name="bert-large stack", kind="stack", layers=24, batch=8, seq=512, hidden=1024, dtype="fp16", graph=True),
        # the first inverted-bottleneck stage of an image classifier over a large batch
        dict(name="mbconv batch", kind="mbconv", batch=128, cin=24, size=56, dtype="fp32", graph=False),
        # a down-sampling residual block over a batch
        dict(name="resnet down", kind="block", batch=32, cin=64, cout=128, size=56, stride=2, dtype="fp32", graph=False),
        # a residual block in half precision, a few images at a time
        dict(name="resnet half", kind="block", batch=8, cin=64, cout=64, size=56, stride=1, dtype="fp16", graph=False),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["mlp", "lenet", "conv", "encoder", "encoder", "encoder", "stack", "mbconv", "block", "block"])
    graph = rng.random() < 0.3
    if kind == "mlp":
        return dict(kind=kind, batch=_log(rng, 1, 32768), features=_log(rng, 64, 1024), hidden1=_log(rng, 32, 512),
                    hidden2=_log(rng, 16, 256), classes=_log(rng, 2, 100), dtype=rng.choice(["fp32", "fp32", "fp16"]), graph=graph)
    if kind == "lenet":
        return dict(kind=kind, batch=_log(rng, 1, 1024), dtype="fp32", graph=graph)
    if kind == "conv":
        kernel = rng.choice([1, 3, 3, 3, 5, 7])
        case = dict(kind=kind, batch=_log(rng, 1, 64), cin=_log(rng, 3, 64), cout=_log(rng, 8, 128), size=_log(rng, 16, 160),
                    kernel=kernel, stride=rng.choice([1, 1, 2]), pad=rng.choice([0, kernel // 2]), dtype=rng.choice(["fp32", "fp32", "fp16"]),
                    graph=graph)
        return _shrink(case, 8e9)
    if kind == "encoder":
        dtype = rng.choice(["fp16", "fp16", "fp16", "fp32"])
        case = dict(kind=kind, layers=rng.choice([1, 1, 2, 3]), batch=_log(rng, 1, 64), seq=_log(rng, 8, 512),
                    hidden=rng.choice([128, 256, 512, 768, 768, 1024]), whole=rng.random() < 0.5, dtype=dtype, graph=graph)
        return _shrink(case, 3e11 if dtype == "fp16" else 8e10)
    if kind == "stack":
        case = dict(kind=kind, layers=_log(rng, 4, 24), batch=_log(rng, 1, 8), seq=_log(rng, 64, 512),
                    hidden=rng.choice([256, 512, 768, 1024]), dtype="fp16", graph=True)
        return _shrink(case, 2.5e12)
    if kind == "mbconv":
        case = dict(kind=kind, batch=_log(rng, 1, 128), cin=8 * rng.randint(2, 5), size=_log(rng, 7, 112),
                    dtype=rng.choice(["fp32", "fp32", "fp16"]), graph=graph)
        return _shrink(case, 8e9)
    stride = rng.choice([1, 2])
    cin = rng.choice([32, 64, 64, 128, 256])
    case = dict(kind="block", batch=_log(rng, 1, 64), cin=cin, cout=cin * stride, size=_log(rng, 7, 64), stride=stride,
                dtype=rng.choice(["fp32", "fp16"]), graph=graph)
    return _shrink(case, 1.2e10)


def _shrink(case, flops):
    """The case with its batch made smaller until it costs at most ``flops`` operations."""
    while case["batch"] > 1 and work(case)["flops"] > flops:
        case["batch"] = max(1, case["batch"] * 3 // 4)
    return case


def _module(case):
    kind = case["kind"]
    if kind == "mlp":
        return MLP(case["features"], case["hidden1"], case["hidden2"], case["classes"])
    if kind == "lenet":
        return LeNet()
    if kind == "conv":
        return nn.Conv2d(case["cin"], case["cout"], case["kernel"], stride=case["stride"], padding=case["pad"], bias=False)
    if kind == "encoder":
        return Encoder(case["layers"], case["hidden"], 4 * case["hidden"], case["whole"])
    if kind == "mbconv":
        return MBConv(case["cin"], 6 * case["cin"], max(1, case["cin"] // 4))
    return BasicBlock(case["cin"], case["cout"], case["stride"])


def _init(module):
    """Weights as trained networks of these kinds have them in scale: N(0, 0.02) for the encoder's products, PyTorch's
    own initialisation elsewhere, batch statistics near one."""
    for m in module.modules():
        if isinstance(m, nn.BatchNorm2d):
            m.running_mean.normal_(0.0, 0.1), m.running_var.uniform_(0.5, 1.5)
            m.weight.data.uniform_(0.5, 1.5), m.bias.data.normal_(0.0, 0.1)
        elif isinstance(m, nn.LayerNorm):
            m.weight.data.uniform_(0.8, 1.2), m.bias.data.normal_(0.0, 0.05)
        elif isinstance(module, Encoder) and isinstance(m, nn.Linear):
            m.weight.data.normal_(0.0, 0.02), m.bias.data.normal_(0.0, 0.02)
    return module.eval()


def _stack_params(case, gen):
    hidden, ffn = case["hidden"], 4 * case["hidden"]

    def normal(*shape, mean=0.0, std=0.02):
        return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float16) * std + mean

    def layer():
        p = {"w" + n: normal(hidden, hidden) for n in "qkvo"}
        p.update({"b" + n: normal(hidden) for n in "qkvo"})
        p.update(w1=normal(ffn, hidden), b1=normal(ffn), w2=normal(hidden, ffn), b2=normal(hidden))
        for n in ("ln1", "ln2"):
            p[n + "_g"], p[n + "_b"] = normal(hidden, mean=1.0, std=0.1), normal(hidden, std=0.05)
        return p

    return [layer() for _ in range(case["layers"])]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    kind, batch = case["kind"], case["batch"]
    if kind == "stack":
        encoder = BertEncoder(_stack_params(case, gen), batch, case["seq"], case["hidden"] // 64, cuda_graph=case["graph"])
        return dict(call=encoder, args=(torch.randn(batch, case["seq"], case["hidden"], generator=gen, device="cuda", dtype=dtype), ))
    torch.manual_seed(seed)
    with torch.device("cuda"), torch.no_grad():
        module = _init(_module(case)).to(dtype)
    if kind == "mlp":
        shape = (batch, case["features"])
    elif kind == "lenet":
        shape = (batch, 1, 32, 32)
    elif kind == "encoder":
        shape = (batch, case["seq"], case["hidden"])
    else:
        shape = (batch, case["cin"], case["size"], case["size"])
    args = (torch.randn(shape, generator=gen, device="cuda", dtype=dtype), )
    if kind == "encoder" and case["whole"]:
        ids = torch.randint(0, 1000, (batch, case["seq"]), generator=gen, device="cuda")
        # texts fill between half and all of the padded length
        lengths = torch.randint((case["seq"] + 1) // 2, case["seq"] + 1, (batch, 1), generator=gen, device="cuda")
        args = (ids, (torch.arange(case["seq"], device="cuda") < lengths).to(torch.int64))
    call = DaceModule(module, dummy_inputs=args, cuda_graph=case["graph"])
    return dict(call=call, args=args)


def run(state):
    return state["call"](*state["args"])


def work(case):
    """Operations of the contractions, and the bytes of the inputs, the parameters and the outputs."""
    kind, n, e = case["kind"], case["batch"], 2 if case["dtype"] == "fp16" else 4
    if kind == "mlp":
        f, a, b, c = case["features"], case["hidden1"], case["hidden2"], case["classes"]
        params = f * a + a * b + b * c
        return dict(bytes=e * (params + a + b + c + n * (f + c)), flops=2.0 * n * params)
    if kind == "lenet":
        linear = 576 * 120 + 120 * 84 + 84 * 10
        return dict(bytes=e * (6 * 9 + 16 * 54 + linear + n * (1024 + 10)),
                    flops=2.0 * n * (30 * 30 * 6 * 9 + 13 * 13 * 16 * 54 + linear))
    if kind in ("encoder", "stack"):
        h, s, layers = case["hidden"], case["seq"], case["layers"]
        per_layer, tokens = 12 * h * h, n * s
        flops = layers * (2.0 * tokens * per_layer + 4.0 * n * s * s * h)
        nbytes = e * (layers * (per_layer + 13 * h) + 2 * tokens * h)
        if case.get("whole"):  # the rows of the embedding table that the ids name, int64 ids and mask
            nbytes += 2 * 8 * tokens + e * (min(1000, tokens) - tokens + s + h + n) * h
            flops += 2.0 * n * h * h
        return dict(bytes=nbytes, flops=flops)
    size = case["size"]
    if kind == "conv":
        k, out = case["kernel"], (size + 2 * case["pad"] - case["kernel"]) // case["stride"] + 1
        taps = case["cin"] * k * k * case["cout"]
        return dict(bytes=e * (n * case["cin"] * size * size + taps + n * case["cout"] * out * out), flops=2.0 * n * out * out * taps)
    if kind == "mbconv":
        c, m, r, px = case["cin"], 6 * case["cin"], max(1, case["cin"] // 4), n * size * size
        return dict(bytes=e * (2 * px * c + 2 * c * m + 9 * m + 2 * m * r), flops=2.0 * px * (2 * c * m + 9 * m) + 4.0 * n * m * r)
    c, m, out = case["cin"], case["cout"], (size - 1) // case["stride"] + 1
    taps = 9 * c * m + 9 * m * m + (c * m if case["stride"] != 1 or c != m else 0)
    return dict(bytes=e * (n * c * size * size + taps + n * m * out * out), flops=2.0 * n * out * out * taps)


def tolerance(case):
    """fp32 sums; fp16 tensors between the operators of a network (2^-11 for each rounding, a handful of them in a row,
    more for a deep stack of layers)."""
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}
    return {"rel": 2e-3 if case.get("layers", 1) <= 4 else 5e-3}
