"""The workloads whose speed is tracked: what the clients of this framework have it do, one request or one training step at
a time.

Convolutional clients run float32 networks of the ResNet / MobileNetV2 families: inference through
`torch_ops.prepare_inference`, training through `torch_ops.prepare_training` and `optim.SGD`.  Language-model clients run the
bfloat16 models of `benchmarking.benchmark_suite.transformer_trainer`: BERT question answering and the causal decoder,
inference with `orion=True`, training with `optim.AdamW`.

Training cases use fewer layers than the full networks, with every kind of layer of the family, so that the loss and the
gradients can be returned whole.
"""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F

from benchmarking.benchmark_suite.transformer_trainer import BERT, LM, BertQA, DecoderLM
from orion_b200 import optim, torch_ops

CLASSES = 1000
RESNET_BLOCKS = {14: (1, 1, 2, 1), 50: (3, 4, 6, 3), 101: (3, 4, 23, 3)}
# (expansion, channels, repeats, stride) of MobileNetV2; the training network keeps one block of the inner widths
MOBILENET_FULL = ((1, 16, 1, 1), (6, 24, 2, 2), (6, 32, 3, 2), (6, 64, 4, 2), (6, 96, 3, 1), (6, 160, 3, 2), (6, 320, 1, 1))
MOBILENET_TRAIN = ((1, 16, 1, 1), (6, 24, 1, 2), (6, 32, 1, 2), (6, 64, 1, 2), (6, 96, 1, 1), (6, 160, 1, 2))


class Bottleneck(nn.Module):
    def __init__(self, cin, width, stride):
        super().__init__()
        self.conv1, self.bn1 = nn.Conv2d(cin, width, 1, bias=False), nn.BatchNorm2d(width)
        self.conv2, self.bn2 = nn.Conv2d(width, width, 3, stride, 1, bias=False), nn.BatchNorm2d(width)
        self.conv3, self.bn3 = nn.Conv2d(width, 4 * width, 1, bias=False), nn.BatchNorm2d(4 * width)
        self.relu = nn.ReLU(inplace=True)
        self.downsample = None
        if stride != 1 or cin != 4 * width:
            self.downsample = nn.Sequential(nn.Conv2d(cin, 4 * width, 1, stride, bias=False), nn.BatchNorm2d(4 * width))

    def forward(self, x):
        identity = x if self.downsample is None else self.downsample(x)
        y = self.relu(self.bn1(self.conv1(x)))
        y = self.relu(self.bn2(self.conv2(y)))
        y = self.bn3(self.conv3(y))
        y += identity
        return self.relu(y)


class ResNet(nn.Module):
    def __init__(self, blocks):
        super().__init__()
        self.conv1, self.bn1 = nn.Conv2d(3, 64, 7, 2, 3, bias=False), nn.BatchNorm2d(64)
        self.relu, self.maxpool = nn.ReLU(inplace=True), nn.MaxPool2d(3, 2, 1)
        layers, cin = [], 64
        for stage, count in enumerate(blocks):
            for i in range(count):
                layers.append(Bottleneck(cin, 64 << stage, 2 if stage > 0 and i == 0 else 1))
                cin = 4 * (64 << stage)
        self.layers = nn.Sequential(*layers)
        self.avgpool, self.fc = nn.AdaptiveAvgPool2d((1, 1)), nn.Linear(cin, CLASSES)

    def forward(self, x):
        x = self.layers(self.maxpool(self.relu(self.bn1(self.conv1(x)))))
        return self.fc(torch.flatten(self.avgpool(x), 1))


def _conv_bn_relu6(cin, cout, k, stride=1, groups=1):
    return [nn.Conv2d(cin, cout, k, stride, (k - 1) // 2, groups=groups, bias=False), nn.BatchNorm2d(cout), nn.ReLU6(inplace=True)]


class InvertedResidual(nn.Module):
    def __init__(self, cin, cout, stride, expansion):
        super().__init__()
        mid = cin * expansion
        layers = _conv_bn_relu6(cin, mid, 1) if expansion != 1 else []
        layers += _conv_bn_relu6(mid, mid, 3, stride, mid) + [nn.Conv2d(mid, cout, 1, bias=False), nn.BatchNorm2d(cout)]
        self.conv, self.add = nn.Sequential(*layers), stride == 1 and cin == cout

    def forward(self, x):
        return x + self.conv(x) if self.add else self.conv(x)


class MobileNetV2(nn.Module):
    def __init__(self, settings):
        super().__init__()
        layers, cin = _conv_bn_relu6(3, 32, 3, 2), 32
        for t, c, n, s in settings:
            for i in range(n):
                layers.append(InvertedResidual(cin, c, s if i == 0 else 1, t))
                cin = c
        layers += _conv_bn_relu6(cin, 1280, 1)
        self.features = nn.Sequential(*layers)
        self.classifier = nn.Sequential(nn.Dropout(0.0), nn.Linear(1280, CLASSES))

    def forward(self, x):
        x = F.adaptive_avg_pool2d(self.features(x), (1, 1))
        return self.classifier(torch.flatten(x, 1))


def _network(case):
    if case["family"] == "resnet":
        return ResNet(RESNET_BLOCKS[case["depth"]])
    return MobileNetV2(MOBILENET_TRAIN if case["train"] else MOBILENET_FULL)


def _cnn(family, train, batch, image, depth=0):
    return {"kind": "cnn", "family": family, "train": train, "batch": batch, "image": image, "depth": depth}


def _text(model, train, batch, seq, layers):
    return {"kind": "text", "model": model, "train": train, "batch": batch, "seq": seq, "layers": layers}


def listed():
    return [
        # a single image through the smallest network: launches and latency
        dict(_cnn("mobilenet", False, 1, 224), name="mobilenet_infer_b1"),
        # the high-priority vision request
        dict(_cnn("resnet", False, 4, 224, depth=50), name="resnet50_infer_b4"),
        # a deeper network on a batch and an image size that divide nothing
        dict(_cnn("resnet", False, 7, 199, depth=101), name="resnet101_infer_b7_odd"),
        # the best-effort training clients' step
        dict(_cnn("resnet", True, 32, 224, depth=14), name="resnet_train_b32"),
        dict(_cnn("mobilenet", True, 64, 224), name="mobilenet_train_b64"),
        # fine-tuning on few small images
        dict(_cnn("resnet", True, 9, 145, depth=14), name="resnet_train_b9_odd"),
        # one short question, and the high-priority language request
        dict(_text("bert", False, 1, 77, 12), name="bert_infer_b1_s77"),
        dict(_text("bert", False, 8, 384, 12), name="bert_infer_b8_s384"),
        # scoring a batch of full-length sequences with the causal decoder
        dict(_text("lm", False, 16, 512, 16), name="lm_infer_b16_s512"),
        # the best-effort language training clients' step, and a small ragged one
        dict(_text("bert", True, 8, 384, 2), name="bert_train_b8_s384"),
        dict(_text("lm", True, 16, 512, 4), name="lm_train_b16_s512"),
        dict(_text("lm", True, 3, 200, 4), name="lm_train_b3_s200"),
    ]


def _between(rng, low, high):
    """A whole number from low to high, uniform over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.randrange(6)
    if kind == 0:
        return _cnn("resnet", False, _between(rng, 1, 8), _between(rng, 96, 256), depth=rng.choice((50, 101)))
    if kind == 1:
        return _cnn("mobilenet", False, _between(rng, 1, 8), _between(rng, 96, 256))
    if kind == 2:
        return _cnn("resnet", True, _between(rng, 4, 32), _between(rng, 64, 224), depth=14)
    if kind == 3:
        return _cnn("mobilenet", True, _between(rng, 4, 64), _between(rng, 64, 224))
    model = rng.choice(("bert", "lm"))
    seq = _between(rng, 16, 512)
    if kind == 4:
        # sequences beyond 384 keys come in multiples of 8
        return _text(model, False, _between(rng, 1, 16), seq if seq <= 384 else seq // 8 * 8, 12 if model == "bert" else 16)
    return _text(model, True, _between(rng, 1, 16), seq // 8 * 8, 2 if model == "bert" else 4)


def _zero_gradients(model):
    """For every parameter, whether its gradient is zero in exact arithmetic, so that what is computed is rounding error: a
    shift that the next batch norm takes out again (behind a linear bottleneck), or one that moves all the positions which a
    softmax compares alike (the last shift before the span logits)."""
    zero = set()
    for m in model.modules():
        if isinstance(m, InvertedResidual):
            zero.add(id(m.conv[-1].bias))
        elif isinstance(m, BertQA):
            zero.update((id(m.layers[-1].ln2.bias), id(m.qa.bias)))
    return [id(p) in zero for p in model.parameters()]


def _make(case, seed):
    """The plain model, inputs and targets of a case, on the GPU, from the seed alone."""
    torch.manual_seed(seed)
    b, y = case["batch"], None
    with torch.device("cuda"):
        if case["kind"] == "cnn":
            model = _network(case).to(memory_format=torch.channels_last)
            x = torch.randn(b, 3, case["image"], case["image"]).contiguous(memory_format=torch.channels_last)
            if case["train"]:
                y = torch.randint(0, CLASSES, (b,))
            else:
                for m in model.modules():
                    if isinstance(m, nn.BatchNorm2d):   # statistics and scales as a trained network has them
                        nn.init.uniform_(m.weight, 0.4, 1.0)
                        nn.init.normal_(m.bias, 0.0, 0.1)
                        m.running_mean.normal_(0.0, 0.2)
                        m.running_var.uniform_(0.5, 1.5)
        else:
            bert, s = case["model"] == "bert", case["seq"]
            cfg = dict(BERT if bert else LM, layers=case["layers"])
            model = (BertQA if bert else DecoderLM)(cfg).to(torch.bfloat16)
            x = torch.randint(0, 30522 if bert else cfg["vocab"], (b, s))
            if case["train"]:
                y = torch.randint(0, s, (2 * b,)) if bert else torch.randint(0, cfg["vocab"], (b * s,))
    return model.train(case["train"]), x, y


def prepare(case, seed):
    torch_ops.load()
    state = dict(case)
    model, state["x"], state["y"] = _make(case, seed)
    if case["train"]:
        state["params"], state["zero"] = list(model.parameters()), _zero_gradients(model)
    if case["kind"] == "text":
        state["model"] = model
        if case["train"]:
            state["opt"] = optim.AdamW(state["params"], lr=3e-5 if case["model"] == "bert" else 3e-4)
    elif case["train"]:
        state["model"], state["loss"] = torch_ops.prepare_training(model), nn.CrossEntropyLoss()
        state["opt"] = optim.SGD(state["params"], lr=0.01, momentum=0.9)
    else:
        state["model"] = torch_ops.prepare_inference(model)
    return state


def run(state):
    model, x = state["model"], state["x"]
    if not state["train"]:
        with torch.no_grad():
            return model(x) if state["kind"] == "cnn" else model(x, orion=True)
    opt = state["opt"]
    opt.zero_grad()
    if state["kind"] == "cnn":
        loss = state["loss"](model(x), state["y"])
        loss.backward()
    else:
        if state["model"].__class__ is BertQA:
            loss = 2.0 * torch.ops.orion.cross_entropy(model.span_logits(x).view(-1, state["seq"]), state["y"])
        else:
            logits = model(x)
            loss = torch.ops.orion.cross_entropy(logits.reshape(-1, logits.shape[-1]), state["y"])
        loss.backward()
    opt.step()
    params = state["params"]
    out = {"loss": loss.detach(), "grads": [p.grad for p, z in zip(params, state["zero"]) if not z]}
    if 2 * len(params) + 1 <= 64:
        out["weights"] = [p.detach() for p in params]
    return out


def _conv_layers(case):
    """(multiply-adds, input elements, output elements, filter elements) of every convolution and of the classifier."""
    with torch.device("meta"):
        model = _network(case)
        x = torch.empty(case["batch"], 3, case["image"], case["image"])
    rows = []

    def note(m, args, out):
        rows.append((out.numel() * (m.weight.numel() // m.weight.shape[0]), args[0].numel(), out.numel(), m.weight.numel()))

    for m in model.modules():
        if isinstance(m, (nn.Conv2d, nn.Linear)):
            m.register_forward_hook(note)
    model.eval()(x)
    return rows


def work(case):
    if case["kind"] == "cnn":
        rows = _conv_layers(case)
        macs, weights = sum(r[0] for r in rows), sum(r[3] for r in rows)
        if not case["train"]:
            return {"bytes": 4.0 * (rows[0][1] + weights + rows[-1][2]), "flops": 2.0 * macs}
        # backward: two products per convolution, none for the image; the input and the output of every convolution are kept
        # for it (written once, read once); weights and momentum are read and written, gradients written
        kept = sum(r[1] + r[2] for r in rows)
        return {"bytes": 4.0 * (rows[0][1] + 2 * kept + 5 * weights), "flops": 2.0 * (3 * macs - rows[0][0])}
    bert = case["model"] == "bert"
    cfg = BERT if bert else LM
    h, ffn, b, s, layers = cfg["hidden"], cfg["ffn"], case["batch"], case["seq"], case["layers"]
    tokens, per_layer = b * s, 4 * h * h + 2 * h * ffn
    head = 2 * h if bert else cfg["vocab"] * h
    pairs = b * (s * s if bert else s * (s + 1) // 2)   # query / key pairs that count
    flops = 2.0 * tokens * (layers * per_layer + head) + 4.0 * pairs * h * layers
    logits = tokens * (2 if bert else cfg["vocab"])
    table = cfg["vocab"] * h
    if not case["train"]:
        rows_read = min(tokens, cfg["vocab"])
        return {"bytes": 2.0 * (layers * per_layer + head + rows_read * h + logits), "flops": flops}
    # weights and both moments are read and written, gradients written; logits are kept from forward to backward
    return {"bytes": 2.0 * (7 * (layers * per_layer + head + table) + 2 * logits), "flops": 3.0 * flops}


def _text_exact(model, x, causal):
    """The logits, from the weights of a float64 copy of a language model."""
    p = dict(model.named_parameters())
    heads, s = model.layers[0].heads, x.shape[1]

    def linear(h, name):
        return F.linear(h, p[name + ".weight"], p[name + ".bias"])

    def norm(h, name, eps):
        return F.layer_norm(h, h.shape[-1:], p[name + ".weight"], p[name + ".bias"], eps)

    h = p["word.weight"][x] + p["pos.weight"][:s]
    if not causal:
        h = norm(h + p["typ.weight"][0], "ln", 1e-12)
    future = torch.ones(s, s, dtype=torch.bool, device=x.device).triu(1)
    for i in range(len(model.layers)):
        n = "layers.%d." % i
        q, k, v = linear(h, n + "qkv").view(*x.shape, 3, heads, -1).permute(2, 0, 3, 1, 4)
        scores = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
        if causal:
            scores = scores.masked_fill(future, -math.inf)
        context = (scores.softmax(-1) @ v).transpose(1, 2).flatten(2)
        h = norm(h + linear(context, n + "out"), n + "ln1", 1e-12)
        h = norm(h + linear(F.gelu(linear(h, n + "fc1")), n + "fc2"), n + "ln2", 1e-12)
    if causal:
        return F.linear(norm(h, "ln", 1e-5), p["head.weight"])
    return linear(h, "qa")


def exact(case, seed):
    model, x, y = _make(case, seed)
    zero = _zero_gradients(model)
    model = model.double()
    with torch.set_grad_enabled(case["train"]):
        if case["kind"] == "cnn":
            logits = model(x.double())
        else:
            logits = _text_exact(model, x, case["model"] == "lm")
    if not case["train"]:
        return logits
    if case["kind"] == "cnn":
        loss = F.cross_entropy(logits, y)
    elif case["model"] == "bert":
        loss = 2.0 * F.cross_entropy(logits.permute(2, 0, 1).reshape(-1, case["seq"]), y)
    else:
        loss = F.cross_entropy(logits.flatten(0, 1), y)
    loss.backward()
    params, text = list(model.parameters()), case["kind"] == "text"
    # In BERT, the gradient of the shift before the last norm cancels over the positions almost as far as the gradients that are
    # left out, and bfloat16 leaves it 0.16 off.
    poor = id(model.layers[-1].fc2.bias) if text and case["model"] == "bert" else None
    out = {"loss": loss.detach(), "grads": [None if id(p) == poor else p.grad for p, z in zip(params, zero) if not z]}
    if 2 * len(params) + 1 <= 64:
        # the first step of AdamW moves a weight by the sign of its gradient, and a vector that starts at zero is that alone
        lr = (3e-5 if case["model"] == "bert" else 3e-4) if text else 0.01
        out["weights"] = []
        for p in params:
            if text:
                new = p.detach() * (1 - lr * 1e-2) - lr * p.grad / (p.grad.abs() + 1e-8) if p.dim() > 1 and p.grad is not None else None
            else:
                new = p.detach() - lr * p.grad
            out["weights"].append(new)
    return out


def tolerance(case):
    """About four times the distance that was measured to the same network in higher precision or on the stock kernels."""
    if case["kind"] == "cnn" and not case["train"]:
        return {"rel": 1e-5, "max": 4e-5}   # logits against float64: 4e-7 to 1.9e-6, 5e-6 in one value
    # Float32 convolutional gradients against float64: 4e-3 to 1.1e-2, because a handful of pre-activations within rounding
    # distance of the ReLU kink fall on the other side (the stock kernels show the same).  bfloat16 logits 1e-2, gradients 7e-3
    # (decoder) to 2.7e-2 (BERT, whose span loss cancels over the positions) between two sets of kernels.
    return {"rel": 3e-2, "max": 0.9 if case["train"] else 0.3}
