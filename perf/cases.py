"""Performance cases of the inference server: what its users have it do, as calls of its public entry points.

A case is one request to a loaded model (or one real-time request and the best-effort requests beside it): the input
goes in from host memory, the model runs, the output comes back to host memory.  ``api`` says through which entry
points:

``rt``       REEFScheduler in REEF mode, the model on the real-time queue; with ``be_clients`` > 0 that many best-effort
             requests of ``be_model`` are queued first, each on a queue of its own, and the pass ends when all are served
``be``       the same with the model on a best-effort queue and nothing on the real-time queue
``graph``    HybridExecutor.execute_graph (an embedding program that drives one model itself)
``execute``  HybridExecutor.execute, the kernel-by-kernel form

``listed()`` are the cases to look at first, ``draw(rng)`` gives more of the same ranges: every model family of the
generator, images of 64 to 320 pixels, 8 to 512 tokens, the TF32 schedules and the exact-fp32 ones.
"""
import hashlib
import os
import tempfile

import numpy as np

from reef_b200 import capi, resources

_RESNET = {"resnet18": (False, [2, 2, 2, 2], [64, 128, 256, 512]),
           "resnet50": (True, [3, 4, 6, 3], [256, 512, 1024, 2048]),
           "resnet152": (True, [3, 8, 36, 3], [256, 512, 1024, 2048])}
_BERT = {"bert_base": dict(layers=12, hidden=768, heads=12, ffn=3072, vocab=30522),
         "bert_small": dict(layers=2, hidden=128, heads=2, ffn=256, vocab=1000)}
_SMALLEST_IMAGE = {"inception_v3": 139, "densenet201": 64, "vgg16": 64}


def _case(name, model, size, api, *, fp32=False, be_model="", be_size=0, be_clients=0):
    """``size``: image edge in pixels, or tokens for the BERT models."""
    return dict(name=name, model=model, size=size, api=api, fp32=fp32, be_model=be_model, be_size=be_size,
                be_clients=be_clients)


def listed():
    return [
        # the smallest call: a two-layer encoder run kernel by kernel, where every launch and every copy shows
        _case("encoder_small_48", "bert_small", 48, "execute"),
        # a thumbnail classifier: a request too small to fill the GPU in any layer
        _case("resnet18_64_rt", "resnet18", 64, "rt"),
        # the ordinary real-time request, no contention: small and large network
        _case("resnet18_224_rt", "resnet18", 224, "rt"),
        _case("resnet152_224_rt", "resnet152", 224, "rt"),
        # branches, 1x7 / 7x1 filters, odd extents (149, 147, 73, 71, 35, 17, 8)
        _case("inception_v3_299_rt", "inception_v3", 299, "rt"),
        # text: one 128-token window, and a long passage
        _case("bert_base_128_rt", "bert_base", 128, "rt"),
        _case("bert_base_384_rt", "bert_base", 384, "rt"),
        # best-effort requests with the GPU to themselves: the most weights and arithmetic of the image models, and the
        # most kernels
        _case("vgg16_224_be", "vgg16", 224, "be"),
        _case("densenet201_224_be", "densenet201", 224, "be"),
        # the exact-fp32 schedule, for users who cannot take TF32, on an image size that divides nothing
        _case("resnet50_193_fp32", "resnet50", 193, "graph", fp32=True),
        # real-time requests that meet best-effort work: preemption, padding and resumption
        _case("resnet152_rt_over_4_be", "resnet152", 224, "rt", be_model="resnet152", be_size=224, be_clients=4),
        _case("bert_base_77_rt_over_4_be", "bert_base", 77, "rt", be_model="resnet50", be_size=224, be_clients=4),
    ]


def _draw_size(rng, model, top):
    if model in _BERT:
        return int(round(8 * (512 / 8) ** rng.random()))
    return rng.randint(_SMALLEST_IMAGE.get(model, 64), top)


def draw(rng):
    model = rng.choice(["resnet18", "resnet50", "resnet152", "inception_v3", "vgg16", "densenet201", "bert_base", "bert_base",
                        "bert_small"])
    fp32 = model in ("resnet18", "resnet50") and rng.random() < 0.4
    api = rng.choice(["rt", "rt", "be", "graph", "execute"])
    case = _case("", model, _draw_size(rng, model, 224 if fp32 else 320), api, fp32=fp32)
    del case["name"]
    if api == "rt" and not fp32 and rng.random() < 0.4:
        case["be_model"] = rng.choice(["resnet18", "resnet50", "densenet201"])
        case["be_size"] = _draw_size(rng, case["be_model"], 224)
        case["be_clients"] = rng.randint(1, 4)
    return case


def _files(model, size, fp32):
    """Path prefix of the model's resources, generated on first use.  The folder is this user's and this tree's own."""
    here = hashlib.sha1(os.getcwd().encode()).hexdigest()[:12]
    root = os.path.join(tempfile.gettempdir(), "reef_cases_%d_%s" % (os.getuid(), here), "%s_%d" % (model, size))
    kind, kw = ("bert_base", dict(_BERT[model], seq=size)) if model in _BERT else (model, dict(image=size))
    d = resources.generate(kind, root, variant="_fp32" if fp32 else "", **kw)
    return os.path.join(d, os.path.basename(d))


def _input(model, size, rng):
    """(storage name, request) on the host: an image ~ N(0, 1), or token ids."""
    if model in _BERT:
        return "input0", rng.integers(0, _BERT[model]["vocab"], size).astype(np.int64)
    return "data", rng.standard_normal(3 * size * size, dtype=np.float32)


class _Executor:
    """One model driven by the program itself."""

    def __init__(self, case, seed):
        base = _files(case["model"], case["size"], case["fp32"])
        self.exe = capi.HybridExecutor(0)
        self.exe.load_model_from_file(base + ".json", base + ".profile.json")
        self.exe.load_param_from_file(base + ".param")
        self.name, self.x = _input(case["model"], case["size"], np.random.default_rng(seed))
        self.go = self.exe.execute_graph if case["api"] == "graph" else self.exe.execute

    def run(self):
        self.exe.set_input(self.name, self.x)
        self.go()
        return self.exe.get_output()


class _Server:
    """A scheduler with its clients: the case's own model, and the best-effort ones beside it."""

    def __init__(self, case, seed):
        self.sched = capi.REEFScheduler(capi.REEFScheduler.REEF, 0)
        rng = np.random.default_rng(seed)
        own = capi.REEFScheduler.RealTimeQueue if case["api"] == "rt" else capi.REEFScheduler.BestEffortQueue
        want = [(case["be_model"], case["be_size"], False, capi.REEFScheduler.BestEffortQueue)] * case["be_clients"]
        self.clients = []
        for model, size, fp32, kind in want + [(case["model"], case["size"], case["fp32"], own)]:
            base = _files(model, size, fp32)
            mid = self.sched.load_model_files(base + ".json", base + ".profile.json", base + ".param")
            self.sched.bind_model_queue(self.sched.create_queue(kind), mid)
            self.clients.append((mid,) + _input(model, size, rng))
        self.sched.run()

    def run(self):
        for mid, name, x in self.clients:
            self.sched.set_input(mid, x, name)
        tasks = [self.sched.new_task(mid) for mid, _, _ in self.clients]    # the case's own request comes last
        for tid in reversed(tasks):
            self.sched.wait_task(tid)
        return [self.sched.get_output(mid) for mid, _, _ in self.clients]

    def __del__(self):
        self.sched.close()


def prepare(case, seed):
    return (_Server if case["api"] in ("rt", "be") else _Executor)(case, seed)


def run(state):
    return state.run()


def _resnet(model, h):
    bottleneck, units, widths = _RESNET[model]
    h = (h - 1) // 2 + 1
    yield 64, 3 * 49, h * h
    h = (h - 1) // 2 + 1
    ci = 64
    for stage, (n, co) in enumerate(zip(units, widths)):
        for unit in range(n):
            if unit == 0 and stage > 0:
                h = (h - 1) // 2 + 1
            if unit == 0:
                yield co, ci, h * h
            mid = co // 4
            yield from [(mid, ci, h * h), (mid, 9 * mid, h * h), (co, mid, h * h)] if bottleneck else \
                [(co, 9 * ci, h * h), (co, 9 * co, h * h)]
            ci = co
    yield 1000, ci, 1


def _vgg16(h):
    ci = 3
    for co, n in ((64, 2), (128, 2), (256, 3), (512, 3), (512, 3)):
        for _ in range(n):
            yield co, 9 * ci, h * h
            ci = co
        h //= 2
    for co, k in ((4096, 512 * h * h), (4096, 4096), (1000, 4096)):
        yield co, k, 1


def _densenet201(h):
    h = (h - 1) // 2 + 1
    yield 64, 3 * 49, h * h
    h = (h - 1) // 2 + 1
    c = 64
    for block, n in enumerate((6, 12, 48, 32)):
        for _ in range(n):
            yield 128, c, h * h
            yield 32, 9 * 128, h * h
            c += 32
        if block < 3:
            c //= 2
            yield c, 2 * c, h * h
            h //= 2
    yield 1000, c, 1


def _inception_v3(h):
    half = lambda v: (v - 3) // 2 + 1     # 3x3 / 2 without padding   # noqa: E731
    h = half(h)
    yield 32, 27, h * h
    yield 32, 9 * 32, (h - 2) ** 2
    yield 64, 9 * 32, (h - 2) ** 2
    h = half(h - 2)
    yield 80, 64, h * h
    yield 192, 9 * 80, (h - 2) ** 2
    h = half(h - 2)
    c = 192
    for pool in (32, 64, 64):
        for co, k in ((64, c), (48, c), (64, 25 * 48), (64, c), (96, 9 * 64), (96, 9 * 96), (pool, c)):
            yield co, k, h * h
        c = 224 + pool
    yield 64, c, h * h
    yield 96, 9 * 64, h * h
    h = half(h)
    yield 384, 9 * c, h * h
    yield 96, 9 * 96, h * h
    for m in (128, 160, 160, 192):
        for co, k in ((192, 768), (m, 768), (m, 7 * m), (192, 7 * m), (m, 768), (m, 7 * m), (m, 7 * m), (m, 7 * m), (192, 7 * m),
                      (192, 768)):
            yield co, k, h * h
    for co, k in ((192, 768), (192, 768), (192, 7 * 192), (192, 7 * 192)):
        yield co, k, h * h
    h = half(h)
    yield 320, 9 * 192, h * h
    yield 192, 9 * 192, h * h
    for c in (1280, 2048):
        for co, k in ((320, c), (384, c), (384, 3 * 384), (384, 3 * 384), (448, c), (384, 9 * 448), (384, 3 * 384), (384, 3 * 384),
                      (192, c)):
            yield co, k, h * h
    yield 1000, 2048, 1


def _work(model, size):
    """(bytes, flops) of one request: weights, request and answer once each; multiply-adds of the layers."""
    if model in _BERT:
        b = _BERT[model]
        H, per_layer = b["hidden"], 4 * b["hidden"] ** 2 + 2 * b["hidden"] * b["ffn"]
        weights = b["layers"] * (per_layer + 9 * H + b["ffn"]) + 2 * size * H     # + the embedding rows of the tokens
        return 4.0 * (weights + size * H) + 8.0 * size, 2.0 * size * b["layers"] * (per_layer + 2 * size * H)
    layers = list(_resnet(model, size) if model in _RESNET else
                  dict(vgg16=_vgg16, densenet201=_densenet201, inception_v3=_inception_v3)[model](size))
    return (4.0 * (sum(co * k for co, k, _ in layers) + 3 * size * size + 1000),
            2.0 * sum(co * k * pixels for co, k, pixels in layers))


def work(case):
    nbytes, flops = _work(case["model"], case["size"])
    if case["be_clients"]:
        be_bytes, be_flops = _work(case["be_model"], case["be_size"])
        nbytes, flops = nbytes + case["be_clients"] * be_bytes, flops + case["be_clients"] * be_flops
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # fp32 schedules: sums in another order, through 50 layers and a softmax.  The others multiply TF32 operands (10
    # mantissa bits, 5e-4 each) and store TF32 activations from layer to layer.
    return {"rel": 5e-5} if case["fp32"] else {"rel": 5e-3}
