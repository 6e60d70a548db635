"""The workloads this backend is timed on: forward passes of the configurations' models and of
the tensor-op micrograph, each through the public call that a program of its kind makes.

A case names the graph (`family` and its sizes), how the data reaches it (`io`) and the GEMM
option of the session (`gemm_mode`):

    io = "host"    `InferenceSession(model).run(None, {...})`: pageable numpy arrays in, new
                   arrays out -- the call of a script or of a request handler
    io = "pinned"  `CudaSession.run(inputs, outputs)` on page-locked buffers that are kept -- the
                   synchronous loop of a server
    io = "queue"   `CudaSession.run_batches` over a queue of page-locked batches -- bulk work
    io = "device"  `CudaSession.run_device` on tensors already on the GPU -- one stage of a
                   pipeline of GPU programs
    gemm_mode 0    the default products; 3 the full-range (3xTF32) products, for models whose
                   activations leave the default's range

Weights are the seeded ones of `altius_b200.configs` and the same for every seed of a case, as
a program keeps its model; the seed makes the inputs (normalised images, uniform digits, normal
activations and attention scores).
"""
import functools
import math

import numpy as np
import torch

from altius_b200 import configs
from altius_b200.session import CudaSessionBuilder, InferenceSession


# ---- cases --------------------------------------------------------------------------------------
def _mnist(name):
    return dict(name=name, family="mnist", batch=1, io="host", gemm_mode=0)


def _mobilenet(name, batch, px, io):
    return dict(name=name, family="mobilenet", batch=batch, px=px, io=io, gemm_mode=0)


def _encoder(name, batch, px, dim, depth, prefix, io, gemm_mode=0, queue=1):
    """A ViT (one prefix token) or distilled DeiT (two): heads of 64, MLP of 4 x dim, patches of 16."""
    return dict(name=name, family="encoder", batch=batch, px=px, dim=dim, depth=depth, prefix=prefix, io=io,
                gemm_mode=gemm_mode, queue=queue)


def _micrograph(name, batch, tokens, dim, heads):
    return dict(name=name, family="micrograph", batch=batch, tokens=tokens, dim=dim, heads=heads, io="device",
                gemm_mode=0)


_LARGEST = dict(batch=96, px=224, dim=768, depth=12, prefix=1)


def listed():
    return [
        # One digit at a time: a graph of microseconds, all latency and host path.
        _mnist("mnist_b1"),
        # One photo per request, the small convolutional model.
        _mobilenet("mobilenet_b1", 1, 224, "host"),
        # Crops of a detector, collected on the GPU: a ragged batch of smaller planes.
        _mobilenet("mobilenet_b13_px192", 13, 192, "device"),
        # A script that classifies a folder of photos batch by batch.
        _mobilenet("mobilenet_b32", 32, 224, "host"),
        # One photo per request, the transformer.
        _encoder("vit_b1", 1, 224, 768, 12, 1, "host"),
        # A server's synchronous loop at the batch the throughput metric is quoted on.
        _encoder("vit_b32", 32, 224, 768, 12, 1, "pinned"),
        # Bulk scoring: a queue of batches, copies under compute.
        _encoder("vit_queue_4xb16", 16, 224, 768, 12, 1, "queue", queue=4),
        # Fine-tuned at a higher resolution (577 tokens), a few images from a GPU pipeline.
        _encoder("vit_b5_px384", 5, 384, 768, 12, 1, "device"),
        # A large offline batch from a GPU pipeline.
        _encoder("vit_b96", io="device", **_LARGEST),
        # The distilled small model at its batch of 64, from a script's arrays.
        _encoder("deit_b64", 64, 224, 384, 12, 2, "host"),
        # The same model on the full-range products, an odd small batch.
        _encoder("deit_b7_wide", 7, 224, 384, 12, 2, "pinned", gemm_mode=3),
        # The tensor-op micrograph of a ViT layer's memory-bound operators.
        _micrograph("micrograph_b64", 64, 197, 768, 12),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    family = rng.choice(["mobilenet", "mobilenet", "encoder", "encoder", "encoder", "encoder", "micrograph"])
    if family == "mobilenet":
        px = rng.choice([160, 192, 224, 224, rng.randint(96, 256)])
        case = _mobilenet(None, _log_int(rng, 1, int(64 * min(1.0, (224 / px) ** 2))), px, rng.choice(["host", "pinned", "device"]))
    elif family == "encoder":
        px = 16 * rng.choice([14, 14, 14, rng.randint(6, 24)])
        dim, prefix = rng.choice([192, 384, 384, 512, 768, 768]), rng.choice([1, 1, 2])
        depth = 12 if rng.random() < 0.6 else rng.randint(2, 12)
        mode = 3 if rng.random() < 0.15 else 0
        io = rng.choice(["host", "pinned", "queue", "device"])
        # at most half of the largest listed case's operations, over all batches of a queue
        case = _encoder(None, 1, px, dim, depth, prefix, io, mode, rng.randint(2, 6) if io == "queue" else 1)
        most = int(0.5 * work(dict(_encoder(None, io="device", **_LARGEST)))["flops"] / work(case)["flops"])
        case["batch"] = _log_int(rng, 1, min(96, most))
    else:
        tokens, heads = rng.randint(17, 256), rng.choice([3, 4, 6, 8, 12, 16])
        dim = 64 * heads if rng.random() < 0.7 else rng.randint(64, 1024)
        case = _micrograph(None, _log_int(rng, 1, 96), tokens, dim, heads)
    del case["name"]
    return case


# ---- what a program has in hand --------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _model(family, sizes):
    sizes = dict(sizes)
    if family == "mnist":
        return configs.mnist_cnn()[0]
    if family == "mobilenet":
        return configs.mobilenet_v3_large(batch=sizes["batch"], img=sizes["px"])[0]
    if family == "encoder":
        dim = sizes["dim"]
        return configs.vision_transformer(sizes["batch"], dim, sizes["depth"], dim // 64, 4 * dim, sizes["prefix"],
                                          img=sizes["px"])[0]
    return configs.micrograph(sizes["batch"], sizes["tokens"], sizes["dim"], sizes["heads"])[0]


def prepare(case, seed):
    sizes = {k: case[k] for k in ("batch", "px", "dim", "depth", "prefix", "tokens", "heads") if k in case}
    model = _model(case["family"], tuple(sorted(sizes.items())))
    if case["io"] == "host" and case["gemm_mode"] == 0:
        session = InferenceSession(model, backend="cuda")
        plain = session.session
    else:
        session = plain = CudaSessionBuilder(model).with_gemm_mode(case["gemm_mode"]).build()
    gen = torch.Generator("cuda").manual_seed(seed)
    fill = torch.rand if case["family"] == "mnist" else torch.randn
    batches = [[fill(shape, generator=gen, device="cuda") for shape, _ in plain.input_info]
               for _ in range(case.get("queue", 1))]
    state = dict(io=case["io"], session=session)
    if case["io"] == "device":
        outs = [torch.empty(shape, device="cuda") for shape, _ in plain.output_info]
        state.update(inputs=batches[0], outputs=outs, in_ptrs=[t.data_ptr() for t in batches[0]],
                     out_ptrs=[t.data_ptr() for t in outs])
        torch.cuda.synchronize()   # the session works on a stream of its own
    elif case["io"] == "host":
        arrays = [t.cpu().numpy() for t in batches[0]]
        names = [model.graph.values[v].name for v in plain.input_ids]
        state.update(inputs=dict(zip(names, arrays)) if plain is not session else arrays)
    else:
        state["tensors"] = [[t.cpu().pin_memory() for t in row] for row in batches]
        state["results"] = [[torch.empty(shape).pin_memory() for shape, _ in plain.output_info] for _ in batches]
        state["inputs"] = [[t.numpy() for t in row] for row in state["tensors"]]
        state["outputs"] = [[t.numpy() for t in row] for row in state["results"]]
    return state


def run(state):
    session, io = state["session"], state["io"]
    if io == "device":
        session.run_device(state["in_ptrs"], state["out_ptrs"])
        return state["outputs"]
    if io == "queue":
        return session.run_batches(state["inputs"], state["outputs"])
    if io == "pinned":
        return session.run(state["inputs"][0], state["outputs"][0])
    if isinstance(session, InferenceSession):
        return session.run(None, state["inputs"])
    return session.run(state["inputs"])


# ---- what the path cannot do without ---------------------------------------------------------------
def _conv_net_work(model):
    """(operations, elements of the result) of a graph whose products are Conv2d, MatMul and Gemm nodes
    with constant weights; every other node keeps the shape of its first input or pools it."""
    g = model.graph
    shape = {v: g.values[v].shape for v in list(g.inputs) + list(g.inits)}
    flops = 0
    for node in g.nodes:
        s = shape[node.inputs[0]]
        if node.op in ("Conv2d", "MaxPool"):
            k, st = node.attrs["kernel_shape"], node.attrs["strides"]
            p = node.attrs["padding"] or [0, 0, 0, 0]
            if node.attrs["auto_pad"] == "SAME_UPPER":
                hw = [-(-s[2 + i] // st[i]) for i in (0, 1)]
            else:
                hw = [(s[2 + i] + p[i] + p[2 + i] - k[i]) // st[i] + 1 for i in (0, 1)]
            c = s[1]
            if node.op == "Conv2d":
                w = shape[node.inputs[1]]
                c = w[0]
                flops += 2 * s[0] * c * hw[0] * hw[1] * w[1] * w[2] * w[3]
            s = (s[0], c, *hw)
        elif node.op == "GlobalAveragePool":
            s = (s[0], s[1], 1, 1)
        elif node.op == "Flatten":
            s = (s[0], math.prod(s[1:]))
        elif node.op == "Reshape":
            s = tuple(int(d) for d in g.inits[node.inputs[1]])
        elif node.op in ("MatMul", "Gemm"):
            w = shape[node.inputs[1]]
            flops += 2 * s[0] * w[0] * w[1]
            s = (s[0], w[0] if node.attrs.get("trans_b") else w[1])
        shape[node.outputs[0]] = s
    return flops, math.prod(shape[g.outputs[0]])


def work(case):
    B = case["batch"]
    if case["family"] == "encoder":
        D, L, P, N = case["dim"], case["depth"], case["prefix"], case["queue"]
        patches = (case["px"] // 16) ** 2
        T = patches + P
        per_image = 2 * patches * 768 * D + 2 * P * D * 1000 + L * (24 * T * D * D + 4 * T * T * D)
        params = 769 * D + (P + T) * D + L * (12 * D * D + 13 * D) + 2 * D + P * 1000 * (D + 1)
        return dict(bytes=4 * (params + N * B * (3 * case["px"] ** 2 + 1000)), flops=N * B * per_image)
    if case["family"] == "micrograph":
        rows, scores = B * case["tokens"], B * case["heads"] * case["tokens"] ** 2
        # Gelu ~25 and LayerNormalization ~8 operations an element, the two reductions 2; Softmax ~20
        return dict(bytes=4 * (rows * (2 * case["dim"] + 2) + 2 * scores + 3 * case["dim"]),
                    flops=35 * rows * case["dim"] + 20 * scores)
    sizes = {k: case[k] for k in ("batch", "px") if k in case}
    model = _model(case["family"], tuple(sorted(sizes.items())))
    flops, results = _conv_net_work(model)
    params = sum(a.size for a in model.graph.inits.values() if a.dtype == np.float32)
    return dict(bytes=4 * (params + math.prod(model.graph.values[model.graph.inputs[0]].shape) + results), flops=flops)


def tolerance(case):
    """fp32 throughout: one operator deep 1e-5; a model's chain of products and normalisations adds
    the rounding of its layers up, each about 1e-6 to 1e-5 of its result."""
    return {"rel": 1e-5 if case["family"] in ("micrograph", "mnist") else 5e-5}
