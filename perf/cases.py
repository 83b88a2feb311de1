"""Workloads the W4A4 linear is timed on, through the package's public entry points.

A case is a dict of plain values.  ``listed()`` gives the standing ones, ``draw(rng)`` one more from
the same ranges; ``prepare`` makes what a serving program has in hand before the call (weights on the
GPU, activations, a captured graph where such a program keeps one), ``run`` is one pass, ``work`` the
bytes and operations a pass cannot do without and ``tolerance`` how far another correct
implementation may be.  Everything is made from the seed on the GPU.

Four kinds of call:

* ``linear``    - ``v9_linear_forward`` issued eagerly: fp16 activations in, fp16 ``(T, d_out)`` out;
* ``operators`` - the operator layer: ``activation_quant_cuda`` then ``fused_dense_sparse_cuda_int4``
  with its ``(d_out, T)`` result;
* ``cached``    - ``v9_linear_forward_cuda_graph`` under the ``auto`` policy (few tokens, one weight);
* ``layer``     - the four linears of a decoder layer (qkv and gate/up behind an RMSNorm, o, down behind
  SiLU * up), as one captured graph for a decode step or eagerly for a prompt.  Attention, rotary
  embedding and residual adds are other libraries' work and left out, so each linear has an input of
  its own.
"""

import torch

from zip_kernel_b200 import _lib, v9_linear
from zip_kernel_b200.backend import graph_cache
from zip_kernel_b200.ops import activation_quant_cuda, fused_dense_sparse_cuda_int4
from zip_kernel_b200.pack_utils import BCOL, BROW, V9WeightContainer

EPS = 1e-5
MAX_TOKENS = 8192

# (d_in, d_out) of the Llama-3-8B and Llama-2-70B linears with fused qkv and gate/up projections
SHAPES = [(4096, 6144), (4096, 4096), (4096, 28672), (14336, 4096),
          (8192, 10240), (8192, 8192), (8192, 57344), (28672, 8192)]
# (hidden, d_out of qkv, ffn) of the two decoders
LAYERS = [(4096, 6144, 14336), (8192, 10240, 28672)]


def _linear(name, kind, tokens, d_in, d_out, density=0.05, prepared=False, permuted=True):
    return {"name": name, "kind": kind, "tokens": tokens, "d_in": d_in, "d_out": d_out, "density": density,
            "prepared": prepared, "permuted": permuted}


def _layer(name, tokens, hidden, qkv, ffn, graph, density=0.05, prepared=False, permuted=False):
    return {"name": name, "kind": "layer", "tokens": tokens, "hidden": hidden, "qkv": qkv, "ffn": ffn, "graph": graph,
            "density": density, "prepared": prepared, "permuted": permuted}


def listed():
    return [
        # one token, the smallest linear of the 8B model, eager: what a program without graphs pays per call
        _linear("eager_1_token", "linear", 1, 4096, 4096),
        # a small batch through the operator surface (quantise once, then the fused GEMM, (d_out, T) result)
        _linear("operators_8_tokens", "operators", 8, 4096, 6144),
        # a decode batch through the per-weight graph cache
        _linear("graph_cache_16_tokens", "cached", 16, 4096, 28672),
        # one decode step of an 8B layer for a single user, and for a batch of 32
        _layer("decode_8b_1_token", 1, 4096, 6144, 14336, True),
        _layer("decode_8b_32_tokens", 32, 4096, 6144, 14336, True),
        # the same for one user of the 70B model: weights far beyond L2
        _layer("decode_70b_1_token", 1, 8192, 10240, 28672, True),
        # a mixed batch between decode and prompt sizes, no multiple of any tile
        _linear("mixed_batch_100_tokens", "linear", 100, 4096, 6144),
        # a prompt chunk against the deep down projection
        _linear("chunk_512_tokens", "linear", 512, 14336, 4096, prepared=True),
        # a prompt on packed weights only (no load-time preparation)
        _linear("prompt_2048_packed", "linear", 2048, 4096, 28672),
        # odd everything: ragged tokens and rows, a group count no power of two, no residual blocks
        _linear("prompt_1537_ragged", "linear", 1537, 2944, 5000, density=0.0),
        # prompt processing of a layer with its fused prologues on prepared weights
        _layer("prompt_layer_2048", 2048, 4096, 6144, 14336, False, prepared=True),
        # the longest prompt and the densest residual
        _linear("prompt_8192_dense_residual", "linear", 8192, 4096, 28672, density=0.15, prepared=True),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "operators", "cached", "layer", "layer"])
    density = rng.choice([0.0, 0.05, 0.05, 0.15])
    permuted = rng.random() < 0.5
    limit = 0.5 * 8192 * 4096 * 28672            # tokens x d_in x d_out: half the largest listed case
    if kind == "layer":
        if rng.random() < 0.5:
            hidden, qkv, ffn = rng.choice(LAYERS)
        else:
            hidden = BCOL * rng.randint(12, 64)
            qkv, ffn = hidden + 256 * rng.randint(1, hidden // 128), BCOL * rng.randint(hidden // 64, 7 * hidden // 256)
        graph = rng.random() < 0.6
        tokens = _log_int(rng, 1, 64) if graph else _log_int(rng, 64, 2048)
        while tokens * hidden * (qkv + hidden + 3 * ffn) > limit:
            tokens = tokens * 3 // 4
        c = _layer("", tokens, hidden, qkv, ffn, graph, density, not graph and rng.random() < 0.7, permuted)
    else:
        if rng.random() < 0.6:
            d_in, d_out = rng.choice(SHAPES)
        else:
            d_in, d_out = BCOL * _log_int(rng, 8, 128), _log_int(rng, 1000, 20000)
        tokens = {"linear": _log_int(rng, 1, MAX_TOKENS), "operators": _log_int(rng, 1, 2048),
                  "cached": 2 ** rng.randint(0, 6)}[kind]
        while tokens * d_in * d_out > limit:
            tokens = tokens * 3 // 4
        c = _linear("", kind, tokens, d_in, d_out, density, kind == "linear" and tokens >= 64 and rng.random() < 0.5, permuted)
    del c["name"]
    return c


def _linears(case):
    """(d_in, d_out) of the linears of a case."""
    if case["kind"] == "layer":
        h, f = case["hidden"], case["ffn"]
        return [(h, case["qkv"]), (h, h), (h, 2 * f), (f, h)]
    return [(case["d_in"], case["d_out"])]


def _container(gen, d_in, d_out, density, permuted, prepared):
    """Packed weights of the package's synthetic recipe (uniform nibbles, scales in [0.001, 0.051], zeros of
    standard deviation 0.2, a Bernoulli mask of residual blocks), drawn on the GPU."""
    dev = gen.device
    ng, nbr = d_in // BCOL, (d_out + BROW - 1) // BROW
    coords = (torch.rand(nbr, ng, generator=gen, device=dev) < density).nonzero()
    nnz = int(coords.shape[0])
    offsets = torch.zeros(nbr + 1, dtype=torch.int32, device=dev)
    offsets[1:] = torch.cumsum(torch.bincount(coords[:, 0], minlength=nbr), 0)
    high = torch.randint(-128, 128, (nnz, BROW, BCOL // 2), generator=gen, device=dev, dtype=torch.int8)
    if d_out % BROW and nnz:
        high[coords[:, 0] == nbr - 1, d_out % BROW:] = 0
    perm = torch.randperm(d_in, generator=gen, device=dev) if permuted else torch.arange(d_in, device=dev)
    W = V9WeightContainer(
        W_low_packed=torch.randint(-128, 128, (d_out, d_in // 2), generator=gen, device=dev, dtype=torch.int8),
        W_high_blocks_packed=high,
        scale_u4=(torch.rand(d_out, ng, generator=gen, device=dev) * 0.05 + 0.001).half(),
        zero_u4=(torch.randn(d_out, ng, generator=gen, device=dev) * 0.2).half(),
        hp_row_offsets=offsets, hp_col_indices=coords[:, 1].to(torch.int32).contiguous(), perm=perm.to(torch.int32),
        block_shape=(BROW, BCOL), d_out=d_out, d_in=d_in)
    return v9_linear.prepare_for_prefill(W) if prepared else W


def _activations(gen, tokens, width):
    """Unit normal with one channel in a hundred twenty times as large."""
    x = torch.randn(tokens, width, generator=gen, device=gen.device)
    x[:, torch.randperm(width, generator=gen, device=gen.device)[:width // 100]] *= 20.0
    return x.half()


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    W = [_container(gen, k, n, case["density"], case["permuted"], case["prepared"]) for k, n in _linears(case)]
    T = case["tokens"]
    state = {"kind": case["kind"], "W": W}
    if case["kind"] != "layer":
        state["X"] = _activations(gen, T, case["d_in"])
        if case["kind"] == "cached":
            graph_cache.set_cuda_graph_policy("auto")
            graph_cache.prewarm_cuda_graph_cache([(state["X"], W[0])])
        return state
    h, f = case["hidden"], case["ffn"]
    state["x"] = [_activations(gen, T, h), _activations(gen, T, h), _activations(gen, T, h),
                  torch.randn(T, 2 * f, generator=gen, device=dev).half()]
    state["norm"] = [(1.0 + 0.1 * torch.randn(h, generator=gen, device=dev)).half() for _ in range(2)]
    if case["graph"]:
        # a decode loop captures its step once, with scratch that lives as long as the graph
        side, state["scratch"] = torch.cuda.Stream(dev), _lib.WorkspaceHolder()
        side.wait_stream(torch.cuda.current_stream(dev))
        with _lib.use_workspace(state["scratch"]), torch.cuda.stream(side):
            _layer_forward(state)
            side.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                state["y"] = _layer_forward(state)
        torch.cuda.current_stream(dev).wait_stream(side)
        state["graph"] = graph
    return state


def _layer_forward(state):
    (qkv, o, gate_up, down), (a, b, c, d), (n1, n2) = state["W"], state["x"], state["norm"]
    return [v9_linear.v9_linear_forward_rmsnorm(a, n1, EPS, qkv),
            v9_linear.v9_linear_forward(b, o),
            v9_linear.v9_linear_forward_rmsnorm(c, n2, EPS, gate_up),
            v9_linear.v9_linear_forward_silu_mul(d, down)]


def run(state):
    kind = state["kind"]
    if kind == "layer":
        if "graph" in state:
            state["graph"].replay()
            return state["y"]
        return _layer_forward(state)
    X, W = state["X"], state["W"][0]
    if kind == "linear":
        return v9_linear.v9_linear_forward(X, W)
    if kind == "cached":
        return graph_cache.v9_linear_forward_cuda_graph(X, W)
    codes, scale_x, sums = activation_quant_cuda(X, W.perm)
    Y = fused_dense_sparse_cuda_int4(W.W_low_packed, W.W_high_blocks_packed, W.hp_row_offsets, W.hp_col_indices,
                                     codes, W.scale_u4, W.zero_u4, sums, scale_x, W.d_out, W.d_in)
    return {"codes": codes, "scale_x": scale_x, "sums": sums, "Y": Y}


def work(case):
    """Packed nibbles, scales, zeros, residual blocks (the expected number of them) and index once; activations in
    and results out once; two operations per multiply-add."""
    T, nbytes, flops = case["tokens"], 0.0, 0.0
    for i, (k, n) in enumerate(_linears(case)):
        ng, nbr = k // BCOL, (n + BROW - 1) // BROW
        nnz = case["density"] * ng * nbr
        nbytes += k * n / 2 + 4 * n * ng + (BROW * BCOL / 2 + 4) * nnz + 4 * (nbr + 1) + (4 * k if case["permuted"] else 0)
        nbytes += T * k * (4 if case["kind"] == "layer" and i == 3 else 2) + 2 * T * n
        if case["kind"] == "operators":
            nbytes += T * (k / 2 + 2 + 4 * ng)        # codes, scale and sums are results of their own
        flops += 2.0 * T * k * n + 2.0 * T * BROW * BCOL * nnz
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Integer codes and sums are exact; outputs are exact integer products folded in fp32 and rounded once to fp16
    (half an ulp is 2^-11 of a value; the fp32 order adds little), so an fp16 step on single values."""
    return {"rel": 1e-3, "max": 1e-2}
