"""Performance cases: the calls a program that uses this package makes, over the sizes it makes them at.

A case names a kind of call and its sizes; `prepare` builds what such a program holds before the call (the quantized matrix
on the GPU, the dense operand, the output, the prepared operation), `run` is one call through the public entry points in
`cellerator_b200.ops`, `work` what the call cannot do without.  The matrices come from the package's seeded generator of
expression data: row lengths lognormal around a median, genes ascending, log1p of negative-binomial counts, codes with one
scale and one zero-point per gene.

Kinds:
  project         Y = act(deq(X) W + bias) with a prepared operation, the matrix's arrays read at every call, fp32 products
  project_once    the same as one call that prepares, runs and releases (`spmm_forward`): cells that are seen once
  project_tensor  prepared with the matrix in hand, 16-bit products allowed: cells that are projected again and again
  project_split   prepared with the matrix in hand, fp32 products
  backward        G' = deq(X)^T G, prepared with the matrix in hand
  backward_once   the same as one call (`spmm_transpose`): the gradient of a batch of cells that is seen once
  backward_fixed  prepared with the matrix in hand, the same bits on every call
  bell            the projection of a quantized Blocked-ELL matrix
  codec           new values into a matrix's codes, and the codes back into values
  lower           a CSR of codes into physical Blocked-ELL (query and materialize)
"""
import math

import torch

from cellerator_b200 import capi, ops, synth


def _csr(name, kind, rows, cols, median, sigma, bits, n=0, dense="f32", epilogue="none", multiply="f32"):
    return dict(name=name, kind=kind, rows=rows, cols=cols, median=median, sigma=sigma, bits=bits, n=n, dense=dense,
                epilogue=epilogue, multiply=multiply)


def _bell(name, kind, rows, cols, ell_blocks, n=0):
    return dict(name=name, kind=kind, rows=rows, cols=cols, ell_blocks=ell_blocks, n=n)


def listed():
    return [
        # a few dozen cells looked up against a gene panel, as an annotation service does for each request: latency
        _csr("query", "project", 64, 2_000, 300, 0.5, 8, 32),
        # a whole small data set against the same panel (the repository's configuration 1)
        _csr("panel", "project", 20_000, 2_000, 300, 0.5, 8, 32),
        # the first layer of an encoder on a mini-batch drawn from the full gene set: seen once, a width that is no
        # power of two, bias and activation in the call
        _csr("minibatch_once", "project_once", 4_099, 33_538, 1_500, 0.6, 8, 50, "bf16", "bias_relu"),
        # a million cells, resident, projected again and again (configuration 2)
        _csr("atlas", "project_tensor", 1_000_000, 33_538, 1_500, 0.6, 8, 64, "bf16", "none", "bf16"),
        # an eighth of it for a caller that wants fp32 products
        _csr("atlas_fp32", "project_split", 125_000, 33_538, 1_500, 0.6, 8, 64, "bf16"),
        # 4-bit codes over highly variable genes, one GPU's share (configuration 4)
        _csr("nibbles", "project_tensor", 500_000, 4_000, 600, 0.5, 4, 128, "bf16", "none", "bf16"),
        # the gene-side gradient of one GPU's share of a million cells (configuration 3 over eight GPUs)
        _csr("gradient", "backward", 125_000, 33_538, 1_500, 0.6, 8, 64),
        # the gradient of a training batch that is seen once
        _csr("gradient_once", "backward_once", 8_191, 33_538, 1_500, 0.6, 8, 64),
        # the gradient of a run that has to be repeatable
        _csr("gradient_fixed", "backward_fixed", 100_003, 33_538, 1_500, 0.6, 8, 64),
        # the blocked tensor-core projection, one GPU's share (configuration 5)
        _bell("blocks", "bell", 249_984, 8_192, 16, 256),
        # a data set that is re-calibrated: values coded again, codes read back
        _csr("codec", "codec", 100_000, 33_538, 1_500, 0.6, 8),
        # the layout step in front of the blocked projection, the same share
        _bell("lowering", "lower", 249_984, 8_192, 16),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["project", "project", "project_once", "project_tensor", "project_tensor", "project_split", "backward",
                       "backward_once", "backward_fixed", "bell", "codec", "lower"])
    if kind in ("bell", "lower"):
        cols = 32 * _spread(rng, 64, 256) - (rng.choice([0, 5]) if kind == "bell" else 0)
        rows = _spread(rng, 2_000, 249_984)
        if kind == "lower":
            rows = rows // 32 * 32
        case = _bell("", kind, rows, cols, rng.choice([8, 12, 16]), rng.choice([128, 256]) if kind == "bell" else 0)
        del case["name"]
        return case
    if kind == "project":
        rows, cols = _spread(rng, 16, 30_000), _spread(rng, 1_000, 4_000)
        n, dense = rng.choice([16, 32, 40, 50, 64, 128]), rng.choice(["f32", "bf16"])
    elif kind == "project_once":
        rows, cols = _spread(rng, 256, 8_192), _spread(rng, 2_000, 33_538)
        n, dense = rng.choice([32, 50, 64, 100, 128]), rng.choice(["f32", "bf16"])
    elif kind == "project_tensor":
        rows, cols = _spread(rng, 5_000, 400_000), _spread(rng, 2_000, 33_538)
        n, dense = rng.choice([32, 64, 128]), "bf16"
    elif kind == "project_split":
        rows, cols = _spread(rng, 5_000, 125_000), _spread(rng, 2_000, 33_538)
        n, dense = rng.choice([32, 64, 128]), rng.choice(["f32", "bf16"])
        if dense == "f32":
            n = min(n, 64)
    elif kind == "backward_once":
        rows, cols = _spread(rng, 256, 16_384), _spread(rng, 2_000, 33_538)
        n, dense = rng.choice([32, 50, 64, 128]), "f32"
    else:
        rows, cols = _spread(rng, 5_000, 125_000), _spread(rng, 2_000, 33_538)
        n, dense = (0 if kind == "codec" else rng.choice([32, 64])), "f32"
    # the more genes, the thinner the rows: 15 % at 2,000, 4.5 % at 33,538
    density = min(0.15, 0.15 * (2_000 / cols) ** 0.43) * rng.uniform(0.8, 1.25)
    case = _csr("", kind, rows, cols, max(8, round(cols * density)), rng.choice([0.5, 0.6]), rng.choice([8, 4]), n, dense,
                rng.choice(["none", "bias", "bias_relu"]) if kind in ("project", "project_once") else "none",
                "bf16" if kind == "project_tensor" or (kind == "backward" and rng.random() < 0.5) else "f32")
    del case["name"]
    return case


def _randn(shape, seed, std, dtype=torch.float32):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").mul_(std).to(dtype)


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    kind, rows, cols = case["kind"], case["rows"], case["cols"]
    n = case["n"]
    s = dict(kind=kind)
    if kind == "bell":
        x = synth.make_qbell_device(rows, cols, 32, case["ell_blocks"], 0.6, 8, device, seed=seed)
        s["x"], s["dense"], s["out"] = x, _randn((cols, n), seed + 1, 0.02, torch.bfloat16), torch.empty(rows, n, device=device)
        s["op"] = ops.PreparedSpmm(capi.PROJECTION_BLOCKED_ELL, rows, cols, n, rows * x.ell_cols, x.bits, x.policy,
                                   torch.bfloat16, device)
        return s
    if kind == "lower":
        h = synth.make_lowering_device(rows, cols, 32, case["ell_blocks"], 0.6, device, seed=seed)
        s["low"] = ops.BellLowering(h["row_offsets"], h["feature_ids"], h["values"], h["features"], h["fb_offsets"],
                                    h["fperm"], h["rperm"], device)
        return s
    # re-calibration keeps a data set's structure: its entries stand where they stood, its values are new ones
    x = s["x"] = synth.make_qcsr_device(rows, cols, case["median"], case["sigma"], 1, cols, case["bits"], device,
                                        seed=1 if kind == "codec" else seed)
    if kind == "codec":
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["values"] = x.dequantize().mul_(torch.rand(x.nnz, generator=g, device=device).mul_(0.2).add_(0.9))
        x.scales.mul_(torch.rand(cols, generator=g, device=device).mul_(0.1).add_(0.95))
        return s
    dtype = torch.bfloat16 if case["dense"] == "bf16" else torch.float32
    multiply = capi.DTYPE_BF16 if case["multiply"] == "bf16" else capi.DTYPE_F32
    if kind.startswith("backward"):
        s["dense"], s["out"] = _randn((rows, n), seed + 1, 1.0), torch.empty(cols, n, device=device)
        if kind != "backward_once":
            s["op"] = ops.PreparedSpmm(capi.PROJECTION_TRANSPOSE, rows, cols, n, x.nnz, x.bits, x.policy, torch.float32, device,
                                       multiply=multiply, device_matrix=x, deterministic=kind == "backward_fixed")
        return s
    s["dense"], s["out"] = _randn((cols, n), seed + 1, 0.02, dtype), torch.empty(rows, n, device=device)
    s["epilogue"] = case["epilogue"]
    s["bias"] = _randn((n,), seed + 2, 0.5) if case["epilogue"].startswith("bias") else None
    if kind != "project_once":
        s["op"] = ops.PreparedSpmm(capi.PROJECTION_CSR, rows, cols, n, x.nnz, x.bits, x.policy, dtype, device,
                                   host_row_ptr=x.host_row_ptr, multiply=multiply,
                                   device_matrix=None if kind == "project" else x)
    return s


def run(s):
    kind = s["kind"]
    if kind == "codec":
        s["x"].quantize_(s["values"])
        return s["x"].packed, s["x"].dequantize()
    if kind == "lower":
        geometry = s["low"].query(32)
        return s["low"].materialize(geometry)
    if kind == "project_once":
        return ops.spmm_forward(s["x"], s["dense"], s["out"], epilogue=s["epilogue"], bias=s["bias"])
    if kind == "backward_once":
        return ops.spmm_transpose(s["x"], s["dense"], s["out"])
    if kind == "bell" or kind.startswith("backward"):
        return s["op"].run(s["x"], s["dense"], s["out"])
    return s["op"].run(s["x"], s["dense"], s["out"], epilogue=s["epilogue"], bias=s["bias"])


def work(case):
    kind, rows, cols, n = case["kind"], case["rows"], case["cols"], case["n"]
    if kind in ("bell", "lower"):
        slots = case["ell_blocks"] * 32
        blocks = -(-rows // 32) * case["ell_blocks"]
        if kind == "bell":
            return {"bytes": rows * slots + blocks * 4 + cols * (2 * n + 8) + rows * n * 4, "flops": 2 * rows * slots * n}
        stored = rows * round(0.6 * slots)
        return {"bytes": (rows + 1) * 4 + stored * 5 + blocks * (4 + 32 * 32), "flops": 0}
    # the mean of a lognormal; clipping at the number of genes takes next to nothing off
    entries = rows * case["median"] * math.exp(case["sigma"] ** 2 / 2)
    matrix = entries * (4 + case["bits"] / 8) + (rows + 1) * 8 + cols * 8
    if kind == "codec":  # genes and values in, codes out; genes and codes in, values out
        return {"bytes": 2 * matrix + 8 * entries, "flops": 0}
    dense = 2 if case["dense"] == "bf16" else 4
    if kind.startswith("backward"):
        return {"bytes": matrix + rows * n * dense + cols * n * 4, "flops": 2 * entries * n}
    return {"bytes": matrix + cols * n * dense + rows * n * 4, "flops": 2 * entries * n}


def tolerance(case):
    kind = case["kind"]
    if kind in ("codec", "lower"):
        return "exact"
    if kind == "bell" or case["multiply"] == "bf16":
        return {"rel": 2e-3}       # products of 16-bit operands, fp32 sums
    if kind in ("project_split", "backward"):
        return {"rel": 2e-5}       # fp32 products put together from 16-bit pieces, fp32 sums
    return {"rel": 1e-5}           # fp32 products, fp32 sums in any order
