"""Performance cases: the work a user has this library do, through its public operators, over the sizes in use.

Five kinds of work:

    spmm             one product through spmm.wmmaSpmm / spmm.cudaSpmm, or a batch of them through ops.spmm_batched
    sddmm            the sampled product, sddmm.wmmaSddmm / sddmm.cudaSddmm or ops.sddmm_batched
    product_train    a layer with a column-vector-sparse weight: sparse_dense_product, forward and backward
    attention        fixed-mask sparse attention, forward (ops.attention_cvse, the caller's workspace)
    attention_train  the same in a training step: fixed_mask_attention, forward and backward

Sizes are those of the pruned ResNet-50-like layers (64 to 2048 rows, 64 to 2048 columns, dense width 256), of the
4096 x 4096 fp32 products (dense width 256 to 8192) and of sequence-4096 attention with 64-wide heads, with ragged sizes
between them.  In a case: V the vector length, m_vec the vector-rows, n the columns of the sparse matrix, k the dense
width (spmm) or contraction length (sddmm), batch the problems of one call that share a structure.
"""
import math

import torch

from vectorsparse_b200 import VS_PATH_CUDA_CORE, VS_PATH_TENSOR, cvse, ops, torch_ops

DEVICE = "cuda:0"
PATHS = {"tensor": VS_PATH_TENSOR, "cuda": VS_PATH_CUDA_CORE}
KINDS = {"fixed": cvse.GEN_FIXED, "uniform": cvse.GEN_UNIFORM}
DTYPES = {"f16": torch.float16, "f32": torch.float32}


def _spmm(path, m_vec, V, n, k, sparsity, pattern, batch, dtype="f16", out="f16"):
    return dict(op="spmm", path=path, dtype=dtype, out=out, m_vec=m_vec, V=V, n=n, k=k, sparsity=sparsity, pattern=pattern,
                batch=batch)


def _sddmm(path, m_vec, V, n, k, sparsity, pattern, batch, out="f16"):
    return dict(op="sddmm", path=path, out=out, m_vec=m_vec, V=V, n=n, k=k, sparsity=sparsity, pattern=pattern, batch=batch)


def _product(m_vec, V, n, k, sparsity, pattern):
    return dict(op="product_train", m_vec=m_vec, V=V, n=n, k=k, sparsity=sparsity, pattern=pattern)


def _attention(op, heads, seq, d, V, sparsity, band):
    return dict(op=op, heads=heads, seq=seq, d=d, V=V, sparsity=sparsity, band=band)


def listed():
    return [
        # the smallest layer of the pruned network, one call: what a call costs before any work
        dict(_spmm("tensor", 64 // 2, 2, 64, 256, 0.7, "skewed", 1), name="spmm_smallest_layer"),
        # the largest layer of the pruned network, one call, as the reference's drivers make it
        dict(_spmm("tensor", 2048 // 8, 8, 512, 256, 0.9, "skewed", 1), name="spmm_largest_layer"),
        # a stream of such products under one pruning mask: throughput serving, the benchmark's default workload
        dict(_spmm("tensor", 2048 // 8, 8, 512, 256, 0.9, "skewed", 256), name="spmm_stream"),
        # a middle layer through the CUDA-core entry point, fine-grained sparsity (V = 1 has no tensor path)
        dict(_spmm("cuda", 1024, 1, 256, 256, 0.8, "skewed", 64), name="spmm_f16_fine_grained"),
        # fp32 products with a large square matrix: vectors of four, an ordinary dense width
        dict(_spmm("cuda", 4096 // 4, 4, 4096, 1024, 0.9, "uniform", 1, "f32", "f32"), name="spmm_f32_v4"),
        # the same fine-grained and as wide as it gets: the largest of the fp32 range
        dict(_spmm("cuda", 4096, 1, 4096, 8192, 0.8, "uniform", 1, "f32", "f32"), name="spmm_f32_fine_grained_wide"),
        # the sampled product of one middle layer, fp32 results (a gradient that is accumulated elsewhere)
        dict(_sddmm("tensor", 512 // 4, 4, 2048, 256, 0.95, "skewed", 1, "f32"), name="sddmm_layer"),
        # a stream of sampled products under one mask
        dict(_sddmm("tensor", 2048 // 8, 8, 512, 256, 0.9, "skewed", 256), name="sddmm_stream"),
        # the CUDA-core sampled product at ragged sizes, a small batch
        dict(_sddmm("cuda", 159, 8, 577, 200, 0.8, "fixed", 16), name="sddmm_f16_ragged"),
        # a training step of a pruned layer on 1984 tokens, ragged rows and columns: forward and both gradients
        dict(_product(302, 4, 1153, 1984, 0.85, "skewed"), name="product_train_ragged"),
        # fixed-mask attention, inference: batch 8 x 16 heads, sequence 4096, local band plus random strided vectors
        dict(_attention("attention", 128, 4096, 64, 8, 0.9, 256), name="attention_inference"),
        # a training step of the same layer at batch 1 and half the sequence
        dict(_attention("attention_train", 16, 2048, 64, 8, 0.9, 128), name="attention_train"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: rows 64 to 4096, columns 64 to 4608, sparsity 50 to 98 %, any V, odd sizes."""
    while True:
        op = rng.choice(["spmm", "spmm", "spmm", "spmm_cuda", "spmm_f32", "sddmm", "sddmm", "sddmm_cuda", "product_train",
                         "attention", "attention_train"])
        sparsity = round(rng.uniform(0.5, 0.98), 3)
        if op in ("attention", "attention_train"):
            seq = _log_int(rng, 32, 512) * 8
            case = _attention(op, _log_int(rng, 1, 128), seq, rng.choice([64, 64, 64, 128]), rng.choice([8, 8, 4, 2]),
                              round(rng.uniform(0.8, 0.95), 3), seq // 16)
            cost = case["heads"] * float(seq) * seq * case["d"] * (4 if op == "attention_train" else 1)
            if cost <= 128 * 4096.0 * 4096 * 64:
                return case
            continue
        V = rng.choice([2, 4, 8]) if op in ("spmm", "sddmm", "product_train") else rng.choice([1, 2, 4, 8])
        m_vec = max(_log_int(rng, 64, 4096) // V, 8)
        n = _log_int(rng, 64, 4608)
        pattern = rng.choice(["skewed", "skewed", "fixed", "uniform"])
        out = rng.choice(["f16", "f16", "f16", "f32"])
        batch = rng.choice([1, 1, _log_int(rng, 2, 256)])
        if op == "spmm":
            case = _spmm("tensor", m_vec, V, n, 64 * _log_int(rng, 1, 32), sparsity, pattern, batch, "f16", out)
        elif op == "spmm_cuda":
            case = _spmm("cuda", m_vec, V, n, 8 * _log_int(rng, 4, 256), sparsity, pattern, batch, "f16", out)
        elif op == "spmm_f32":
            case = _spmm("cuda", m_vec, V, n, 4 * _log_int(rng, 16, 2048), sparsity, pattern, batch, "f32", "f32")
        elif op == "sddmm":
            case = _sddmm("tensor", m_vec, V, n, 64 * _log_int(rng, 1, 32), sparsity, pattern, batch, out)
        elif op == "sddmm_cuda":
            case = _sddmm("cuda", m_vec, V, n, 8 * _log_int(rng, 4, 256), sparsity, pattern, batch, out)
        else:
            case = _product(m_vec, V, n, 64 * _log_int(rng, 1, 64), sparsity, pattern)
        dense = 2.0 * m_vec * V * n * case["k"] * case.get("batch", 3)
        if dense <= 1.4e11 and dense * (1 - sparsity) <= 2e10:
            return case


def _nnz_vec(case):
    """Number of nonzero vectors (the uniform pattern rounds over the whole matrix and may differ by a few)."""
    if "seq" in case:
        return case["seq"] // case["V"] * max(int(round((1 - case["sparsity"]) * case["seq"])), case["band"])
    return case["m_vec"] * max(int(round((1 - case["sparsity"]) * case["n"])), 1)


def _pattern(case, seed, gen):
    """The sparse structure: "fixed" vectors per row, "uniform" over the matrix, or "skewed": row densities of a
    Beta(2,2) profile (the middle one of three uniforms), as magnitude pruning leaves them.  The number of nonzero
    vectors depends on the sizes only."""
    m_vec, n, V = case["m_vec"], case["n"], case["V"]
    if case["pattern"] != "skewed":
        return cvse.generate(KINDS[case["pattern"]], seed, m_vec, n, V, case["sparsity"])
    density = torch.rand((m_vec, 3), generator=gen, device=DEVICE).sort(dim=1).values[:, 1:2]
    score = torch.rand((m_vec, n), generator=gen, device=DEVICE) / (density + 1e-3)
    keep = score.view(-1).topk(_nnz_vec(case), largest=False, sorted=False).indices
    mask = torch.zeros(m_vec * n, dtype=torch.uint8, device=DEVICE)
    mask[keep] = 1
    return cvse.from_dense_mask(mask.view(m_vec, n).cpu().numpy(), V)


def prepare(case, seed):
    op, V = case["op"], case["V"]
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)

    def normal(shape, sigma=1.0):
        return (torch.randn(shape, generator=gen, device=DEVICE) * sigma).to(torch.float16)

    def uniform(shape, dtype):
        return (torch.rand(shape, generator=gen, device=DEVICE) * 2 - 1).to(dtype)

    if op in ("attention", "attention_train"):
        heads, seq, d = case["heads"], case["seq"], case["d"]
        a = cvse.generate(cvse.GEN_BAND, seed, seq // V, seq, V, case["sparsity"], band=case["band"])
        q, k, v = (normal((heads, seq, d)) for _ in range(3))
        s = dict(op=op, a=a, V=V, d=d, n=seq, scale=d ** -0.5, q=q, k=k, v=v)
        if op == "attention":
            s.update(structure=a.to_device(DEVICE), out=torch.empty_like(q),
                     workspace=torch.empty((heads, a.nnz_vec * V), dtype=torch.float16, device=DEVICE))
        else:
            s.update(mask=torch_ops.AttentionMask(a, DEVICE), grad_out=normal((heads, seq, d)))
            for t in (q, k, v):
                t.requires_grad_(True)
        return s

    m_vec, n, k = case["m_vec"], case["n"], case["k"]
    a = _pattern(case, seed, gen)
    s = dict(op=op, a=a, V=V, n=n, k=k)
    if op == "product_train":
        s.update(mask=torch_ops.AttentionMask(a, DEVICE), values=normal((a.nnz_vec * V,), 0.02).requires_grad_(True),
                 b=normal((n, k)).requires_grad_(True), grad_c=normal((m_vec * V, k)))
        return s

    batch = case["batch"]
    row = (a.nnz_vec * V + 7) // 8 * 8   # batched value arrays keep 16-byte aligned rows
    s.update(structure=a.to_device(DEVICE), batch=batch, path=PATHS[case["path"]])
    lead = (batch,) if batch > 1 else ()
    if op == "spmm":
        if case["dtype"] == "f32":
            s.update(values=uniform(lead + (row,), torch.float32), rhs=uniform(lead + (n, k), torch.float32))
        else:
            s.update(values=normal(lead + (row,), 0.02), rhs=normal(lead + (n, k)))
        s["out"] = torch.empty(lead + (m_vec * V, k), dtype=DTYPES[case["out"]], device=DEVICE)
    else:
        s.update(lhs=normal(lead + (m_vec * V, k)), rhs=normal(lead + (n, k)))
        s["out"] = torch.zeros(lead + (row,), dtype=DTYPES[case["out"]], device=DEVICE)
    return s


def run(s):
    op, a, V = s["op"], s["a"], s["V"]
    if op == "spmm":
        args = (a.m_vec, V, s["k"], s["n"], *s["structure"], s["values"], s["rhs"], s["out"])
        if s["batch"] > 1:
            ops.spmm_batched(s["path"], *args)
        elif s["path"] == VS_PATH_TENSOR:
            ops.spmm.wmmaSpmm(*args)
        else:
            ops.spmm.cudaSpmm(*args)
        return s["out"]
    if op == "sddmm":
        args = (a.m_vec, s["k"], s["n"], a.nnz_vec, *s["structure"], s["lhs"], s["rhs"], s["out"], V)
        if s["batch"] > 1:
            ops.sddmm_batched(s["path"], *args)
        elif s["path"] == VS_PATH_TENSOR:
            ops.sddmm.wmmaSddmm(*args)
        else:
            ops.sddmm.cudaSddmm(*args)
        return s["out"]
    if op == "product_train":
        c = torch_ops.sparse_dense_product(s["values"], s["b"], s["mask"])
        grads = torch.autograd.grad(c, (s["values"], s["b"]), s["grad_c"])
        return (c.detach(), *grads)
    if op == "attention":
        ops.attention_cvse(VS_PATH_TENSOR, a.m_vec, V, s["n"], s["d"], a.nnz_vec, *s["structure"], s["q"], s["k"], s["v"],
                           s["out"], s["workspace"], s["scale"])
        return s["out"]
    out = torch_ops.fixed_mask_attention(s["q"], s["k"], s["v"], s["mask"], s["scale"])
    grads = torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["grad_out"])
    return (out.detach(), *grads)


def work(case):
    """Bytes: dense operands, values and structure once each; flops: two per stored value and dense column."""
    V, vec = case["V"], _nnz_vec(case)
    if "seq" in case:
        heads, seq, d, train = case["heads"], case["seq"], case["d"], case["op"] == "attention_train"
        structure = vec * 4 + (2 * (seq // V) + 1) * 4
        if train:
            structure += vec * 8 + (seq + 1) * 4
        # q, k, v in and the result out; in training dO in and three gradients out as well.  Two products forward; four
        # more backward (dV, dP, dQ, dK)
        return {"bytes": structure + heads * (8 if train else 4) * seq * d * 2, "flops": (12.0 if train else 4.0) * heads * vec * V * d}
    m, n, k = case["m_vec"] * V, case["n"], case["k"]
    structure = vec * 4 + (2 * case["m_vec"] + 1) * 4
    if case["op"] == "product_train":   # values, b, dC in; C, dvalues, db out; three products
        return {"bytes": structure + vec * 8 + (n + 1) * 4 + 2 * 2 * (vec * V + n * k + m * k), "flops": 6.0 * vec * V * k}
    es_in, es_out = (4 if case.get("dtype") == "f32" else 2), (4 if case["out"] == "f32" else 2)
    if case["op"] == "spmm":
        per = vec * V * es_in + n * k * es_in + m * k * es_out
    else:
        per = (m + n) * k * es_in + vec * V * es_out
    return {"bytes": structure + case["batch"] * per, "flops": 2.0 * case["batch"] * vec * V * k}


def tolerance(case):
    """fp16 results carry a rounding of 2^-11 each; the attention pipeline rounds scores and probabilities to fp16 on
    the way, its gradients cancel on top of that.  fp32 results: fp32 sums in another order."""
    if case["op"] == "attention_train":
        return {"rel": 1e-2}
    if case["op"] == "attention":
        return {"rel": 5e-3}
    if case["op"] == "product_train" or case["out"] == "f16":
        return {"rel": 2e-3}
    return {"rel": 1e-5}
