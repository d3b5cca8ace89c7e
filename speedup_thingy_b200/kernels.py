"""Operator table with the names, argument meaning and error behaviour of the reference's
``recursive_training_engine.kernels.optimized`` (optimized.py:12-154; arithmetic of kernels/reference.py:9-157).

Assigning these functions over the reference's symbols (or importing this module in its place) routes the
six operators the reference model actually calls -- ``k_fused_rmsnorm`` (layers.py:33), ``k_rope_apply``
(layers.py:50), ``k_flash_causal_dense`` (layers.py:73), ``k_flash_causal_grouped`` (layers.py:725),
``k_out_proj_grouped`` (layers.py:727), ``k_logits_shortlist`` (output.py:125) -- and the benchmarked
``k_logits_full`` / ``k_qkv_dense`` / ``k_cross_entropy_unreduced`` through the sm_100a kernels of the C ABI.
Every operator is an autograd function whose forward and backward are C-ABI launches, native where it is called per layer
(csrc/host_ops.cpp, where a launch costs the host 3-4 us and a call 6 more, against 15-20 us per launch from Python); tensors go in and come out as the
reference's do (fresh outputs, inputs untouched, non-contiguous inputs accepted).

There is no fallback: CPU tensors raise ``RuntimeError`` mentioning ``strict_cuda`` whatever the flag says
(optimized.py:51-55), and a missing library or device raises when the first operator is called.
GEMM-bearing operators compute in bf16 with fp32 accumulation (the reference's autocast arithmetic) and return
the input's dtype.
"""
from __future__ import annotations

import torch

from . import _abi as A
from .ops import CudaOps

STRICT_CUDA = True
REQUIRE_FLASH = True
_OPS: dict[int, CudaOps] = {}


# --------------------------------------------------------------------------- policy functions (optimized.py:12-49)
def set_strict_cuda(enabled: bool, *, require_flash: bool = True) -> None:
    """Recorded for `backend_status`; the kernels reject CPU tensors either way (there is nothing to fall back to)."""
    global STRICT_CUDA, REQUIRE_FLASH
    STRICT_CUDA, REQUIRE_FLASH = bool(enabled), bool(require_flash)


def triton_available() -> bool:
    """The reference's gate for its accelerated paths; here it reports whether the sm_100a library can run."""
    return torch.cuda.is_available()


def backend_status() -> dict[str, object]:
    cuda = torch.cuda.is_available()
    return {"mode": CudaOps.name if cuda else "unavailable", "strict_cuda": True, "require_flash": REQUIRE_FLASH,
            "cuda_available": cuda, "triton_available": False, "uses_reference_fallback": False}


def cuda_required() -> None:
    if not torch.cuda.is_available():
        raise RuntimeError("CUDA is required for this optimized kernel path (rte_b200 has no CPU or Triton path)")


def _require_cuda_tensor(*tensors) -> None:
    if any(isinstance(t, torch.Tensor) and not t.is_cuda for t in tensors):
        raise RuntimeError("strict_cuda requires CUDA tensors in optimized hot-path kernels (rte_b200 has no fallback)")


def _ops_for(t: torch.Tensor) -> CudaOps:
    idx = t.device.index if t.device.index is not None else torch.cuda.current_device()
    if idx not in _OPS:
        ops = CudaOps(torch.device("cuda", idx))
        A.load_host().bind_status(ops.status)
        _OPS[idx] = ops
    return _OPS[idx]


def _native(t: torch.Tensor):
    """The native operators, with the launch table of `t`'s device in place."""
    _ops_for(t)
    return A.load_host()


def _bf16(t: torch.Tensor) -> torch.Tensor:
    return t.detach().to(torch.bfloat16).contiguous()


def _f32(t: torch.Tensor) -> torch.Tensor:
    return t.detach().to(torch.float32).contiguous()


def _check_gemm_dims(*dims: int) -> None:
    if any(v % 8 for v in dims):
        raise ValueError(f"rte_b200 GEMM operands need dimensions that are multiples of 8, got {dims}")


# --------------------------------------------------------------------------- RMSNorm (reference.py:9-17)
def k_fused_rmsnorm(x, weight, residual=None, eps: float = 1e-5):
    """(rmsnorm(x [+ residual]) * weight, x + residual | None), statistics in fp32 (reference.py:9-17)."""
    _require_cuda_tensor(x, weight, residual)
    if x.shape[-1] != weight.shape[-1]:
        raise ValueError("k_fused_rmsnorm: weight must match the last dimension of x")
    return _native(x).rmsnorm(x, weight, residual, float(eps))


# --------------------------------------------------------------------------- rotary embedding (reference.py:20-28)
def k_rope_apply(q, k, cos, sin):
    """q*cos + rotate_half(q)*sin on adjacent pairs, same for k; cos/sin [S, head_dim] (reference.py:20-28)."""
    _require_cuda_tensor(q, k, cos, sin)
    if q.shape[-2:] != k.shape[-2:] or cos.shape[-2:] != q.shape[-2:] or cos.numel() != q.shape[-2] * q.shape[-1]:
        raise ValueError("k_rope_apply: q/k [..., S, head_dim] with cos/sin [S, head_dim]")
    return _native(q).rope(q, k, cos, sin)


# --------------------------------------------------------------------------- causal attention (reference.py:40-41,54-55)
def k_flash_causal_dense(q, k, v):
    """softmax(q k^T / sqrt(head_dim), causal) v over [B, H, S, head_dim] (reference.py:40-41)."""
    _require_cuda_tensor(q, k, v)
    if q.ndim != 4 or q.shape != k.shape or q.shape != v.shape:
        raise ValueError("k_flash_causal_*: q, k, v must share the shape [B, H, S, head_dim]")
    if q.shape[2] > 256 or q.shape[3] not in (8, 16, 32, 64, 128):
        raise ValueError("k_flash_causal_*: S <= 256 and head_dim in {8,16,32,64,128}")
    return _native(q).attention(q, k, v, _ops_for(q).identity_rope_table(q.shape[2], q.shape[3]))


k_flash_causal_grouped = k_flash_causal_dense          # same arithmetic over the active heads (reference.py:54-55)


# --------------------------------------------------------------------------- GEMM-bearing operators
def k_qkv_dense(x, wq, wk, wv):
    """(x @ wq, x @ wk, x @ wv), weights [in, out] (reference.py:31-37)."""
    _require_cuda_tensor(x, wq, wk, wv)
    return _native(x).qkv_dense(x, wq, wk, wv)


def k_logits_full(hidden, vocab_weight):
    """hidden @ vocab_weight^T (reference.py:137-138)."""
    _require_cuda_tensor(hidden, vocab_weight)
    if hidden.shape[-1] != vocab_weight.shape[-1]:
        raise ValueError("k_logits_full: hidden [..., d] against vocab_weight [V, d]")
    return _native(hidden).matmul_oi(hidden, vocab_weight)


def k_out_proj_grouped(x, wo, row_indices):
    """x @ wo[row_indices, :] with the selected rows gathered by the C-ABI row gather (reference.py:58-59)."""
    _require_cuda_tensor(x, wo, row_indices)
    if x.shape[-1] != row_indices.numel():
        raise ValueError("k_out_proj_grouped: x [..., len(row_indices)]")
    return _native(x).out_proj(x, wo, row_indices)


# --------------------------------------------------------------------------- shortlist logits (reference.py:141-143)
class _LogitsShortlist(torch.autograd.Function):
    @staticmethod
    def forward(ctx, hidden, vocab_weight, shortlist):
        ops = _ops_for(hidden)
        d, K = hidden.shape[-1], shortlist.shape[-1]
        h16, w16 = _bf16(hidden).view(-1, d), _bf16(vocab_weight)
        ids = shortlist.detach().to(torch.int32).contiguous().view(-1, K)
        rows = h16.shape[0]
        logits = torch.empty(rows, K, dtype=torch.bfloat16, device=hidden.device)
        scratch = torch.empty(rows, dtype=torch.float32, device=hidden.device)
        ops.shortlist_ce(h16, w16, ids, None, 1, scratch, logits, None)
        ctx.save_for_backward(h16, w16, ids)
        ctx.meta = (hidden.shape, hidden.dtype, vocab_weight.dtype)
        return logits.to(hidden.dtype).view(*shortlist.shape)

    @staticmethod
    def backward(ctx, dlogits):
        h16, w16, ids = ctx.saved_tensors
        ops = _ops_for(h16)
        hshape, hd, wd = ctx.meta
        rows, d = h16.shape
        V, K = w16.shape[0], ids.shape[1]
        _check_gemm_dims(V)
        # gradient over shortlist slots -> otherwise-zero dense rows, so both products run on the tensor cores
        dense = torch.empty(rows, V, dtype=torch.bfloat16, device=h16.device)
        ops.scatter_cols(_bf16(dlogits).view(rows, K), ids, dense)
        dh = torch.empty(rows, d, dtype=torch.float32, device=h16.device)
        ops.gemm(dense, w16, dh, M=rows, N=d, K=V, b_mn=True, epilogue=A.EPI_F32)
        dw = torch.empty(V, d, dtype=torch.float32, device=h16.device)
        ops.gemm_wgrad(dense, h16, dw, M=V, N=d, K=rows)
        return dh.view(hshape).to(hd), dw.to(wd), None


def k_logits_shortlist(hidden, vocab_weight, shortlist):
    """(hidden[..., None, :] * vocab_weight[shortlist]).sum(-1); ids must be distinct within a row for the
    backward pass (they are: output.py:46-70)."""
    _require_cuda_tensor(hidden, vocab_weight, shortlist)
    if hidden.shape[:-1] != shortlist.shape[:-1]:
        raise ValueError("k_logits_shortlist: hidden [..., d] with shortlist [..., K]")
    return _LogitsShortlist.apply(hidden, vocab_weight, shortlist)


# --------------------------------------------------------------------------- cross entropy (reference.py:146-147)
def k_cross_entropy_unreduced(logits, targets):
    """Per-token loss.  Backward reads the logits again: autograd refuses it if they have been modified in place by then."""
    _require_cuda_tensor(logits, targets)
    if logits.shape[:-1] != targets.shape:
        raise ValueError("k_cross_entropy_unreduced: logits [..., V] with targets [...]")
    return _native(logits).cross_entropy(logits, targets)


# --------------------------------------------------------------------------- host-side helpers of the table
def k_recurrent_exact_loop(step_fn, h, h0, depth: int, boundaries: set):
    """Control flow only (reference.py:127-134)."""
    states = {}
    for t in range(depth):
        h = step_fn(h, h0)
        if t + 1 in boundaries:
            states[t + 1] = h
    return h, states


def k_metrics_reduce(values: dict) -> dict:
    """One device-to-host read per key, as reference.py:156-157."""
    return {k: float(v.detach().float().mean().cpu()) for k, v in values.items()}


def k_sample_audit_mask(p, seed: int):
    """Bernoulli audit mask from a generator on p's device seeded with `seed` (reference.py:151-154): a host-side
    sampling decision, kept as the reference draws it so that the same seed gives the same mask."""
    gen = torch.Generator(device=p.device)
    gen.manual_seed(seed)
    return torch.bernoulli(p, generator=gen).bool()


class PackedByRecipe:
    """Result of `k_pack_by_recipe` (reference.py:81-88): same field names."""
    __slots__ = ("packed", "permutation", "inverse_permutation", "keys", "offsets", "unique_keys")

    def __init__(self, packed, permutation, inverse_permutation, keys, offsets, unique_keys):
        self.packed, self.permutation, self.inverse_permutation = packed, permutation, inverse_permutation
        self.keys, self.offsets, self.unique_keys = keys, offsets, unique_keys


class _GatherRows(torch.autograd.Function):
    """out[i] = src[index[i]] for a PERMUTATION `index` through the C-ABI row gather; the backward is the gather by
    the inverse permutation (no atomics)."""

    @staticmethod
    def forward(ctx, src, index, inverse):
        ops = _ops_for(src)
        flat = src.detach().contiguous().view(src.shape[0], -1)
        out = torch.empty_like(flat)
        ops.gather_rows(flat, index.to(torch.int32), out, flat.shape[0], flat.shape[1] * flat.element_size())
        ctx.save_for_backward(index, inverse)
        return out.view(src.shape)

    @staticmethod
    def backward(ctx, d_out):
        index, inverse = ctx.saved_tensors
        ops = _ops_for(d_out)
        flat = d_out.contiguous().view(d_out.shape[0], -1)
        out = torch.empty_like(flat)
        ops.gather_rows(flat, inverse.to(torch.int32), out, flat.shape[0], flat.shape[1] * flat.element_size())
        return out.view(d_out.shape), None, None


def _gather_ok(t: torch.Tensor) -> None:
    if (t[0].numel() * t.element_size()) % 16:
        raise ValueError("rte_b200 row gathers move 16-byte units: a row must be a multiple of 16 bytes")


def k_pack_by_recipe(hidden, recipe_ids, depth_ids, audit_flags=None):
    """Stable sort of the samples by (recipe, depth, audited) and the packed copy of `hidden` in that order
    (reference.py:91-104).  The keys are sorted on the device by torch (index bookkeeping); the rows move through
    rte_gather_rows."""
    _require_cuda_tensor(hidden, recipe_ids, depth_ids, audit_flags)
    audit = torch.zeros_like(recipe_ids) if audit_flags is None else audit_flags.long()
    keys = recipe_ids.long() * 1_000_000 + depth_ids.long() * 10 + audit
    sorted_keys, perm = torch.sort(keys, stable=True)
    inverse = torch.empty_like(perm)
    inverse[perm] = torch.arange(perm.numel(), device=perm.device)
    unique, counts = torch.unique_consecutive(sorted_keys, return_counts=True)
    offsets = torch.cat([counts.new_zeros(1), counts.cumsum(0)])
    _gather_ok(hidden)
    return PackedByRecipe(_GatherRows.apply(hidden, perm, inverse), perm, inverse, sorted_keys, offsets, unique)


def k_unpack_from_recipe(packed, inverse_permutation):
    """packed[inverse_permutation] (reference.py:107-108)."""
    _require_cuda_tensor(packed, inverse_permutation)
    _gather_ok(packed)
    perm = torch.empty_like(inverse_permutation)
    perm[inverse_permutation] = torch.arange(inverse_permutation.numel(), device=inverse_permutation.device)
    return _GatherRows.apply(packed, inverse_permutation, perm)


def k_qkv_grouped(x, wq, wk, wv, column_indices):
    """x @ w[:, column_indices] for the three projections (reference.py:44-51); the gathered columns are multiplied by
    the tcgen05 GEMM, autograd scatters their gradients back into the full weights."""
    _require_cuda_tensor(x, wq, wk, wv, column_indices)
    cols = column_indices.long()
    return k_qkv_dense(x, wq.index_select(1, cols), wk.index_select(1, cols), wv.index_select(1, cols))


def _swiglu_io(x, wu, wg, wd):
    """(x @ wu) * silu(x @ wg) @ wd with [in, out] weights through the packed SwiGLU FFN (GEMM + SiLU-gate + GEMM)."""
    wug = torch.cat([wu.t(), wg.t()], dim=0)            # [2M, d] = (up rows | gate rows)
    flat = x.reshape(-1, x.shape[-1])
    return packed_swiglu_ffn(flat, wug, wd).view(*x.shape[:-1], wd.shape[-1])


def k_swiglu_dense(x, wu, wg, wd):
    """reference.py:62-68."""
    _require_cuda_tensor(x, wu, wg, wd)
    return _swiglu_io(x, wu, wg, wd)


def k_swiglu_grouped(x, wu, wg, wd, slab_indices):
    """reference.py:71-78: SwiGLU over the hidden units `slab_indices` only."""
    _require_cuda_tensor(x, wu, wg, wd, slab_indices)
    idx = slab_indices.long()
    return _swiglu_io(x, wu.index_select(1, idx), wg.index_select(1, idx), wd.index_select(0, idx))


def k_macro_phi(h, h0, d_gain, v, u, bias, eps: float = 1e-5):
    """The operator table's simplified macro operator (reference.py:111-124): h + d_gain*h + silu(z @ v) @ u + bias with
    z = [rmsnorm(h) | mean_S rmsnorm(h) | h0].  (The model itself runs the bounded-residual form, rte_macro_phi_fwd.)
    Norm and both products run in the sm_100a kernels; concatenation and the element-wise tail are tensor glue."""
    _require_cuda_tensor(h, h0, d_gain, v, u, bias)
    normed, _ = k_fused_rmsnorm(h, torch.ones(h.shape[-1], device=h.device, dtype=h.dtype), None, eps)
    pooled = normed.mean(dim=1, keepdim=True).expand_as(normed)
    z = torch.cat([normed, pooled, h0], dim=-1)
    native = _native(z)
    low = native.matmul_io(torch.nn.functional.silu(native.matmul_io(z, v)), u)
    return h + d_gain * h + low + bias


# --------------------------------------------------------------------------- packed SwiGLU FFN
def packed_swiglu_ffn(x, wug, wdown_rows):
    """Drop-in for ``triton_packed_swiglu_ffn`` (kernels/active_swiglu_triton.py:111-125; layers.py:90-116,284-339):
    x [tokens, d], wug [2*active_m, d] = (up rows | gate rows), wdown_rows [active_m, d].  Same shape errors;
    saves (x, wug, wdown_rows, ug, z) in bf16 as the reference's _TritonPackedSwiGLUFFN does (:62-108)."""
    _require_cuda_tensor(x, wug, wdown_rows)
    if x.ndim != 2 or wug.ndim != 2 or wdown_rows.ndim != 2:
        raise ValueError("expected x [N,D], wug [2M,D], wdown_rows [M,D]")
    if wug.shape[0] % 2 != 0:
        raise ValueError("wug first dimension must be 2M")
    if wdown_rows.shape[0] != wug.shape[0] // 2:
        raise ValueError("wdown_rows first dimension must match M")
    _check_gemm_dims(x.shape[1], wdown_rows.shape[0])
    return _native(x).packed_ffn(x, wug, wdown_rows)


triton_packed_swiglu_ffn = packed_swiglu_ffn          # the symbol layers.py:12-22 imports


def active_union_swiglu(x, wug_weight, wd_weight, active_ids):
    """ActiveUnionSwiGLU.forward (layers.py:267-282): SwiGLU over the sorted unique `active_ids` only.
    wug_weight [2F, d], wd_weight [d, F]; the active rows are gathered by the C-ABI row gather."""
    _require_cuda_tensor(x, wug_weight, wd_weight, active_ids)
    ids = torch.unique(active_ids.reshape(-1).to(torch.int64), sorted=True)
    f = wd_weight.shape[1]
    rows = torch.cat([ids, ids + f]).to(torch.int32)
    # index_select keeps autograd's scatter of the row gradients into the dense weights
    wug_active = wug_weight.index_select(0, rows.long())
    wd_rows = wd_weight.t().index_select(0, ids)
    flat = x.reshape(-1, x.shape[-1])
    return packed_swiglu_ffn(flat, wug_active, wd_rows).view(*x.shape[:-1], -1)
