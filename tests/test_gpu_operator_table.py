"""The drop-in operator table (`speedup_thingy_b200.kernels`, the counterpart of the reference's
`kernels/optimized.py`) on a B200: outputs against the reference-generated per-op golden vectors
(`tests/golden/per_op.npz`, inputs regenerated from the same seed) and against the oracle's fp32 restatements,
gradients against autograd through those restatements.  Tolerances: fp32 operators 1e-4, bf16 operators 2e-2 of
the output scale."""
from pathlib import Path

import numpy as np
import pytest
import torch

from oracle import rte_oracle as O
from speedup_thingy_b200 import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GOLD = np.load(Path(__file__).resolve().parent / "golden" / "per_op.npz")


def _golden_inputs():
    """Same draws, in the same order, as tests/golden/make_golden.py::per_op_vectors."""
    g = torch.Generator().manual_seed(11)
    x, w = torch.randn(3, 5, 24, generator=g), torch.randn(24, generator=g)
    q, k, v = (torch.randn(2, 3, 7, 8, generator=g) for _ in range(3))
    logits = torch.randn(4, 6, 17, generator=g)
    tg = torch.randint(0, 17, (4, 6), generator=g)
    return x, w, q, k, v, logits, tg


def _close(a, b, rel, abs_=0.0):
    a, b = a.detach().float().cpu(), torch.as_tensor(b).float()
    assert a.shape == b.shape
    err = (a - b).abs().max().item()
    assert err <= rel * b.abs().max().item() + abs_, err


def test_rmsnorm_matches_reference_golden_and_grads():
    x, w, *_ = _golden_inputs()
    xg, wg = x.to(DEV).requires_grad_(), w.to(DEV).requires_grad_()
    out, summed = K.k_fused_rmsnorm(xg, wg)
    assert summed is None
    _close(out, GOLD["rmsnorm"], 1e-5, 1e-5)
    xr, wr = x.clone().requires_grad_(), w.clone().requires_grad_()
    ref = O.rmsnorm(xr, wr)
    probe = torch.randn_like(ref)
    (ref * probe).sum().backward()
    (out * probe.to(DEV)).sum().backward()
    _close(xg.grad, xr.grad, 1e-4, 1e-5)
    _close(wg.grad, wr.grad, 1e-4, 1e-5)


def test_rmsnorm_with_residual_returns_sum_and_routes_both_grads():
    g = torch.Generator().manual_seed(3)
    x, r, w = torch.randn(4, 9, 64, generator=g), torch.randn(4, 9, 64, generator=g), torch.randn(64, generator=g)
    leaves = [t.to(DEV).requires_grad_() for t in (x, r, w)]
    out, summed = K.k_fused_rmsnorm(leaves[0], leaves[2], leaves[1])
    ref_leaves = [t.clone().requires_grad_() for t in (x, r, w)]
    y = ref_leaves[0] + ref_leaves[1]
    ref = O.rmsnorm(y, ref_leaves[2])
    _close(out, ref, 1e-5, 1e-5)
    _close(summed, y, 1e-6, 1e-6)
    (ref.sum() + (y * y).sum()).backward()
    (out.sum() + (summed * summed).sum()).backward()
    for a, b in zip(leaves, ref_leaves):
        _close(a.grad, b.grad, 1e-4, 1e-5)
    assert torch.equal(leaves[0].detach().cpu(), x)            # inputs untouched


def test_rope_matches_reference_golden_and_is_orthogonal():
    _, _, q, k, *_ = _golden_inputs()
    cos, sin = O.rope_tables(7, 8)
    qg, kg = q.to(DEV).requires_grad_(), k.to(DEV).requires_grad_()
    rq, rk = K.k_rope_apply(qg, kg, cos.to(DEV), sin.to(DEV))
    _close(rq, GOLD["rope_q"], 1e-5, 1e-6)
    _close(rk, GOLD["rope_k"], 1e-5, 1e-6)
    probe = torch.randn(2, 3, 7, 8, generator=torch.Generator().manual_seed(1))
    ((rq + 2 * rk) * probe.to(DEV)).sum().backward()
    qr = q.clone().requires_grad_()
    (O.rope_apply(qr, cos, sin) * probe).sum().backward()
    _close(qg.grad, qr.grad, 1e-5, 1e-6)
    _close(kg.grad, 2 * qr.grad, 1e-5, 1e-6)             # the rotation is linear: d/dk of 2*rope(k) = 2 * adjoint(probe)
    # bf16 data path
    rq16, _ = K.k_rope_apply(q.to(DEV).bfloat16(), k.to(DEV).bfloat16(), cos.to(DEV), sin.to(DEV))
    assert rq16.dtype == torch.bfloat16
    _close(rq16, GOLD["rope_q"], 2e-2)


@pytest.mark.parametrize("B,H,S,hd", [(2, 3, 7, 8), (3, 4, 64, 64), (2, 2, 130, 32)])
def test_flash_causal_dense_output_and_grads(B, H, S, hd):
    if (B, H, S, hd) == (2, 3, 7, 8):
        _, _, _, _, v, *_ = _golden_inputs()
        q, k = torch.from_numpy(GOLD["rope_q"]), torch.from_numpy(GOLD["rope_k"])
    else:
        g = torch.Generator().manual_seed(S)
        q, k, v = (torch.randn(B, H, S, hd, generator=g) for _ in range(3))
    leaves = [t.to(DEV).requires_grad_() for t in (q, k, v)]
    out = K.k_flash_causal_grouped(*leaves)
    ref_leaves = [t.bfloat16().float().requires_grad_() for t in (q, k, v)]
    ref = O.causal_attention(*ref_leaves)
    if (B, H, S, hd) == (2, 3, 7, 8):
        _close(out, GOLD["attn"], 2e-2)
    _close(out, ref, 2e-2)
    probe = torch.randn(B, H, S, hd, generator=torch.Generator().manual_seed(2))
    (ref * probe).sum().backward()
    (out * probe.to(DEV)).sum().backward()
    for a, b in zip(leaves, ref_leaves):
        _close(a.grad, b.grad, 3e-2)


def test_cross_entropy_matches_reference_golden_and_grads():
    *_, logits, tg = _golden_inputs()
    lg = logits.to(DEV).requires_grad_()
    loss = K.k_cross_entropy_unreduced(lg, tg.to(DEV))
    assert loss.shape == tg.shape
    _close(loss, GOLD["ce"], 2e-2)
    lr = logits.bfloat16().float().requires_grad_()
    ref = torch.nn.functional.cross_entropy(lr.flatten(0, 1), tg.flatten(), reduction="none").view_as(tg)
    wgt = torch.rand(4, 6, generator=torch.Generator().manual_seed(4)) + 0.5
    (ref * wgt).sum().backward()
    (loss * wgt.to(DEV)).sum().backward()
    _close(lg.grad, lr.grad, 2e-2)


def test_logits_full_qkv_dense_and_out_proj_grouped():
    g = torch.Generator().manual_seed(5)
    h, W = torch.randn(3, 40, 64, generator=g), torch.randn(96, 64, generator=g) * 0.2
    hg, Wg = h.to(DEV).requires_grad_(), W.to(DEV).requires_grad_()
    out = K.k_logits_full(hg, Wg)
    hr, Wr = h.bfloat16().float().requires_grad_(), W.bfloat16().float().requires_grad_()
    ref = hr @ Wr.t()
    _close(out, ref, 2e-2)
    probe = torch.randn(3, 40, 96, generator=g)
    (ref * probe.bfloat16().float()).sum().backward()
    (out * probe.to(DEV)).sum().backward()
    _close(hg.grad, hr.grad, 2e-2)
    _close(Wg.grad, Wr.grad, 2e-2)

    wq, wk, wv = (torch.randn(64, 48, generator=g) * 0.2 for _ in range(3))
    outs = K.k_qkv_dense(h.to(DEV), wq.to(DEV), wk.to(DEV), wv.to(DEV))
    for o, w in zip(outs, (wq, wk, wv)):
        _close(o, h.bfloat16().float() @ w.bfloat16().float(), 2e-2)

    wo = (torch.randn(64, 40, generator=g) * 0.2)
    rows = torch.tensor([8, 9, 10, 11, 12, 13, 14, 15, 40, 41, 42, 43, 44, 45, 46, 47])
    x = torch.randn(5, 7, 16, generator=g)
    xg, wog = x.to(DEV).requires_grad_(), wo.to(DEV).requires_grad_()
    out = K.k_out_proj_grouped(xg, wog, rows.to(DEV))
    xr, wor = x.bfloat16().float().requires_grad_(), wo.bfloat16().float().requires_grad_()
    ref = xr @ wor[rows, :]
    _close(out, ref, 2e-2)
    ref.sum().backward()
    out.sum().backward()
    _close(xg.grad, xr.grad, 2e-2)
    _close(wog.grad, wor.grad, 2e-2)
    assert (wog.grad.cpu()[:8] == 0).all()                    # unselected rows get an exact zero


def test_logits_shortlist_shape_values_and_grads():
    g = torch.Generator().manual_seed(6)
    h, W = torch.randn(2, 33, 64, generator=g), torch.randn(96, 64, generator=g) * 0.2
    sl = torch.stack([torch.randperm(96, generator=g)[:16] for _ in range(66)]).view(2, 33, 16)
    hg, Wg = h.to(DEV).requires_grad_(), W.to(DEV).requires_grad_()
    out = K.k_logits_shortlist(hg, Wg, sl.to(DEV))
    assert out.shape == (2, 33, 16)
    hr, Wr = h.bfloat16().float().requires_grad_(), W.bfloat16().float().requires_grad_()
    ref = (hr.unsqueeze(-2) * Wr[sl]).sum(-1)
    _close(out, ref, 2e-2)
    probe = torch.randn(2, 33, 16, generator=g).bfloat16().float()
    (ref * probe).sum().backward()
    (out * probe.to(DEV)).sum().backward()
    _close(hg.grad, hr.grad, 2e-2)
    _close(Wg.grad, Wr.grad, 2e-2)


def test_strict_cuda_and_status_contract():
    with pytest.raises(RuntimeError, match="strict_cuda"):
        K.k_fused_rmsnorm(torch.randn(2, 3, 4), torch.ones(4))
    st = K.backend_status()
    assert st["mode"] == "cuda_sm100a_ext" and st["uses_reference_fallback"] is False and st["cuda_available"]
    K.cuda_required()
    with pytest.raises(RuntimeError, match="strict_cuda"):
        K.k_swiglu_dense(torch.randn(4, 8), torch.randn(8, 8), torch.randn(8, 8), torch.randn(8, 8))
    with pytest.raises(ValueError):
        K.k_fused_rmsnorm(torch.randn(2, 8, device=DEV), torch.ones(4, device=DEV))


@pytest.mark.parametrize("N,d,m", [(50, 64, 64), (1500, 128, 192), (40, 64, 24)])
def test_packed_swiglu_ffn_matches_reference_math_and_grads(N, d, m):
    g = torch.Generator().manual_seed(N)
    x, wug, wdr = torch.randn(N, d, generator=g), torch.randn(2 * m, d, generator=g) * 0.2, torch.randn(m, d, generator=g) * 0.2
    L = [t.to(DEV).requires_grad_() for t in (x, wug, wdr)]
    out = K.triton_packed_swiglu_ffn(*L)
    R = [t.bfloat16().float().requires_grad_() for t in (x, wug, wdr)]
    up, gate = (R[0] @ R[1].t()).chunk(2, dim=-1)
    ref = (up * torch.nn.functional.silu(gate)) @ R[2]
    _close(out, ref, 2e-2)
    probe = torch.randn(N, d, generator=g)
    (ref * probe).sum().backward()
    (out * probe.to(DEV)).sum().backward()
    for a, b in zip(L, R):
        _close(a.grad, b.grad, 3e-2)
    with pytest.raises(ValueError):
        K.packed_swiglu_ffn(L[0], L[1][:-1], L[2])


def test_active_union_swiglu_evaluates_only_the_active_rows():
    g = torch.Generator().manual_seed(8)
    d, F_ = 64, 256
    x, wug, wd = torch.randn(3, 20, d, generator=g), torch.randn(2 * F_, d, generator=g) * 0.2, torch.randn(d, F_, generator=g) * 0.2
    ids = torch.randperm(F_, generator=g)[:64].repeat(2)             # duplicates collapse (layers.py:262)
    L = [t.to(DEV).requires_grad_() for t in (x, wug, wd)]
    out = K.active_union_swiglu(L[0], L[1], L[2], ids.to(DEV))
    R = [t.bfloat16().float().requires_grad_() for t in (x, wug, wd)]
    u = torch.unique(ids)
    ref = ((R[0] @ R[1][u].t()) * torch.nn.functional.silu(R[0] @ R[1][u + F_].t())) @ R[2].t()[u]
    _close(out, ref, 2e-2)
    ref.sum().backward()
    out.sum().backward()
    _close(L[1].grad, R[1].grad, 3e-2)
    _close(L[2].grad, R[2].grad, 3e-2)
    inactive = torch.ones(F_, dtype=torch.bool)
    inactive[u] = False
    assert (L[1].grad.cpu()[:F_][inactive] == 0).all()


def _ref_leaves(*ts):
    return [t.bfloat16().float().requires_grad_() for t in ts]


def test_swiglu_dense_and_grouped_match_reference_math_and_grads():
    """k_swiglu_dense / k_swiglu_grouped (kernels/reference.py:62-78), weights stored [in, out]."""
    g = torch.Generator().manual_seed(21)
    x, wu, wg, wd = (torch.randn(3, 20, 64, generator=g), torch.randn(64, 128, generator=g) * 0.2,
                     torch.randn(64, 128, generator=g) * 0.2, torch.randn(128, 64, generator=g) * 0.2)
    slabs = torch.cat([torch.arange(32, 64), torch.arange(96, 128)])
    for fn, extra, ref_fn in ((K.k_swiglu_dense, (), lambda X, U, G, D: (X @ U) * torch.nn.functional.silu(X @ G) @ D),
                              (K.k_swiglu_grouped, (slabs,),
                               lambda X, U, G, D: (X @ U[:, slabs]) * torch.nn.functional.silu(X @ G[:, slabs]) @ D[slabs, :])):
        L = [t.to(DEV).requires_grad_() for t in (x, wu, wg, wd)]
        out = fn(*L, *[e.to(DEV) for e in extra])
        R = _ref_leaves(x, wu, wg, wd)
        ref = ref_fn(*R)
        _close(out, ref, 2e-2)
        probe = torch.randn(ref.shape, generator=g)
        (ref * probe).sum().backward()
        (out * probe.to(DEV)).sum().backward()
        for a, b in zip(L, R):
            _close(a.grad, b.grad, 2.5e-2, 1e-4)


def test_qkv_grouped_matches_reference_math_and_grads():
    g = torch.Generator().manual_seed(22)
    x = torch.randn(2, 16, 64, generator=g)
    ws = [torch.randn(64, 64, generator=g) * 0.2 for _ in range(3)]
    cols = torch.cat([torch.arange(16, 32), torch.arange(48, 64)])
    L = [t.to(DEV).requires_grad_() for t in (x, *ws)]
    outs = K.k_qkv_grouped(*L, cols.to(DEV))
    R = _ref_leaves(x, *ws)
    refs = [R[0] @ w[:, cols] for w in R[1:]]
    probe = torch.randn(refs[0].shape, generator=g)
    for o, r in zip(outs, refs):
        _close(o, r, 2e-2)
    sum((r * probe).sum() for r in refs).backward()
    sum((o * probe.to(DEV)).sum() for o in outs).backward()
    for a, b in zip(L, R):
        _close(a.grad, b.grad, 2.5e-2, 1e-4)


def test_macro_phi_simplified_form_matches_reference_math():
    """k_macro_phi (kernels/reference.py:111-124)."""
    g = torch.Generator().manual_seed(23)
    B, S, d, m = 3, 16, 64, 16
    h, h0 = torch.randn(B, S, d, generator=g), torch.randn(B, S, d, generator=g)
    d_gain, bias = torch.randn(d, generator=g) * 0.1, torch.randn(d, generator=g) * 0.1
    v, u = torch.randn(3 * d, m, generator=g) * 0.1, torch.randn(m, d, generator=g) * 0.1
    out = K.k_macro_phi(*[t.to(DEV) for t in (h, h0, d_gain, v, u, bias)])
    normed = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5)
    z = torch.cat([normed, normed.mean(1, keepdim=True).expand_as(normed), h0], dim=-1)
    ref = h + d_gain * h + torch.nn.functional.silu(z @ v) @ u + bias
    _close(out, ref, 2e-2)


def test_pack_by_recipe_round_trip_and_grads():
    """k_pack_by_recipe / k_unpack_from_recipe (kernels/reference.py:91-108): stable order by (recipe, depth, audited)."""
    g = torch.Generator().manual_seed(24)
    hidden = torch.randn(10, 6, 8, generator=g)
    recipe = torch.tensor([2, 0, 1, 2, 0, 1, 1, 0, 2, 0])
    depth = torch.tensor([1, 2, 1, 1, 2, 0, 1, 1, 0, 2])
    hg = hidden.to(DEV).requires_grad_()
    packed = K.k_pack_by_recipe(hg, recipe.to(DEV), depth.to(DEV))
    keys = recipe * 1_000_000 + depth * 10
    order = torch.sort(keys, stable=True).indices
    assert torch.equal(packed.permutation.cpu(), order)
    assert torch.equal(packed.packed.detach().cpu(), hidden[order])
    assert torch.equal(packed.keys.cpu(), keys[order])
    assert packed.offsets[-1].item() == 10 and packed.unique_keys.numel() == packed.offsets.numel() - 1
    back = K.k_unpack_from_recipe(packed.packed, packed.inverse_permutation)
    assert torch.equal(back.detach().cpu(), hidden)
    probe = torch.randn(10, 6, 8, generator=g)
    (packed.packed * probe.to(DEV)).sum().backward()
    want = torch.empty_like(probe)
    want[order] = probe
    assert torch.equal(hg.grad.cpu(), want)
    mask = K.k_sample_audit_mask(torch.full((64,), 0.25, device=DEV), 5)
    assert mask.dtype == torch.bool and mask.shape == (64,)


@pytest.mark.parametrize("rows,V,dtype", [(5, 8, torch.bfloat16), (33, 1000, torch.bfloat16), (64, 2056, torch.bfloat16), (7, 2047, torch.bfloat16),
                                          (9, 32768, torch.bfloat16), (3, 65541, torch.bfloat16), (3, 8192, torch.bfloat16), (5, 8191, torch.bfloat16),
                                          (11, 3, torch.bfloat16), (17, 4, torch.float32), (33, 2047, torch.float32),
                                          (20, 4100, torch.float32), (4, 32772, torch.float32)])
def test_cross_entropy_row_widths(rows, V, dtype):
    """Widths around the register limits of the row kernel, and the rows that only the general kernel takes."""
    gen = torch.Generator().manual_seed(V)
    logits = (3 * torch.randn(rows, V, generator=gen)).to(dtype)
    targets = torch.randint(0, V, (rows,), generator=gen)
    targets[0], targets[-1] = V - 1, 0
    weight = torch.randn(rows, generator=gen)
    ref = logits.float().clone().requires_grad_(True)
    ref_loss = torch.nn.functional.cross_entropy(ref, targets, reduction="none")
    (ref_loss * weight).sum().backward()
    x = logits.cuda().requires_grad_(True)
    loss = K.k_cross_entropy_unreduced(x, targets.cuda())
    (loss * weight.cuda()).sum().backward()
    assert torch.allclose(loss.cpu(), ref_loss, atol=1e-4, rtol=1e-5)
    assert torch.allclose(x.grad.cpu().float(), ref.grad, atol=1e-5, rtol=1e-2 if dtype == torch.bfloat16 else 1e-4)


@pytest.mark.parametrize("dtype,V", [(torch.float32, 4096), (torch.bfloat16, 8192), (torch.float32, 9000)])
def test_cross_entropy_whose_saved_logits_come_back_on_another_boundary(dtype, V):
    """Logits off the 16-byte boundary whose saved copy (`save_on_cpu`) returns on it: rows of just that length are too long for one
    kernel in forward and not in backward.  The same gradients as without the hooks."""
    g = torch.Generator().manual_seed(V)
    rows = 37
    buf = torch.empty(rows * V + 1, dtype=dtype, device=DEV)
    x = buf[1:].view(rows, V)
    x.copy_(torch.randn(rows, V, generator=g) * 3)
    x.requires_grad_()
    targets, w = torch.randint(0, V, (rows,), generator=g).to(DEV), torch.randn(rows, generator=g).to(DEV)
    want, = torch.autograd.grad(K.k_cross_entropy_unreduced(x, targets), x, w)
    with torch.autograd.graph.save_on_cpu():
        loss = K.k_cross_entropy_unreduced(x, targets)
    got, = torch.autograd.grad(loss, x, w)
    _close(got, want.cpu(), 1e-6 if dtype == torch.float32 else 2 ** -8)       # (one rounding of the result; the sums' order may differ)


@pytest.mark.parametrize("V,dtype", [(512, torch.bfloat16), (511, torch.bfloat16), (8192, torch.bfloat16), (9001, torch.bfloat16), (16384, torch.bfloat16),
                                     (512, torch.float32), (4099, torch.float32), (8192, torch.float32)])
@pytest.mark.parametrize("level,fill", [(0.0, "-inf"), (-300.0, "-inf"), (0.0, "lowest")])
def test_cross_entropy_of_masked_and_nan_columns(V, dtype, level, fill):
    """Rows whose unmasked logits sit in one thread's, one warp's or half of the columns, at zero and far below it: the masked
    columns' gradient is exactly zero, loss and gradient are the plain row's.  A block of NaN logits makes the loss NaN."""
    gen = torch.Generator().manual_seed(V)
    keeps = [(0, 4), (0, V // 2), (V // 2, V), (V - 3, V)]
    x = (level + torch.randn(len(keeps), V, generator=gen)).to(dtype)
    targets = torch.tensor([b - 1 for _, b in keeps])
    fill = -torch.inf if fill == "-inf" else torch.finfo(dtype).min
    for r, (a, b) in enumerate(keeps):
        x[r, :a] = x[r, b:] = fill
    ref = x.float().clone().requires_grad_(True)
    loss = torch.nn.functional.cross_entropy(ref, targets, reduction="none")
    loss.sum().backward()
    got = x.cuda().requires_grad_(True)
    out = K.k_cross_entropy_unreduced(got, targets.cuda())
    out.sum().backward()
    assert torch.allclose(out.detach().cpu(), loss.detach(), atol=1e-4, rtol=1e-5)
    g = got.grad.cpu().float()
    assert (g[x == fill] == 0).all() and torch.allclose(g, ref.grad, atol=1e-5, rtol=1e-2 if dtype == torch.bfloat16 else 1e-4)
    bad = x.clone()
    bad[x == fill] = torch.nan
    assert K.k_cross_entropy_unreduced(bad.cuda(), targets.cuda()).isnan().all()


@pytest.mark.parametrize("d", [4, 132, 512, 2048])
@pytest.mark.parametrize("xt,wt,rt", [(torch.bfloat16, torch.bfloat16, None), (torch.bfloat16, torch.float32, torch.float32), (torch.float32, torch.bfloat16, torch.bfloat16),
                                      (torch.float16, torch.float32, None)])
def test_rmsnorm_row_widths_and_types(d, xt, wt, rt):
    gen = torch.Generator().manual_seed(d)
    x, w, g = torch.randn(11, d, generator=gen).to(xt), torch.randn(d, generator=gen).to(wt), torch.randn(11, d, generator=gen)
    r = torch.randn(11, d, generator=gen).to(rt) if rt is not None else None
    leaves = [t.float().requires_grad_(True) for t in (x, w) + ((r,) if r is not None else ())]
    y = leaves[0] + leaves[2] if r is not None else leaves[0]
    ref = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * leaves[1]
    (ref * g).sum().backward()
    dev = [t.detach().cuda().requires_grad_(True) for t in (x, w) + ((r,) if r is not None else ())]
    out, total = K.k_fused_rmsnorm(dev[0], dev[1], dev[2] if r is not None else None)
    assert out.dtype == torch.result_type(x, w) and (total is None) == (r is None)
    (out.float() * g.cuda()).sum().backward()
    tol = 2e-2 if torch.bfloat16 in (out.dtype, xt, wt, rt) else 2e-3 if xt == torch.float16 else 1e-5
    assert torch.allclose(out.cpu().float(), ref.detach(), atol=tol, rtol=tol)
    if r is not None:
        assert total.dtype == torch.result_type(x, r) and torch.allclose(total.cpu().float(), y.detach(), atol=tol, rtol=tol)
    for a, b in zip(dev, leaves):
        assert a.grad.dtype == a.dtype and torch.allclose(a.grad.cpu().float(), b.grad, atol=tol * max(1.0, b.grad.abs().max().item()), rtol=tol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("layout", ["heads_first", "tokens_first", "odd_offset"])
def test_rope_and_attention_take_strided_views(layout, dtype):
    """q, k, v as a projection leaves them ([B, S, H, hd] transposed), contiguous, and on no 16-byte boundary."""
    B, H, S, hd = 2, 3, 37, 16
    gen = torch.Generator().manual_seed(0)
    base = [torch.randn(B, H, S, hd, generator=gen).to(dtype) for _ in range(3)]

    def place(t):
        t = t.cuda()
        if layout == "tokens_first":
            return t.transpose(1, 2).contiguous().transpose(1, 2)
        if layout == "odd_offset":
            return torch.cat([t.new_zeros(B, H, S, 1), t], dim=-1)[..., 1:]
        return t

    ang = torch.randn(S, hd, generator=gen)
    cos, sin = ang.cos(), ang.sin()
    rot = lambda t: torch.stack([-t[..., 1::2], t[..., 0::2]], -1).flatten(-2)  # noqa: E731
    q, k, v = (place(t) for t in base)
    rq, rk = K.k_rope_apply(q, k, cos.cuda(), sin.cuda())
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-5
    for got, t in ((rq, base[0]), (rk, base[1])):
        assert got.is_contiguous() and torch.allclose(got.cpu().float(), t.float() * cos + rot(t.float()) * sin, atol=tol, rtol=tol)
    out = K.k_flash_causal_dense(q, k, v)
    ref = torch.nn.functional.scaled_dot_product_attention(*(t.bfloat16().float() for t in base), is_causal=True)
    assert out.dtype == dtype and torch.allclose(out.cpu().float(), ref, atol=3e-2, rtol=3e-2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gradients_off_the_16_byte_grid(dtype):
    """A gradient that is a contiguous view one element into its buffer: the results of an aligned one."""
    gen = torch.Generator().manual_seed(1)

    def both(run, shape):
        base = torch.randn(shape, generator=gen).to(dtype).cuda()
        odd = torch.cat([base.new_zeros(1), base.view(-1)])[1:].view(shape)
        assert odd.data_ptr() % 16 and odd.is_contiguous()
        for a, b in zip(run(base), run(odd)):
            assert torch.equal(a, b)

    x, w, r = (torch.randn(*s, generator=gen).to(dtype).cuda().requires_grad_() for s in ((9, 64), (64,), (9, 64)))
    out, total = K.k_fused_rmsnorm(x, w, r)
    both(lambda g: torch.autograd.grad((out, total), (x, w, r), (g, g), retain_graph=True), (9, 64))
    q, k, v = (torch.randn(2, 33, 3, 32, generator=gen).to(dtype).cuda().transpose(1, 2).requires_grad_() for _ in range(3))
    y = K.k_flash_causal_dense(q, k, v).transpose(1, 2)
    both(lambda g: torch.autograd.grad(y, (q, k, v), g, retain_graph=True), (2, 33, 3, 32))


@pytest.mark.parametrize("hq,hk,kt", [(3, 3, torch.float32), (8, 2, torch.float32), (4, 4, torch.bfloat16)])
@pytest.mark.parametrize("used", ["q", "k", "both"])
def test_rope_gradient_through_either_output(hq, hk, kt, used):
    """q and k with equal and unequal head counts and types; the input of an output that no loss used gets zeros."""
    gen = torch.Generator().manual_seed(hq)
    q, k = torch.randn(2, hq, 7, 16, generator=gen), torch.randn(2, hk, 7, 16, generator=gen).to(kt)
    ang = torch.randn(7, 16, generator=gen)
    probes = [torch.randn(t.shape, generator=gen) for t in (q, k)]
    rot = lambda t: torch.stack([-t[..., 1::2], t[..., 0::2]], -1).flatten(-2)  # noqa: E731
    ref = [t.float().requires_grad_() for t in (q, k)]
    sum((((t * ang.cos() + rot(t) * ang.sin()) * p).sum() for t, p in zip(ref, probes))).backward()
    dev = [t.cuda().requires_grad_() for t in (q, k)]
    outs = K.k_rope_apply(*dev, ang.cos().cuda(), ang.sin().cuda())
    terms = [(o.float() * p.cuda()).sum() for o, p in zip(outs, probes)]
    grads = torch.autograd.grad(sum(t for t, n in zip(terms, "qk") if used in (n, "both")), dev)
    for g, t, n in zip(grads, ref, "qk"):
        want = t.grad if used in (n, "both") else torch.zeros_like(t)
        tol = 2e-2 if g.dtype == torch.bfloat16 else 1e-5
        assert g.shape == t.shape and torch.allclose(g.cpu().float(), want, atol=tol, rtol=tol)


def test_empty_rows_and_columns():
    """No columns, positions or head columns: an error in Python (the host divides by them).  No rows: empty results and
    zero parameter gradients."""
    e = lambda *s: torch.zeros(*s, device=DEV)  # noqa: E731
    with pytest.raises(ValueError, match="k_fused_rmsnorm"):
        K.k_fused_rmsnorm(e(3, 0), e(0))
    for shape in ((2, 3, 0, 8), (2, 3, 5, 0), (0, 8), (1, 2, 3, 0, 8), (1, 2, 3, 5, 0)):
        with pytest.raises(ValueError, match="k_rope_apply"):
            K.k_rope_apply(e(*shape), e(*shape), e(*shape[-2:]), e(*shape[-2:]))
    x, w = e(0, 64).requires_grad_(), torch.ones(64, device=DEV, requires_grad=True)
    out, _ = K.k_fused_rmsnorm(x, w)
    out.sum().backward()
    assert out.shape == x.grad.shape == (0, 64) and (w.grad == 0).all()


def test_a_refused_launch_raises_rte_error_forward_and_backward():
    from speedup_thingy_b200._abi import RteError
    wide = torch.zeros(3, 4096, device=DEV)
    with pytest.raises(RteError, match="rte_rmsnorm_op_fwd failed"):
        K.k_fused_rmsnorm(wide, wide[0])
    x, w = (torch.zeros(16, 16, dtype=torch.bfloat16, device=DEV, requires_grad=True) for _ in range(2))
    odd = torch.zeros(16 * 16 + 1, dtype=torch.bfloat16, device=DEV)[1:].view(16, 16)        # a product's operand off 16 bytes
    with pytest.raises(RteError, match="rte_gemm_bf16 failed"):
        K.k_logits_full(x, w).backward(odd)
    with pytest.raises(RteError, match="rte_gemm_bf16 failed"):
        K.k_logits_full(odd, w)


@pytest.mark.parametrize("N,d,m", [(5901, 64, 2048), (5800, 64, 2048)])
def test_packed_swiglu_on_both_sides_of_the_fusion_rule(N, d, m):
    gen = torch.Generator().manual_seed(N)
    x, wug, wd = (0.2 * torch.randn(*s, generator=gen) for s in ((N, d), (2 * m, d), (m, d)))
    g = torch.randn(N, d, generator=gen)
    res = []
    for dev in ("cpu", "cuda"):
        t = [a.to(dev).detach().clone().requires_grad_(True) for a in (x, wug, wd)]
        if dev == "cuda":
            y = K.packed_swiglu_ffn(*t)
        else:
            ug = t[0] @ t[1].t()
            y = (ug[:, :m] * torch.nn.functional.silu(ug[:, m:])) @ t[2]
        (y * g.to(dev)).sum().backward()
        res.append([y.detach().cpu()] + [a.grad.cpu() for a in t])
    for a, b in zip(*res):
        assert (a - b).norm() <= 1e-2 * a.norm()


def test_products_of_an_odd_width_write_fp32_rows():
    x, w = torch.randn(70, 64, device="cuda"), torch.randn(2047, 64, device="cuda")
    ref = x.bfloat16().float() @ w.bfloat16().float().t()
    got = K.k_logits_full(x, w)
    assert got.dtype == torch.float32 and torch.allclose(got, ref, atol=1e-3, rtol=1e-3)
