"""SVD-factor sparse FFN on a B200 (`speedup_thingy_b200.svd_ffn`) against the oracle and the reference-generated
golden case.  Selections are bit-exact given the scores (checked with constructed ties and by replaying the
kernel's own inputs through the oracle, allowing differences only within float rounding of the threshold);
values within 2e-2 of the output scale (bf16 arithmetic)."""
from pathlib import Path

import numpy as np
import pytest
import torch

from oracle import rte_oracle as O
from speedup_thingy_b200.ops import CudaOps
from speedup_thingy_b200.svd_ffn import SVDFactorSparseFFN, svd_sparse_ffn
from tests.golden.cases import SVD_FFN, svd_ffn_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GOLD = np.load(Path(__file__).resolve().parent / "golden" / "svd_ffn.npz")


def _close(a, b, rel=2e-2):
    a, b = a.detach().float().cpu(), torch.as_tensor(b).float()
    assert a.shape == b.shape
    err = (a - b).abs().max().item()
    assert err <= rel * b.abs().max().item() + 1e-6, (err, b.abs().max().item())


@pytest.mark.parametrize("rows,F_,k", [(9, 64, 8), (33, 2048, 256), (5, 100, 100), (7, 4096, 1)])
def test_radix_select_is_the_stable_topk_with_constructed_ties(rows, F_, k):
    """up_m = top_k = k with zero gates: candidates = top-k of |up_hat| and every candidate ties at score 0 in
    the re-rank, so `selected` must be exactly the lowest-index top-k of |up_hat|."""
    ops = CudaOps(DEV)
    g = torch.Generator().manual_seed(F_ + k)
    uh = (torch.randn(rows, F_, generator=g) * 3).round() / 2                       # heavy ties
    uh[0] = 1.0                                                                      # all-equal row
    hats = torch.cat([uh, torch.zeros(rows, F_)], dim=1)
    ug = torch.cat([torch.ones(rows, F_), torch.zeros(rows, F_)], dim=1).bfloat16()
    z = torch.empty(rows, F_, dtype=torch.bfloat16, device=DEV)
    sel = torch.empty(rows, F_, dtype=torch.uint8, device=DEV)
    cnt = torch.empty(rows, dtype=torch.int32, device=DEV)
    ops.svd_ffn_select(hats.to(DEV), ug.to(DEV), torch.ones(F_, device=DEV), z, sel, cnt, up_m=k, gate_m=0, product_m=0, top_k=k)
    torch.cuda.synchronize()
    want = O.topk_membership(uh.abs(), k)
    assert torch.equal(sel.cpu().bool(), want)
    assert (cnt.cpu() == k).all() and (z.cpu() == 0).all()


@pytest.mark.parametrize("rows,F_,k", [(5000, 104, 13), (3, 4, 1), (64, 2048, 2047), (40, 9984, 700), (2500, 256, 256)])
def test_threshold_search_selects_the_k_largest_in_every_row(rows, F_, k):
    """The threshold search over many tokens per warp: rows of continuous scores (it ends on a probe or by ranking the
    last few keys), rows of two values (more equal keys than it ranks) and rows of very different scale in turn."""
    ops = CudaOps(DEV)
    g = torch.Generator().manual_seed(rows + F_)
    uh = torch.randn(rows, F_, generator=g) * torch.logspace(-6, 6, rows).roll(rows // 2).unsqueeze(1)
    uh[::3] = (uh[::3] > 0).float()
    hats = torch.cat([uh, torch.zeros(rows, F_)], dim=1)
    ug = torch.cat([uh, torch.ones(rows, F_)], dim=1).bfloat16()
    z = torch.empty(rows, F_, dtype=torch.bfloat16, device=DEV)
    sel = torch.empty(rows, F_, dtype=torch.uint8, device=DEV)
    cnt = torch.empty(rows, dtype=torch.int32, device=DEV)
    ops.svd_ffn_select(hats.to(DEV), ug.to(DEV), torch.ones(F_, device=DEV), z, sel, cnt, up_m=k, gate_m=0, product_m=0, top_k=k)
    torch.cuda.synchronize()
    want = O.topk_membership(uh.abs(), k)
    assert torch.equal(sel.cpu().bool(), want) and (cnt.cpu() == k).all()
    assert torch.equal(z.cpu() != 0, want & (ug[:, :F_] != 0))


@pytest.mark.parametrize("rows,F_,k", [(40, 2048, 256), (9, 132, 40), (600, 1024, 3)])
def test_scores_that_share_their_upper_bits(rows, F_, k):
    """More scores than the ranking list holds between two neighbouring keys, different below, some equal; an infinite score and
    one that is not a number rank first, in that order from the top: NaN, infinity."""
    ops = CudaOps(DEV)
    g = torch.Generator().manual_seed(rows + F_)
    uh = 1.0 + torch.randint(0, 500, (rows, F_), generator=g) * 2.0 ** -20
    uh[1::2, : F_ // 2] *= 4.0
    uh[0, 7], uh[0, 3] = float("nan"), float("inf")
    hats = torch.cat([uh, torch.zeros(rows, F_)], dim=1)
    ug = torch.cat([torch.ones(rows, F_), torch.zeros(rows, F_)], dim=1).bfloat16()
    z, sel = torch.empty(rows, F_, dtype=torch.bfloat16, device=DEV), torch.empty(rows, F_, dtype=torch.uint8, device=DEV)
    ops.svd_ffn_select(hats.to(DEV), ug.to(DEV), torch.ones(F_, device=DEV), z, sel, None, up_m=k, gate_m=0, product_m=0, top_k=k)
    torch.cuda.synchronize()
    order = uh.clone()
    order[0, 7], order[0, 3] = 1e30, 1e29
    assert torch.equal(sel.cpu().bool(), O.topk_membership(order, k))


def test_z_of_every_gate_has_the_bits_of_the_swiglu_pass():
    """Everything selected: z over all 65536 bf16 gates against rte_swiglu_fwd, whose divide rounds correctly.  Gates from -88.7 to
    -87.3 among them, whose denominators are above 2^126."""
    ops = CudaOps(DEV)
    F_ = 2048
    gate = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).view(32, F_)
    ups = torch.randn(3, F_, generator=torch.Generator().manual_seed(0)).bfloat16()
    ug = torch.cat([torch.cat([torch.full_like(u, 1.0) * u for u in ups.unsqueeze(1).expand(3, 32, F_)]), gate.repeat(3, 1)], dim=1).to(DEV)
    z, want = (torch.empty(96, F_, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    ops.svd_ffn_select(torch.ones(96, 2 * F_, device=DEV), ug, torch.ones(F_, device=DEV), z, None, None, up_m=F_, gate_m=0, product_m=0, top_k=F_)
    ops.swiglu_fwd(ug, want, 96, F_)
    assert torch.equal(z.isnan(), want.isnan())
    keep = ~want.isnan()
    assert torch.equal(z.view(torch.int16)[keep], want.view(torch.int16)[keep])


@pytest.mark.parametrize("gate_m,product_m", [(20, 0), (0, 20)])
def test_scores_of_gates_far_below_zero_keep_their_order(gate_m, product_m):
    """Gates whose exp(-gate) is finite and above 2^126: |silu| shrinks by at least 1 % from one to the next, so the largest are known."""
    ops = CudaOps(DEV)
    rows, F_ = 40, 128
    place = torch.stack([torch.randperm(F_, generator=torch.Generator().manual_seed(i)) for i in range(rows)])
    gate = (-87.4 - 0.01 * torch.arange(F_)).expand(rows, F_).gather(1, place)
    hats = torch.cat([torch.full((rows, F_), 2.0), gate], dim=1).to(DEV)
    ug = torch.ones(rows, 2 * F_, dtype=torch.bfloat16, device=DEV)
    z, sel = torch.empty(rows, F_, dtype=torch.bfloat16, device=DEV), torch.empty(rows, F_, dtype=torch.uint8, device=DEV)
    ops.svd_ffn_select(hats, ug, torch.ones(F_, device=DEV), z, sel, None, up_m=0, gate_m=gate_m, product_m=product_m, top_k=20)
    ops.check_status()
    assert torch.equal(sel.cpu().bool(), place < 20)


@pytest.mark.parametrize("rows,F_,up_m,gate_m,product_m,top_k", [
    (60, 2048, 300, 280, 310, 256),                  # three lists, more candidates than are selected
    (300, 132, 40, 30, 20, 25),                      # F % 8 == 4
    (50, 260, 90, 0, 60, 64), (50, 260, 0, 70, 0, 33), (50, 1028, 120, 40, 0, 100),       # a list or two missing
    (3700, 64, 20, 20, 20, 7),                       # several tokens per warp
    (40, 128, 128, 0, 5, 60), (33, 4, 3, 2, 2, 2),   # everything a candidate; one group of four
])
@pytest.mark.parametrize("spread", [False, True])
def test_selection_is_bit_exact_over_all_lists(rows, F_, up_m, gate_m, product_m, top_k, spread):
    """Selected neurons and candidate counts against the oracle in 64 bits, where no score hangs on a last bit: four gates whose SiLU differ by
    more than 0.2 % from one another's multiples, norms that are powers of two, ups of two mantissa bits -- so scores are equal or far
    apart, and many more than 32 share a key and a score across every cut.  `spread`: bf16 ups of all mantissas in rows of one gate."""
    ops = CudaOps(DEV)
    g = torch.Generator().manual_seed(F_ + top_k)
    gates = torch.tensor([1.0, 20.0, -3.0, 0.0])
    pick = lambda *s: torch.randint(0, s[0], s[1:], generator=g)  # noqa: E731

    def side():
        sign = 1 - 2 * pick(2, rows, F_).float()
        if spread:
            return torch.randn(rows, F_, generator=g).bfloat16().float(), gates[pick(3, rows, 1)].expand(rows, F_)
        return sign * (1 + pick(4, rows, F_) * 0.25) * 2.0 ** pick(3, rows, F_), gates[pick(4, rows, F_)]

    (uh, gh), (up, gate) = side(), side()
    wn = 2.0 ** pick(3, F_).float()
    hats, ug = torch.cat([uh, gh], dim=1).to(DEV), torch.cat([up, gate], dim=1).bfloat16().to(DEV)
    z, sel = torch.empty(rows, F_, dtype=torch.bfloat16, device=DEV), torch.empty(rows, F_, dtype=torch.uint8, device=DEV)
    cnt = torch.empty(rows, dtype=torch.int32, device=DEV)
    ops.svd_ffn_select(hats, ug, wn.to(DEV), z, sel, cnt, up_m=up_m, gate_m=gate_m, product_m=product_m, top_k=top_k)
    ops.check_status()
    cand = O.svd_ffn_candidates(uh.double(), gh.double(), wn.double(), up_m, gate_m, product_m)
    zd = up.double() * torch.nn.functional.silu(gate.double())
    want = O.svd_ffn_select(zd, cand, wn.double(), top_k)
    assert torch.equal(cnt.cpu().long(), cand.sum(-1))
    assert torch.equal(sel.cpu().bool(), want)
    assert torch.equal(z.cpu() != 0, want & (zd != 0))


@pytest.mark.parametrize("rows,F_", [(37, 2048), (5, 100)])            # eight neurons per thread | one
def test_swiglu_backward_of_the_selected_neurons(rows, F_):
    ops = CudaOps(DEV)
    g = torch.Generator().manual_seed(F_)
    ug, dz = (torch.randn(rows, n, generator=g).bfloat16() for n in (2 * F_, F_))
    sel = torch.rand(rows, F_, generator=g) < 0.15
    dug = torch.empty(rows, 2 * F_, dtype=torch.bfloat16, device=DEV)
    ops.svd_ffn_swiglu_bwd(ug.to(DEV), dz.to(DEV), sel.to(torch.uint8).to(DEV), dug)
    leaf = ug.float().requires_grad_()
    (leaf[:, :F_] * torch.nn.functional.silu(leaf[:, F_:]) * sel * dz.float()).sum().backward()
    _close(dug, leaf.grad)
    assert (dug.cpu().view(rows, 2, F_)[~sel.unsqueeze(1).expand(rows, 2, F_)] == 0).all()


def _module(t, c, max_tokens):
    dev = lambda k: t[k].to(DEV)  # noqa: E731
    return SVDFactorSparseFFN(dev("w_up"), dev("w_gate"), dev("w_down"), t["up_a"], t["up_b"], t["gate_a"], t["gate_b"],
                              top_k=c["top_k"], up_m=c["up_m"], gate_m=c["gate_m"], product_m=c["product_m"], max_tokens=max_tokens)


def _replay_selection(m, N, c):
    """The oracle's selection on the kernel's own inputs; returns (oracle mask, mask of threshold-margin entries)."""
    hats, ug, wn = m.hats[:N].cpu(), m.ug[:N].cpu().float(), m.wn.cpu()
    F_ = m.F
    cand = O.svd_ffn_candidates(hats[:, :F_], hats[:, F_:], wn, c["up_m"], c["gate_m"], c["product_m"])
    z = ug[:, :F_] * torch.nn.functional.silu(ug[:, F_:])
    return O.svd_ffn_select(z, cand, wn, c["top_k"]), cand


def test_golden_case_selection_values_and_gradients():
    c, t = SVD_FFN, svd_ffn_inputs()
    m = _module(t, c, 64)
    x = t["x"].to(DEV).requires_grad_()
    for w in (m.w_up, m.w_gate, m.w_down):
        w.requires_grad_()
    out = svd_sparse_ffn(m, x)
    (out * t["probe"].to(DEV)).sum().backward()
    m.ops.check_status()
    N = 33
    sel = m.selected[:N].cpu().bool()
    assert (sel.sum(-1) == c["top_k"]).all()
    want, _ = _replay_selection(m, N, c)
    assert (sel != want).float().mean() < 2e-3                      # only float-rounding swaps at a threshold
    gold_sel = torch.from_numpy(GOLD["selected"])
    assert (sel & gold_sel).sum() >= 0.9 * gold_sel.sum()           # bf16 scores vs the reference's fp32 scores
    # values: the oracle with the kernel's selection injected
    L = {k: t[k].bfloat16().float().requires_grad_() for k in ("x", "w_up", "w_gate", "w_down")}
    ref, _ = O.svd_sparse_ffn(L["x"], L["w_up"], L["w_gate"], L["w_down"], t["up_a"], t["up_b"], t["gate_a"], t["gate_b"],
                              top_k=c["top_k"], up_m=c["up_m"], gate_m=c["gate_m"], product_m=c["product_m"], selected=sel)
    (ref * t["probe"]).sum().backward()
    _close(out, ref.detach())
    _close(x.grad, L["x"].grad)
    _close(m.w_up.grad, L["w_up"].grad)
    _close(m.w_gate.grad, L["w_gate"].grad)
    _close(m.w_down.grad, L["w_down"].grad)
    never = ~sel.any(0)
    assert (m.w_down.grad.cpu()[never] == 0).all() and (m.w_up.grad.cpu()[never] == 0).all()


def test_c4_shaped_module_against_the_oracle():
    """d 512, F 2048, rank 128, top_k 256, up_m = gate_m = product_m = 256 on 2048 tokens."""
    c = dict(top_k=256, up_m=256, gate_m=256, product_m=256)
    g = torch.Generator().manual_seed(4)
    N, d, F_, r = 2048, 512, 2048, 128
    rn = lambda *s, scale: torch.randn(*s, generator=g) * scale  # noqa: E731
    t = dict(w_up=rn(F_, d, scale=0.044), w_gate=rn(F_, d, scale=0.044), w_down=rn(F_, d, scale=0.044),
             up_a=rn(d, r, scale=0.044), up_b=rn(r, F_, scale=0.09), gate_a=rn(d, r, scale=0.044), gate_b=rn(r, F_, scale=0.09))
    m = _module(t, c, N)
    x = rn(N, d, scale=1.0)
    out = m.forward(x.to(DEV))
    m.ops.check_status()
    sel = m.selected[:N].cpu().bool()
    assert (sel.sum(-1) == 256).all()
    want, cand = _replay_selection(m, N, c)
    assert (sel != want).float().mean() < 1e-3
    assert abs(m.avg_candidate_size - float(cand.sum(-1).float().mean())) < 2.0
    xr = x.bfloat16().float()
    ref, _ = O.svd_sparse_ffn(xr, t["w_up"].bfloat16().float(), t["w_gate"].bfloat16().float(), t["w_down"].bfloat16().float(),
                              t["up_a"], t["up_b"], t["gate_a"], t["gate_b"], selected=sel, **c)
    _close(out, ref)
    # and the fp32 oracle's own selection overlaps almost everywhere
    _, sel32 = O.svd_sparse_ffn(x, t["w_up"], t["w_gate"], t["w_down"], t["up_a"], t["up_b"], t["gate_a"], t["gate_b"], **c)
    assert (sel & sel32).sum() >= 0.93 * sel32.sum()


@pytest.mark.parametrize("N,F_", [(300, 512), (700, 2048), (513, 2064)])          # below and above a million activations
def test_module_backward_rounds_like_the_two_launches_at_every_size(N, F_):
    """Whichever route the size takes, the hidden gradients are those of the product with a bf16 result and the masked SwiGLU pass.  Integer
    gradients and down weights: d z is exact before it is rounded."""
    d, r, k = 128, 16, 40
    g = torch.Generator().manual_seed(N)
    rn = lambda *s: torch.randn(*s, generator=g) * 0.1  # noqa: E731
    w_down = torch.randint(-8, 9, (F_, d), generator=g).float()
    t = dict(w_up=rn(F_, d), w_gate=rn(F_, d), w_down=w_down, up_a=rn(d, r), up_b=rn(r, F_), gate_a=rn(d, r), gate_b=rn(r, F_))
    m = _module(t, dict(top_k=k, up_m=k, gate_m=k, product_m=k), N)
    m.forward(torch.randn(N, d, generator=g).to(DEV))
    dout = torch.randint(-8, 9, (N, d), generator=g).float().to(DEV)
    m.backward(dout, *(torch.empty(F_, d, device=DEV) for _ in range(3)))
    dz, want = torch.empty(N, F_, dtype=torch.bfloat16, device=DEV), torch.empty(N, 2 * F_, dtype=torch.bfloat16, device=DEV)
    m.ops.gemm(dout.bfloat16(), m.wd16, dz, M=N, N=F_, K=d)
    m.ops.svd_ffn_swiglu_bwd(m.ug[:N], dz, m.selected[:N], want)
    m.ops.check_status()
    assert torch.equal(m.dug[:N], want)


def test_what_the_buffers_cannot_hold_is_refused_before_a_launch():
    c, t = SVD_FFN, svd_ffn_inputs()
    m = _module(t, c, 64)
    x = t["x"].to(DEV)
    want = m.forward(x)
    for name in ("w_up", "w_gate", "w_down"):
        good = getattr(m, name)
        for bad in (good.bfloat16(), good.cpu(), good.t(), good[:-1]):
            setattr(m, name, bad)
            with pytest.raises(ValueError, match=name):
                m.forward(x)
        setattr(m, name, good)
    with pytest.raises(ValueError, match="last dimension"):
        m.forward(x.reshape(-1, m.d)[:32].reshape(16, 2 * m.d))
    assert torch.equal(m.forward(x), want)
    dw = [torch.empty_like(m.w_up) for _ in range(3)]
    with pytest.raises(ValueError, match="rows"):
        m.backward(want.reshape(-1, m.d)[:-1], *dw)
    with pytest.raises(ValueError, match="dw_down"):
        m.backward(want, dw[0], dw[1], dw[2].bfloat16())
    m.backward(want, *dw)
    m.ops.check_status()
