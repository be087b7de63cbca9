"""The pairwise tcgen05 kernels (FASTMAX_FLAG_PAIRWISE) against the CPU oracle at the sizes where they can go wrong: one row,
the edges of the 128-row tiles and of the 256-row forward items, one item per block and many, an absent second tile, keys
without queries, both forms of the polynomial (square completed or not), outputs the copy engine cannot write."""
import math

import numpy as np
import pytest
import torch

from oracle import fastmax_oracle as orc

pytestmark = pytest.mark.gpu


def host(t):
    return t.detach().float().cpu().numpy().astype(np.float64)


CASES = [  # B, H, nq, nk, D, causal, order
    (1, 2, 1, 1, 64, False, 2),
    (1, 2, 2, 5, 16, True, 2),
    (2, 2, 127, 127, 32, True, 2),
    (1, 2, 128, 128, 64, True, 2),
    (1, 2, 129, 129, 64, True, 1),
    (1, 2, 256, 257, 64, True, 2),
    (1, 2, 257, 129, 64, False, 2),
    (1, 3, 385, 640, 32, True, 2),
    (1, 2, 640, 64, 16, False, 1),
    (4, 40, 200, 200, 64, True, 2),    # more items than SMs, second tile ragged
    (10, 40, 100, 100, 32, False, 2),  # items of one tile, several per block
    (2, 2, 1100, 1100, 64, True, 2),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("poly", [(1.0, 1.0, 0.5), (1.0, 0.9, 0.01)])   # square completed; general form
@pytest.mark.parametrize("case", CASES)
def test_pairwise_kernels_match_oracle(case, poly, dtype):
    from reproducing_fastmax_results_b200 import _lib as L

    B, H, nq, nk, D, causal, order = case
    g = torch.Generator(device="cuda").manual_seed(nq + nk + D)
    # head-split views of (b, n, h*d) buffers
    mk = lambda n: torch.randn(B, n, H, D, device="cuda", generator=g).to(dtype).transpose(1, 2)
    q, do, k, v = mk(nq), mk(nq), mk(nk), mk(nk)
    p = orc.Poly(*poly, 1.0 / (8.0 * math.sqrt(D)), order)
    args = (causal, p.inv_temp, p.a0, p.a1, p.a2, order)
    o, gg, _ = L.forward(q, k, v, *args, flags=L.FLAG_PAIRWISE)
    dq, dk, dv, _ = L.backward(q, k, v, o, gg, do, *args, flags=L.FLAG_PAIRWISE)
    L.check_status()
    assert L.wait_histogram() == {}
    for b, h in {(0, 0), (B - 1, H - 1)}:
        a = [host(t[b, h]) for t in (q, k, v, do)]
        o_ref, g_ref = orc.fastmax_naive(a[0], a[1], a[2], causal, p)
        refs = (o_ref, g_ref) + tuple(orc.fastmax_naive_grads(a[0], a[1], a[2], a[3], causal, p))
        for name, x, r, tol in zip(("o", "g", "dq", "dk", "dv"), (o, gg, dq, dk, dv), refs,
                                   (2e-2, 2e-3, 2e-2, 2e-2, 2e-2) if dtype == torch.bfloat16 else (5e-6,) * 5):
            if np.abs(r).max() > 1e-9:   # dq and dk of a single visible key are analytically zero
                assert orc.max_norm_err(host(x[b, h]), r) < tol, (name, b, h)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_pairwise_outputs_in_rows_the_copy_engine_cannot_write(dtype):
    from reproducing_fastmax_results_b200 import _lib as L

    B, H, N, D = 1, 3, 300, 64
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k, v, do = (torch.randn(B, H, N, D, device="cuda", generator=g).to(dtype) for _ in range(4))
    odd = lambda: torch.zeros(B, H, N, D + 1, device="cuda", dtype=dtype)
    bufs = [odd() for _ in range(4)]
    views = [t[..., :D] for t in bufs]
    o, gg, _ = L.forward(q, k, v, True, 0.05, order=2, flags=L.FLAG_PAIRWISE)
    grads = L.backward(q, k, v, o, gg, do, True, 0.05, order=2, flags=L.FLAG_PAIRWISE)[:3]
    o2, g2, _ = L.forward(q, k, v, True, 0.05, order=2, flags=L.FLAG_PAIRWISE, out=views[0])
    grads2 = L.backward(q, k, v, o, gg, do, True, 0.05, order=2, flags=L.FLAG_PAIRWISE, grads_out=tuple(views[1:]))[:3]
    L.check_status()
    assert torch.equal(gg, g2)
    for a, b in zip((o,) + tuple(grads), (o2,) + tuple(grads2)):
        assert torch.equal(a, b)
    assert all(float(t[..., D].abs().max()) == 0.0 for t in bufs)   # the column beside the rows is untouched


def test_pairwise_form_is_left_to_the_moment_engines_where_it_does_not_apply():
    """Carried states, and tensors expanded with a zero stride, run as without the flag."""
    from reproducing_fastmax_results_b200 import _lib as L

    B, H, N, D = 1, 16, 256, 64
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(B, H, N, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    o, _, state = L.forward(q, k, v, True, 0.05, order=2, want_state=True, flags=L.FLAG_PAIRWISE)
    o_ref, _, state_ref = L.forward(q, k, v, True, 0.05, order=2, want_state=True)
    shared = k[:, :1].expand(B, H, N, D)   # one key head for all query heads
    oe, ge, _ = L.forward(q, shared, v, True, 0.05, order=2, flags=L.FLAG_PAIRWISE)
    oc, gc, _ = L.forward(q, shared.contiguous(), v, True, 0.05, order=2, flags=L.FLAG_PAIRWISE)
    L.check_status()
    for a, b, tol in ((o, o_ref, 1e-2), (state, state_ref, 1e-4), (oe, oc, 1e-2), (ge, gc, 1e-3)):
        assert orc.max_norm_err(host(a), host(b)) < tol


@pytest.mark.parametrize("flags", [0, 4])
@pytest.mark.parametrize("D", [64, 32])
def test_expanded_keys_of_a_long_sequence_with_few_heads(D, flags):
    """One key and value head for all eight query heads (zero stride) at a length that the tensor-memory engine cuts into
    segments: accepted, forward, state-only call and backward, with the results of contiguous copies."""
    from reproducing_fastmax_results_b200 import _lib as L

    B, H, N = 1, 8, 8192
    g = torch.Generator(device="cuda").manual_seed(6)
    q, do = (torch.randn(B, H, N, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    k1, v1 = (torch.randn(B, 1, N, D, device="cuda", generator=g).bfloat16().expand(B, H, N, D) for _ in range(2))

    def run(k, v):
        o, gg, _ = L.forward(q, k, v, True, 0.05, order=2, flags=flags)
        state = L.forward(k, k, v, True, 0.05, order=2, want_state=True, want_output=False, flags=flags)[2]
        grads = L.backward(q, k, v, o, gg, do, True, 0.05, order=2, flags=flags)[:3]
        L.check_status()
        return (o, gg, state) + tuple(grads)

    for a, b in zip(run(k1, v1), run(k1.contiguous(), v1.contiguous())):
        assert orc.max_norm_err(host(a), host(b)) < 2e-2


@pytest.mark.parametrize("dtype,n", [(torch.bfloat16, 5500), (torch.float32, 2000)])
def test_more_heads_than_one_group_of_the_item_order(dtype, n):
    """25 heads whose streamed tiles exceed the share of L2: two groups, the last one smaller; every head, forward and backward."""
    from reproducing_fastmax_results_b200 import _lib as L

    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v, do = (torch.randn(1, 25, n, 64, device="cuda", generator=g).to(dtype) for _ in range(4))
    p = orc.Poly(1.0, 1.0, 0.5, 1.0 / 64.0, 2)
    args = (True, p.inv_temp, p.a0, p.a1, p.a2, 2)
    o, gg, _ = L.forward(q, k, v, *args, flags=L.FLAG_PAIRWISE)
    dq, dk, dv, _ = L.backward(q, k, v, o, gg, do, *args, flags=L.FLAG_PAIRWISE)
    L.check_status()
    rows = np.array([300, 1023, n - 1])
    tol = 2e-2 if dtype == torch.bfloat16 else 5e-6
    for h in range(25):
        a = [host(t[0, h]) for t in (q, k, v, do)]
        oh, gh = host(o[0, h]), host(gg[0, h])
        o_ref, _ = orc.sampled_forward_rows(a[0], a[1], a[2], rows, True, p)
        dq_ref = orc.sampled_dq_rows(a[0], a[1], a[2], oh, gh, a[3], rows, True, p)
        dk_ref, dv_ref = orc.sampled_dkv_cols(a[0], a[1], a[2], oh, gh, a[3], rows, True, p)
        for name, x, r in (("o", o, o_ref), ("dq", dq, dq_ref), ("dk", dk, dk_ref), ("dv", dv, dv_ref)):
            err = np.linalg.norm(host(x[0, h])[rows] - r) / np.linalg.norm(r)
            assert err < tol, (name, h, err)


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("nq,nk,causal", [(2, 3, True), (63, 63, True), (128, 129, True), (300, 300, True), (65, 200, False), (300, 257, False)])
def test_bf16_heads_of_16_dims_keep_float32_weights(nq, nk, causal, order):
    """Against float64 the results are as close as those of the CUDA-core engine, whose weights, gradients of the weights and sums
    are float32: what separates both from float64 is the rounding of the results (and of o) to bf16.  With weights in bf16 the
    error of dq, dk and dv is 1.7 to 1.9 times as large; the two engines' sums in another order flip single roundings (5 %)."""
    from reproducing_fastmax_results_b200 import _lib as L

    B, H, D = 2, 12, 16
    g = torch.Generator(device="cuda").manual_seed(nq + nk)
    mk = lambda n: torch.randn(B, n, H, D, device="cuda", generator=g).bfloat16().transpose(1, 2)
    q, do, k, v = mk(nq), mk(nq), mk(nk), mk(nk)
    it = 1.0 / (8.0 * math.sqrt(D))
    q6, k6, v6 = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    s = (q6 @ k6.transpose(-1, -2)) * it
    f = 1 + s + (0.5 * s * s if order == 2 else 0)
    if causal:
        f = f * torch.ones(nq, nk, device="cuda", dtype=torch.float64).tril(nk - nq)
    o6 = (f @ v6) / f.sum(-1, keepdim=True)
    exact = [o6.detach(), *torch.autograd.grad(o6, (q6, k6, v6), do.double())]

    def errors(flags):
        L.profile_collect()
        L.profile(True)
        o, gg, _ = L.forward(q, k, v, causal, it, order=order, flags=flags)
        grads = L.backward(q, k, v, o, gg, do, causal, it, order=order, flags=flags)[:3]
        L.check_status()
        L.profile(False)
        return [float((a.double() - b).norm() / b.norm()) for a, b in zip((o, *grads), exact)], set(L.profile_collect())

    got, kinds = errors(L.FLAG_PAIRWISE)
    engine, kinds_engine = errors(L.FLAG_NO_TENSOR_CORES)
    assert {"pair_f32_fwd", "pair_f32_bwd_q", "pair_f32_bwd_kv"} <= kinds and "scan_fwd" in kinds_engine
    for name, a, b in zip(("o", "dq", "dk", "dv"), got, engine):
        assert a < 1.05 * b, (name, a, b)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", [(12, 40, 320, 320, 64, True), (12, 40, 320, 60, 32, False), (20, 40, 60, 60, 64, True), (8, 40, 130, 300, 32, True)])
def test_items_of_different_lengths_follow_one_another_on_a_block(case, dtype):
    """Several items per block, some of one tile, some without a second held tile: the rings of score buffers, row sums and held
    tiles go round with every alignment.  Every head is checked, against float64."""
    from reproducing_fastmax_results_b200 import _lib as L

    B, H, nq, nk, D, causal = case
    g = torch.Generator(device="cuda").manual_seed(nq + nk)
    q, do = (torch.randn(B, H, nq, D, device="cuda", generator=g).to(dtype) for _ in range(2))
    k, v = (torch.randn(B, H, nk, D, device="cuda", generator=g).to(dtype) for _ in range(2))
    it = 1.0 / (8.0 * math.sqrt(D))
    o, gg, _ = L.forward(q, k, v, causal, it, flags=L.FLAG_PAIRWISE)
    dq, dk, dv, _ = L.backward(q, k, v, o, gg, do, causal, it, flags=L.FLAG_PAIRWISE)
    L.check_status()
    assert L.wait_histogram() == {}
    qd, kd, vd = (t.double().requires_grad_(True) for t in (q, k, v))
    s = qd @ kd.transpose(-1, -2) * it
    f = 1.0 + s + 0.5 * s * s
    if causal:
        f = f * torch.ones(nq, nk, device="cuda", dtype=torch.float64).tril(nk - nq)
    ref = (f @ vd) / f.sum(-1, keepdim=True)
    grads = torch.autograd.grad(ref, (qd, kd, vd), do.double())
    # bf16: operands and results of 8 bits (2^-9 each, five roundings in a row); float32: 2e-7 measured in every size
    tol = 1e-2 if dtype == torch.bfloat16 else 2e-6
    for name, x, r in (("o", o, ref.detach()), ("dq", dq, grads[0]), ("dk", dk, grads[1]), ("dv", dv, grads[2])):
        err = (x.double() - r).norm(dim=(-1, -2)) / r.norm(dim=(-1, -2))
        assert float(err.max()) < tol, (name, float(err.max()), int(err.argmax()))


@pytest.mark.parametrize("case", [(2, 70, 333, 333, 64, False, 2), (1, 3, 700, 700, 64, True, 2), (1, 2, 260, 1031, 32, False, 2),
                                  (2, 90, 513, 513, 32, True, 2), (1, 4, 300, 300, 64, False, 1)])
def test_row_sums_of_bf16_heads_are_added_in_a_fixed_order(case):
    """g, which every gradient is divided by, does not depend on how many warps share a tile: a row's weights are added in four
    chains of column pairs, whose two lanes meet last.  With scores of few bits all that is rounded is each weight and each
    addition, so the bits of g are those of the same additions here."""
    from reproducing_fastmax_results_b200 import _lib as L

    B, H, nq, nk, D, causal, order = case
    g = torch.Generator(device="cuda").manual_seed(nq + nk)
    mk = lambda n: (torch.randint(-64, 65, (B, H, n, D), device="cuda", generator=g) / 32.0).to(torch.bfloat16)
    q, k, v = mk(nq), mk(nk), mk(nk)
    it = 1.0 / 8.0
    _, gg, _ = L.forward(q, k, v, causal, it, order=order, flags=L.FLAG_PAIRWISE)
    L.check_status()
    s = q.double() @ k.double().transpose(-1, -2)   # exact
    if order == 2:   # 1 + s / 8 + s^2 / 128 = ((s + 8)^2 + 64) / 128: one rounding
        p, scale = ((s + 8.0) ** 2 + 64.0).float(), 1.0 / 128.0
    else:
        p, scale = (1.0 + s * it).float(), 1.0
    if causal:
        p = p * torch.ones(nq, nk, device="cuda").tril(nk - nq)
    p = torch.nn.functional.pad(p, (0, -nk % 8)).cpu().unflatten(-1, (-1, 4, 2)).numpy()   # [..., 8 columns, chain, lane]
    sums = np.zeros(p.shape[:3] + (4, 2), np.float32)
    for m in range(p.shape[3]):
        sums += p[:, :, :, m]
    total = (sums[..., 0, :] + sums[..., 1, :]) + (sums[..., 2, :] + sums[..., 3, :])
    want = (total[..., 0] + total[..., 1]) * np.float32(scale)
    first = 128 if causal else 0   # the first rows of a causal sequence sum rounded weights
    assert np.array_equal(gg[:, :, first:].cpu().numpy(), want[:, :, first:])
