"""Long bf16 sequences as windows of pairs plus moment states (FASTMAX_FLAG_PAIRWISE beyond the lengths the pairwise form is
cheaper for), against the CPU oracle's sampled rows and columns: ragged last windows, a last window of one token, no mask,
order 1, head-split views, the states handed from forward to backward or built again, the final state of a prompt."""
import math

import numpy as np
import pytest
import torch

from oracle import fastmax_oracle as orc

pytestmark = pytest.mark.gpu


def host(t):
    return t.detach().double().cpu().numpy()


CASES = [  # B, H, nq, nk, D, causal, order
    (1, 2, 7681, 7681, 64, True, 2),   # five windows of 1536 and one token
    (2, 2, 8000, 8000, 64, True, 2),
    (1, 3, 3840, 3840, 32, True, 2),   # five whole windows
    (2, 1, 4001, 4001, 32, True, 2),
    (1, 2, 5000, 4700, 64, False, 2),
    (1, 2, 1400, 9000, 32, False, 2),
    (1, 2, 2305, 2305, 64, True, 1),
    (1, 2, 1700, 900, 32, False, 1),
]


@pytest.mark.parametrize("hand_over", [True, False])
@pytest.mark.parametrize("case", CASES)
def test_windows_match_oracle(case, hand_over):
    from reproducing_fastmax_results_b200 import _lib as L

    B, H, nq, nk, D, causal, order = case
    g = torch.Generator(device="cuda").manual_seed(nq + nk + D)
    mk = lambda n: torch.randn(B, n, H, D, device="cuda", generator=g).bfloat16().transpose(1, 2)
    q, do, k, v = mk(nq), mk(nq), mk(nk), mk(nk)
    p = orc.Poly(0.9, 1.1, 0.45, 1.0 / (8.0 * math.sqrt(D)), order)
    args = (causal, p.inv_temp, p.a0, p.a1, p.a2, order)
    km = L.KeyMoments()
    L.profile_collect()
    L.profile(True)
    o, gg, _ = L.forward(q, k, v, *args, flags=L.FLAG_PAIRWISE, key_moments=km)
    assert km.buf is not None
    dq, dk, dv, _ = L.backward(q, k, v, o, gg, do, *args, flags=L.FLAG_PAIRWISE, key_moments=km if hand_over else None)
    L.check_status()
    L.profile(False)
    assert L.profile_collect()["tc_moments"][1] == (2 if hand_over else 3)
    assert L.wait_histogram() == {}
    rng = np.random.default_rng(nq)
    for b, h in {(0, 0), (B - 1, H - 1)}:
        a = [host(t[b, h]) for t in (q, k, v, do)]
        oh, gh = host(o[b, h]), host(gg[b, h])
        win = [w for w in (127, 511, 512, 767, 768, 1535, 1536, 3071, 3072) if w < min(nq, nk)]
        rq = np.unique(np.concatenate([win, [nq - 1], rng.integers(64, nq, 24)]))
        rk = np.unique(np.concatenate([win, [nk - 1], rng.integers(64, nk, 24)]))
        o_ref, g_ref = orc.sampled_forward_rows(a[0], a[1], a[2], rq, causal, p)
        assert orc.max_norm_err(oh[rq], o_ref) < 2e-2 and orc.max_norm_err(gh[rq], g_ref) < 1e-3
        dq_ref = orc.sampled_dq_rows(a[0], a[1], a[2], oh, gh, a[3], rq, causal, p)
        dk_ref, dv_ref = orc.sampled_dkv_cols(a[0], a[1], a[2], oh, gh, a[3], rk, causal, p)
        for name, x, ref, rows in (("dq", dq, dq_ref, rq), ("dk", dk, dk_ref, rk), ("dv", dv, dv_ref, rk)):
            err = np.linalg.norm(host(x[b, h])[rows] - ref) / np.linalg.norm(ref)
            assert err < 2e-2, (name, b, h, err)


@pytest.mark.parametrize("D,N", [(64, 5200), (32, 2500)])
def test_prompt_of_windows_returns_its_state(D, N):
    from reproducing_fastmax_results_b200 import _lib as L

    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn(1, 20, N, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    L.profile_collect()
    L.profile(True)
    o, gg, state = L.forward(q, k, v, True, 0.02, order=2, want_state=True, flags=L.FLAG_PAIRWISE)
    L.check_status()
    L.profile(False)
    assert L.profile_collect()["tc_moments"][1] == 1
    o2, g2, state2 = L.forward(q, k, v, True, 0.02, order=2, want_state=True, flags=L.FLAG_NO_TENSOR_CORES)
    torch.cuda.synchronize()
    for a, b, tol in ((o, o2, 2e-2), (gg, g2, 1e-3), (state, state2, 5e-3)):
        assert orc.max_norm_err(host(a), host(b)) < tol
    assert float(state[..., D + 1:].abs().max()) == 0.0


F32_CASES = [  # B, H, n, order, head-split views
    (1, 2, 4097, 2, False),   # eight windows of 512 and one token
    (2, 2, 4500, 2, True),
    (1, 3, 4608, 2, True),    # nine whole windows
    (1, 2, 1300, 1, False),
]


@pytest.mark.parametrize("hand_over", [True, False])
@pytest.mark.parametrize("case", F32_CASES)
def test_float32_windows_match_oracle(case, hand_over):
    from reproducing_fastmax_results_b200 import _lib as L

    B, H, n, order, split = case
    D = 32
    g = torch.Generator(device="cuda").manual_seed(n)
    mk = lambda: (torch.randn(B, n, H, D, device="cuda", generator=g).transpose(1, 2) if split else torch.randn(B, H, n, D, device="cuda", generator=g))
    q, k, v, do = (mk() for _ in range(4))
    p = orc.Poly(0.9, 1.1, 0.45, 1.0 / (8.0 * math.sqrt(D)), order)
    args = (True, p.inv_temp, p.a0, p.a1, p.a2, order)
    km = L.KeyMoments()
    L.profile_collect()
    L.profile(True)
    o, gg, _ = L.forward(q, k, v, *args, flags=L.FLAG_PAIRWISE, key_moments=km)
    assert km.buf is not None
    dq, dk, dv, _ = L.backward(q, k, v, o, gg, do, *args, flags=L.FLAG_PAIRWISE, key_moments=km if hand_over else None)
    L.check_status()
    L.profile(False)
    assert L.profile_collect()["tc_moments"][1] == (2 if hand_over else 3)
    assert L.wait_histogram() == {}
    rng = np.random.default_rng(n)
    for b, h in {(0, 0), (B - 1, H - 1)}:
        a = [host(t[b, h]) for t in (q, k, v, do)]
        oh, gh = host(o[b, h]), host(gg[b, h])
        rows = np.unique(np.concatenate([[0, 127, 511, 512, 639, 1023, 1024, n - 1], rng.integers(0, n, 24)]))
        o_ref, g_ref = orc.sampled_forward_rows(a[0], a[1], a[2], rows, True, p)
        assert orc.max_norm_err(oh[rows], o_ref) < 2e-6 and orc.max_norm_err(gh[rows], g_ref) < 2e-6
        dq_ref = orc.sampled_dq_rows(a[0], a[1], a[2], oh, gh, a[3], rows, True, p)
        dk_ref, dv_ref = orc.sampled_dkv_cols(a[0], a[1], a[2], oh, gh, a[3], rows, True, p)
        for name, x, ref in (("dq", dq, dq_ref), ("dk", dk, dk_ref), ("dv", dv, dv_ref)):
            err = np.linalg.norm(host(x[b, h])[rows] - ref) / np.linalg.norm(ref)
            assert err < 3e-6, (name, b, h, err)


@pytest.mark.parametrize("binding", ["ctypes", "extension", "entry point"])
@pytest.mark.parametrize("variant", ["dstate_in", "dstate_out", "gradient rows", "prompt"])
@pytest.mark.parametrize("dtype,D,N", [(torch.bfloat16, 64, 8192), (torch.float32, 32, 4096)])
def test_key_moments_of_another_form_are_not_read(dtype, D, N, variant, binding, monkeypatch):
    """A forward of the window form leaves packed states; a backward of the same problem that also takes or returns gradient
    moments, or writes into rows the copy engine cannot, runs on the moment engines and must not read them (nor may the
    window form read what a prompt's state left).  Same gradients with and without the hand-over.  "entry point": the array is
    passed whatever its size, and fastmax_backward itself leaves it unread."""
    import reproducing_fastmax_results_b200 as pkg
    from reproducing_fastmax_results_b200 import _lib as L

    ext = pkg.load_extension()
    B, H = 1, 8
    g = torch.Generator(device="cuda").manual_seed(N + D)
    q, k, v, do = (torch.randn(B, H, N, D, device="cuda", generator=g).to(dtype) for _ in range(4))
    it = 1.0 / (8.0 * math.sqrt(D))
    poly = (1.0, 1.0, 0.5, 2)
    dstate = torch.randn(L.new_state(B, H, D).shape, device="cuda", generator=g) * 1e-2 if variant == "dstate_in" else None
    want_state, want_dstate = variant == "prompt", variant == "dstate_out"

    def rows():
        if variant != "gradient rows":
            return None
        return [torch.zeros(B, H, N, D + 1, device="cuda", dtype=dtype)[..., :D] for _ in range(3)]

    def run(hand_over):
        if binding != "extension":
            km = L.KeyMoments()
            o, gg, _ = L.forward(q, k, v, True, it, *poly, want_state=want_state, flags=L.FLAG_PAIRWISE, key_moments=km)
            if binding == "entry point":
                monkeypatch.setattr(L.load(), "fastmax_backward_key_moments_bytes", lambda *_: km.buf.numel() * 4)
            res = L.backward(q, k, v, o, gg, do, True, it, *poly, dstate_in=dstate, want_dstate=want_dstate, grads_out=rows(),
                             flags=L.FLAG_PAIRWISE, key_moments=km if hand_over else None)
            buf = km.buf
        else:
            o, gg, _, buf = ext.forward(q, k, v, True, it, *poly, None, want_state, True, ext.PAIRWISE, None, None, True)
            res = ext.backward(q, k, v, o, gg, do, True, it, *poly, None, dstate, want_dstate, True, ext.PAIRWISE, rows(),
                               buf if hand_over else None)[:4]
        L.check_status()
        assert buf.numel() % 4 == 1   # packed states, whatever else the forward returned
        return [t for t in res if t is not None and t.numel()]

    for a, b in zip(run(True), run(False)):
        assert orc.max_norm_err(host(a), host(b)) < (1e-2 if dtype == torch.bfloat16 else 2e-6)


@pytest.mark.parametrize("order", [2, 1])
def test_float32_windows_with_many_items_per_block(order):
    """Several items per block in the moments, apply and chain kernels: their rings go on from one item to the next."""
    from reproducing_fastmax_results_b200 import _lib as L

    g = torch.Generator(device="cuda").manual_seed(order)
    q, k, v, do = (torch.randn(1, 40, 4100, 32, device="cuda", generator=g) for _ in range(4))
    res = []
    for flags in (L.FLAG_PAIRWISE, L.FLAG_NO_TENSOR_CORES):
        o, gg, _ = L.forward(q, k, v, True, 0.02, order=order, flags=flags)
        res.append((o, gg) + tuple(L.backward(q, k, v, o, gg, do, True, 0.02, order=order, flags=flags)[:3]))
    L.check_status()
    assert L.wait_histogram() == {}
    for name, a, b in zip(("o", "g", "dq", "dk", "dv"), *res):   # both at 1e-7 to 3e-7 against float64
        assert float((a - b).norm() / b.norm()) < 3e-6, name
