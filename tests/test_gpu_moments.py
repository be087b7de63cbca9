"""State-only calls on tensor memory (moments without an output) where their geometry changes: fewer tiles than a block
takes, a last chunk of one token, token cuts whose sums are added, a carried state, gradient moments; against the CUDA-core
engine's exact features."""
import pytest
import torch

from oracle import fastmax_oracle as orc

pytestmark = pytest.mark.gpu


def host(t):
    return t.detach().double().cpu().numpy()


@pytest.mark.parametrize("order,B,H,N", [(2, 1, 13, 1), (2, 1, 13, 129), (2, 2, 16, 640), (2, 1, 16, 4097), (2, 4, 40, 300),
                                         (1, 1, 64, 1000), (1, 2, 100, 127), (1, 1, 64, 40), (2, 1, 150, 1700)])
@pytest.mark.parametrize("carried", [False, True])
def test_state_only_calls_match_the_cuda_core_engine(order, B, H, N, carried):
    from reproducing_fastmax_results_b200 import _lib as L

    g = torch.Generator(device="cuda").manual_seed(N + H)
    mk = lambda: (torch.randn(B, N, H, 64, device="cuda", generator=g) * 0.7).bfloat16().transpose(1, 2)
    q, k, v, do = mk(), mk(), mk(), mk()
    init = torch.randn(L.new_state(B, H, 64, order).shape, device="cuda", generator=g) if carried else None
    if carried:
        init[..., 65:] = 0.0
    o, gg, _ = L.forward(q, k, v, True, 0.05, order=order)
    res = []
    for flags in (0, L.FLAG_NO_TENSOR_CORES):
        s = L.forward(k, k, v, True, 0.05, order=order, state_in=init, want_state=True, want_output=False, flags=flags)[2]
        ds = L.backward(q, k, v, o, gg, do, True, 0.05, order=order, dstate_in=init, want_dstate=True, want_grads=False, flags=flags)[3]
        L.check_status()
        res.append((s, ds))
    assert L.wait_histogram() == {}
    for a, b, tol in zip(*res, (5e-3, 2e-2)):
        assert float(a[..., 65:].abs().max()) == 0.0
        assert orc.max_norm_err(host(a), host(b)) < tol


@pytest.mark.parametrize("carried", [False, True])
@pytest.mark.parametrize("H,N,order", [(16, 32768, 2), (32, 8192, 2), (64, 2000, 1), (64, 8192, 1)])
def test_states_are_the_same_bits_on_every_run(H, N, order, carried):
    """Few heads, so that the tokens are cut over several blocks which add their sums in the order in which they end."""
    from reproducing_fastmax_results_b200 import _lib as L

    g = torch.Generator(device="cuda").manual_seed(N)
    k, v = (torch.randn(1, H, N, 64, device="cuda", generator=g).bfloat16() for _ in range(2))
    start = torch.randn(L.new_state(1, H, 64, order).shape, device="cuda", generator=g) if carried else None
    call = lambda: L.forward(k, k, v, True, 1.0 / 64, order=order, want_state=True, want_output=False, state_in=start)[2]
    first = call()
    assert all(torch.equal(first, call()) for _ in range(10))
