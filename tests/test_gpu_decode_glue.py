"""The small kernels of a decode layer, bitwise against the torch operations they stand for."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,hidden", [(1, 8), (3, 512), (64, 4096), (5, 4104)])
def test_add_rmsnorm(rows, hidden):
    from moeflow_b200.ops.kernels import add_rmsnorm, rmsnorm

    g = torch.Generator().manual_seed(rows)
    x, add = (torch.randn(rows, hidden, generator=g).bfloat16().cuda() for _ in range(2))
    gamma = torch.randn(hidden, generator=g).bfloat16().cuda()
    total, normed = add_rmsnorm(x, add, gamma, 1e-6)
    assert torch.equal(total, x + add)
    assert torch.equal(normed, rmsnorm(x + add, gamma, 1e-6))


@pytest.mark.parametrize("B,kv,S,d", [(1, 1, 1, 8), (4, 4, 37, 128), (65, 2, 9, 64)])
def test_kv_append(B, kv, S, d):
    from moeflow_b200.ops.kernels import kv_append

    g = torch.Generator().manual_seed(B)
    qkv = torch.randn(B, 3 * kv * d, generator=g).bfloat16().cuda()
    k, v = qkv[:, kv * d : 2 * kv * d], qkv[:, 2 * kv * d :]
    kc, vc = (torch.randn(B, kv, S, d, generator=g).bfloat16().cuda() for _ in range(2))
    for pos in {0, S // 2, S - 1, S, -1}:
        kw, vw = kc.clone(), vc.clone()
        if 0 <= pos < S:
            kw[:, :, pos], vw[:, :, pos] = k.view(B, kv, d), v.view(B, kv, d)
        kv_append(k, v, kc, vc, torch.tensor(pos, device="cuda"))
        assert torch.equal(kc, kw) and torch.equal(vc, vw)


@pytest.mark.parametrize("tokens", [1, 64, 65])
def test_two_residuals(tokens):
    from moeflow_b200.ops.dense import DenseProjection

    g = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, 192, generator=g).bfloat16().cuda()
    w = torch.randn(256, 192, generator=g).bfloat16().cuda()
    a, b = (torch.randn(tokens, 256, generator=g).bfloat16().cuda() for _ in range(2))
    project = DenseProjection(w)
    plain = project(x, torch.empty(tokens, 256, dtype=torch.bfloat16, device="cuda"))
    assert torch.equal(project(x, torch.empty_like(a), a, b), (a + b) + plain)


def test_rows_off_the_16_byte_grid_and_host_tensors_are_refused():
    """The kernels read 16 bytes at a time from raw device pointers."""
    from conftest import SMALL_GPU
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.ops.kernels import add_rmsnorm, rmsnorm
    from moeflow_b200.testing import make_logits, make_weights

    H = SMALL_GPU.hidden_size
    off = torch.zeros(2 * H + 1, dtype=torch.bfloat16, device="cuda")[1:].view(2, H)
    fine, gamma = torch.zeros(2, H, dtype=torch.bfloat16, device="cuda"), torch.ones(H, dtype=torch.bfloat16, device="cuda")
    for call in (lambda: rmsnorm(off, gamma), lambda: rmsnorm(fine, off[0]), lambda: rmsnorm(fine, gamma, out=off),
                 lambda: add_rmsnorm(off, fine, gamma), lambda: add_rmsnorm(fine, off, gamma), lambda: add_rmsnorm(fine, fine, off[0])):
        with pytest.raises(RuntimeError):
            call()
    layer = FixedEPLayer(SMALL_GPU, 0, 1, *make_weights(SMALL_GPU, 0, device="cuda"), capacity=2, backend="cuda")
    lg = make_logits(2, SMALL_GPU, 1, device="cuda")
    bias = torch.zeros(SMALL_GPU.n_routed_experts)
    for args in ((off, lg, None), (fine.cpu(), lg, None), (fine, lg.cpu(), None), (fine, lg, bias),
                 (fine, lg, None, torch.tensor(1, dtype=torch.int32))):
        with pytest.raises(ValueError):
            layer.forward(*args)
    assert not layer.forward(fine, lg, bias.cuda()).any() and layer.check_status()["code"] == 0


@pytest.mark.parametrize("rows,hidden,experts", [(1, 8, 1), (3, 264, 7), (4, 4096, 36), (64, 4096, 36), (200, 1024, 17), (5, 16384, 9), (700, 512, 3)])
def test_add_rmsnorm_logits(rows, hidden, experts):
    from moeflow_b200.ops.kernels import add_rmsnorm, add_rmsnorm_logits

    g = torch.Generator().manual_seed(rows)
    x, add = (torch.randn(rows, hidden, generator=g).bfloat16().cuda() for _ in range(2))
    gamma = torch.rand(hidden, generator=g).bfloat16().cuda() + 0.5
    gate = torch.randn(experts + 3, hidden, generator=g).bfloat16().cuda()
    logits = torch.full((rows + 2, experts), 9.0, device="cuda")
    total, h = add_rmsnorm_logits(x, add, gamma, gate, experts, logits)
    want_total, want_h = add_rmsnorm(x, add, gamma)
    assert torch.equal(total, want_total) and torch.equal(h, want_h)
    exact = h.double() @ gate[:experts].double().t()
    # each product is exact in fp32; a sum of n of them in any order errs by at most n * 2**-24 of their absolute sum
    bound = hidden * 2.0**-24 * (h.double().abs() @ gate[:experts].double().abs().t())
    assert bool(((logits[:rows].double() - exact).abs() <= bound + 1e-30).all()) and bool((logits[rows:] == 9).all())


def test_add_rmsnorm_logits_refuses_what_does_not_fit():
    from moeflow_b200.ops.kernels import add_rmsnorm_logits

    x, gamma = torch.zeros(4, 64, dtype=torch.bfloat16, device="cuda"), torch.ones(64, dtype=torch.bfloat16, device="cuda")
    gate, logits = torch.zeros(8, 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(4, 8, device="cuda")
    add_rmsnorm_logits(x, x, gamma, gate, 8, logits)
    for bad in (lambda: add_rmsnorm_logits(x, x[:3], gamma, gate, 8, logits), lambda: add_rmsnorm_logits(x, x, gamma, gate[:, :32].contiguous(), 8, logits),
                lambda: add_rmsnorm_logits(x, x, gamma, gate, 9, logits), lambda: add_rmsnorm_logits(x, x, gamma, gate, 8, logits[:3].contiguous()),
                lambda: add_rmsnorm_logits(x, x, gamma, gate.float(), 8, logits), lambda: add_rmsnorm_logits(x, x, gamma, gate, 8, logits.double())):
        with pytest.raises(ValueError):
            bad()


def test_add_rmsnorm_logits_of_rows_that_are_not_finite():
    """They stay in their own row, and a gate row's in its own column."""
    from moeflow_b200.ops.kernels import add_rmsnorm, add_rmsnorm_logits

    g = torch.Generator().manual_seed(1)
    x, add = (torch.randn(9, 1024, generator=g).bfloat16().cuda() for _ in range(2))
    gamma, gate = torch.rand(1024, generator=g).bfloat16().cuda() + 0.5, torch.randn(36, 1024, generator=g).bfloat16().cuda()
    clean, logits = torch.empty(9, 36, device="cuda"), torch.empty(9, 36, device="cuda")
    add_rmsnorm_logits(x, add, gamma, gate, 36, clean)
    x[2, 5], add[4, 1023], x[7, 0], add[7, 0], gate[35, 8] = float("inf"), float("nan"), float("inf"), float("-inf"), float("nan")
    total, h = add_rmsnorm_logits(x, add, gamma, gate, 36, logits)
    for got, want in zip((total, h), add_rmsnorm(x, add, gamma)):
        torch.testing.assert_close(got, want, rtol=0, atol=0, equal_nan=True)
    rows = [0, 1, 3, 5, 6, 8]
    assert torch.equal(logits[rows, :35], clean[rows, :35]) and bool(logits[:, 35].isnan().all()) and bool(logits[[2, 4, 7]].isnan().all())
