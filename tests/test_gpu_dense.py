"""The dense projection kernel (``ops/dense.py``) against a float64 product of the same bf16 values, at the edges of its
token tiles, of its K cut and of its weight blocks."""

import pytest
import torch

from moeflow_b200.experts import swiglu_clamp

pytestmark = pytest.mark.gpu


def _case(tokens, rows, k, seed=0, pitch_extra=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(tokens, k + pitch_extra, generator=g).bfloat16().cuda()[:, :k]
    w = (torch.randn(rows, k, generator=g) / k**0.5).bfloat16().cuda()
    return x, w


def _bound(x, w, exact):
    """One bf16 rounding of the result, and fp32 sums of k products in any order (k * 2**-24 of the absolute sum)."""
    return exact.abs() * 2.0**-8 + (x.double().abs() @ w.double().abs().t()) * (x.shape[1] * 2.0**-24)


@pytest.mark.parametrize("tokens", [1, 15, 16, 17, 64, 65, 130])
@pytest.mark.parametrize("rows,k", [(128, 64), (384, 4096), (5120, 192), (4096, 1536)])
def test_plain_projection(tokens, rows, k):
    from moeflow_b200.ops.dense import DenseProjection

    x, w = _case(tokens, rows, k, pitch_extra=8 if tokens == 17 else 0)
    out = torch.full((tokens + 2, rows), 7.0, dtype=torch.bfloat16, device="cuda")
    project = DenseProjection(w)
    got = project(x, out)
    exact = x.double() @ w.double().t()
    assert int(project.status.item()) == 0
    assert ((got.double() - exact).abs() <= _bound(x, w, exact)).all()
    assert (out[tokens:] == 7.0).all()  # rows past the batch are not touched
    residual = torch.randn(tokens, rows, generator=torch.Generator().manual_seed(9)).bfloat16().cuda()
    assert torch.equal(project(x, torch.empty_like(residual), residual), residual + got)
    assert torch.equal(project(x, torch.empty_like(residual)), got)  # the same sum on every run


@pytest.mark.parametrize("tokens", [1, 33, 64, 100])
@pytest.mark.parametrize("inter,k", [(64, 64), (320, 128), (1536, 4096)])
def test_gate_up_projection(tokens, inter, k):
    from moeflow_b200.ops.dense import DenseProjection

    x, w = _case(tokens, 2 * inter, k, seed=1)
    out = torch.zeros(tokens, inter, dtype=torch.bfloat16, device="cuda")
    project = DenseProjection(2 * w, gate_up=True, limit=1.5)
    project(x, out)
    h = x.double() @ (2 * w).double().t()
    exact = swiglu_clamp(h.float(), 1.5).double()
    # |d silu| <= 1.1 and |silu(gate)| <= 1.5, |up| <= 1.5 (the clamp): both sums enter with at most 1.7 times their own error
    slack = (x.double().abs() @ (2 * w).double().abs().t()) * (k * 2.0**-24)
    bound = exact.abs() * 2.0**-8 + 1.7 * (slack[:, :inter] + slack[:, inter:]) + 1e-6
    assert int(project.status.item()) == 0
    assert ((out.double() - exact).abs() <= bound).all()


@pytest.mark.parametrize("cols", [1, 127, 288])
def test_fp32_output_stores_only_the_real_columns(cols):
    from moeflow_b200.ops.dense import DenseProjection

    x, w = _case(5, (cols + 127) // 128 * 128, 512, seed=2)
    store = torch.full((6, cols + 160), 7.0, device="cuda")  # what a block of 128 columns would run over
    out = store[:5, :cols]
    DenseProjection(w, out_cols=cols)(x, out)
    exact = x.double() @ w[:cols].double().t()
    slack = (x.double().abs() @ w[:cols].double().abs().t()) * (512 * 2.0**-24)
    assert ((out.double() - exact).abs() <= slack).all() and (store[:5, cols:] == 7.0).all() and (store[5] == 7.0).all()


@pytest.mark.parametrize("tokens", [1, 5])
def test_token_rows_of_any_layout_type_and_device(tokens):
    """What the kernel cannot read in place is copied: expanded, overlapping, odd or transposed rows, other types, host memory."""
    from moeflow_b200.models.glm_moe import RouterLogits, SharedExpert

    k, inter = 256, 128
    g = torch.Generator().manual_seed(3)
    base = torch.randn(4 * tokens * k, generator=g).bfloat16().cuda()
    gate_w = torch.randn(48, k, generator=g).cuda()
    shared = SharedExpert((torch.randn(2 * inter, k, generator=g) / 16).bfloat16().cuda(),
                          (torch.randn(k, inter, generator=g) / 11).bfloat16().cuda(), 8, 10.0)
    router = RouterLogits(gate_w, 8)
    rows = {
        "expanded": base[:k].expand(tokens, k),
        "overlapping": base.as_strided((tokens, k), (8, 1)),
        "odd pitch": base.as_strided((tokens, k), (k + 1, 1)),
        "odd start": base.as_strided((tokens, k), (k, 1), 1),
        "row stride 1": base.as_strided((1, k), (1, 1)).expand(tokens, k),
        "transposed": base[: tokens * k].view(k, tokens).t(),
        "fp32": base[: tokens * k].view(tokens, k).float(),
        "host": base[: tokens * k].view(tokens, k).cpu(),
        "empty": base[:0].view(0, k),
    }
    for name, x in rows.items():
        plain = x.clone(memory_format=torch.contiguous_format).bfloat16().cuda()
        first = router(x).clone()
        assert torch.equal(first, router(plain)), name
        first = shared(x).clone()
        assert torch.equal(first, shared(plain)) and first.shape == (x.shape[0], k), name
    assert int(shared.status.item()) == 0 and int(router.status.item()) == 0


def test_operands_that_do_not_fit_are_refused():
    from moeflow_b200.ops.dense import DenseProjection

    x, w = _case(3, 256, 128)
    project, bf16 = DenseProjection(w), dict(dtype=torch.bfloat16, device="cuda")
    good, wide = torch.zeros(3, 256, **bf16), torch.zeros(3, 512, **bf16)
    bad = [good.float(), good.cpu(), good[:2], good[:, :255], wide[:, ::2], good[0]]
    for r in bad:
        with pytest.raises(ValueError):
            project(x, good, r)
        with pytest.raises(ValueError):
            project(x, good, good, r)
    for out in [good.half(), *bad[1:], good[:1].expand(3, 256)]:
        with pytest.raises(ValueError):
            project(x, out)
    with pytest.raises(ValueError):
        project(x, good.float(), good)  # residuals belong to a bf16 product
    with pytest.raises(ValueError):
        project(x, good, None, good)
    with pytest.raises(ValueError):
        project(x[:, :64], good)
    want = project(x, good.clone(), good)
    assert torch.equal(project(x, wide[:, 256:], good[:1].expand(3, 256)), want)  # a strided out, an expanded residual
    narrow = DenseProjection(w, out_cols=100)
    assert torch.equal(narrow(x, torch.zeros(3, 100, **bf16)), want[:, :100])
