"""Linear layers of one or two tokens (csrc/kernels/gemv.cu): the product alone, behind the residual add and RMSNorm, and as a gate / up pair, against f64."""
import pytest
import torch

from gemm_b200 import _native
from gemm_b200.ops import elementwise as ew
from gemm_b200.ops import gemm, mxfp8

pytestmark = pytest.mark.gpu

# features around what a CTA takes (8, 16 or 32) and around the steps of the dispatch, K around a warp's 256 columns and the loads in flight
SHAPES = [(1, 64), (9, 256), (130, 72), (1024, 2048), (1023, 3072), (2368, 320), (2369, 1024), (4736, 1088), (6144, 4096), (24576, 512), (151, 8192)]


def _weight(n, k, seed):
    torch.manual_seed(seed)
    return (torch.randn(n, k, device="cuda") * k ** -0.5).bfloat16()


def _tile(w):
    ok = w.shape[0] % 128 == 0 and w.shape[1] % 64 == 0
    return (mxfp8.tile_weight(w) if ok else w), ok


def _bound(x, w):                     # f32 sums of k products, in any order
    return x.shape[1] ** 0.5 * 2 ** -22 * (x.double().abs() @ w.double().abs().t()) + 1e-6


@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("n,k", SHAPES + [(256, 25600)])
def test_product(m, n, k):
    w = _weight(n, k, n + k)
    x = torch.randn(m, k + 8, device="cuda").bfloat16()[:, :k]
    bias = torch.randn(n, device="cuda")
    wt, tiled = _tile(w)
    got = gemm.gemv(x, wt, bias=bias, w_tiled=tiled)
    _native.assert_status_ok()
    ref = x.double() @ w.double().t()
    assert got.n == 1 and ((got.buf[0].double() - bias - ref).abs() <= _bound(x, w) + 2 ** -22 * bias.abs()).all()


@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("slabs", [0, 1, 3])
def test_behind_the_norm(m, n, k, slabs):
    w = _weight(n, k, n + k + slabs)
    res = torch.randn(m, k, device="cuda").bfloat16()
    keep = res.clone()
    nw = torch.rand(k, device="cuda").add_(0.5).bfloat16()
    delta = gemm.PendingPartials(torch.randn(slabs, m, k, device="cuda")) if slabs else None
    wt, tiled = _tile(w)
    got, new = gemm.gemv_norm(res, delta, nw, 1e-6, wt, w_tiled=tiled)
    # the rows that the separate kernel forms
    rows = res.clone()
    h = ew.rmsnorm(delta, nw, 1e-6, residual=rows) if slabs else ew.rmsnorm(rows, nw, 1e-6)
    _native.assert_status_ok()
    assert torch.equal(res, keep) and torch.equal(new, rows)
    assert ((got.buf[0].double() - h.double() @ w.double().t()).abs() <= _bound(h, w)).all()


@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("n,k", SHAPES)
def test_gate_up(m, n, k):
    w = _weight(2 * n, k, n + k + 7)
    res, nw = torch.randn(m, k, device="cuda").bfloat16(), torch.rand(k, device="cuda").add_(0.5).bfloat16()
    wt, tiled = _tile(w)
    act, new = gemm.gemv_norm(res, None, nw, 1e-6, wt, w_tiled=tiled, swiglu=True)
    y = ew.rmsnorm(res.clone(), nw, 1e-6).double() @ w.double().t()
    ref = torch.nn.functional.silu(y[:, :n]) * y[:, n:]
    _native.assert_status_ok()
    assert new is res and ((act.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-4).all()
