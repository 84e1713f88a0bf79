"""Prefill-sized bf16 layers against f32 products, at the edges of tiles, of the K steps and of the rings: gate / up projections on SM pairs (256 features x up
to 256 tokens, one to many tiles per pair), plain ones with more blocks of features than SMs (groups of eight token tiles)."""
import pytest
import torch

from gemm_b200 import _native
from gemm_b200.ops import gemm, mxfp8

pytestmark = pytest.mark.gpu

SHAPES = [(65, 256, 64), (96, 256, 4096), (129, 512, 128), (257, 512, 72), (300, 768, 320), (511, 256, 1024), (2049, 1024, 520), (288, 4096, 4096), (5000, 1280, 256),
          (2600, 6144, 448)]
# token counts that the pairs leave to a CTA per tile (and the first ones past them), features that are no whole number of pairs' blocks, two rounds in either form
EDGES = [(80, 3072, 64), (96, 1024, 128), (97, 1024, 128), (128, 256, 192), (112, 9728, 64), (300, 384, 320), (320, 12288, 64), (300, 2048, 4160), (320, 6144, 64)]
WIDE = [(256, 18944, 64), (300, 18951, 128), (2048, 19200, 192), (2305, 24576, 64), (4500, 18944, 72)]


def _inputs(m, n, k):
    torch.manual_seed(m + n + k)
    x = torch.randn(m, k + 8, device="cuda").bfloat16()[:, :k]               # rows wider than the operand
    w = (torch.randn(n, k, device="cuda") * k ** -0.5).bfloat16()
    return x, w


def _close(got, ref):
    # f32 sums of exact bf16 products, then one rounding to bf16 (f32 results: none)
    _native.assert_status_ok()
    bound = ref.abs() * (2 ** -8 if got.dtype == torch.bfloat16 else 0) + 1e-4
    assert ((got.float() - ref).abs() <= bound).all(), (got.float() - ref).abs().max()


def _kernels(call):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]


@pytest.mark.parametrize("m,n,k", SHAPES + EDGES)
def test_swiglu_takes_the_kernel_of_the_rule(m, n, k):
    x, w = _inputs(m, 2 * n, k)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    names = _kernels(lambda: gemm.linear_swiglu(x, w))
    pairs = n % 256 == 0 and _native.cuda().gb_gemm_takes_pairs(n, k, m, sms) == 1
    assert len([s for s in names if ("gemm_pair_kernel" if pairs else "gemm_tc_kernel") in s]) == 1, names
    assert pairs or not any("gemm_pair_kernel" in s for s in names), names


@pytest.mark.parametrize("m,n,k", SHAPES + EDGES)
def test_swiglu(m, n, k):
    x, w = _inputs(m, 2 * n, k)
    y = x.float() @ w.float().t()
    ref = torch.nn.functional.silu(y[:, :n]) * y[:, n:]
    tiled = k % 64 == 0
    out = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm.linear_swiglu(x, mxfp8.tile_weight(w) if tiled else w, out=out[:m], w_tiled=tiled)
    _close(out[:m], ref)
    assert (out[m] == 7).all()


@pytest.mark.parametrize("m,n,k", WIDE)
@pytest.mark.parametrize("tiled", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_linear_with_many_features(m, n, k, tiled, dtype):
    x, w = _inputs(m, n, k)
    bias = torch.randn(n, device="cuda") if m % 2 else None
    ref = x.float() @ w.float().t() + (bias if bias is not None else 0)
    if tiled and (k % 64 or n % 128):
        pytest.skip("tiled weights have whole blocks")
    out = torch.full((m + 1, n), 7.0, dtype=dtype, device="cuda")
    gemm.linear(x, mxfp8.tile_weight(w) if tiled else w, bias=bias, out=out[:m], w_tiled=tiled)
    _close(out[:m], ref)
    assert (out[m] == 7).all()


def test_gate_up_pairs_have_token_tiles_of_at_most_128():
    x, w = _inputs(512, 6144, 256)
    assert _native.cuda().gb_gemm_takes_pairs(3072, 256, 512, 148) == 1
    with pytest.raises(RuntimeError, match="unsupported variant"):
        gemm.linear_swiglu(x, w, tn=256)
    with pytest.raises(RuntimeError, match="unsupported variant"):
        gemm.linear_swiglu(x, w, tn=256, act="gelu_tanh")


def _mx(n, k):
    w = mxfp8.quantize((torch.randn(n, k, device="cuda") * k ** -0.5).bfloat16())
    return mxfp8.MxTensor(mxfp8.tile_weight(w.data), w.sf, w.rows, w.k, w.sf_layout, True)


@pytest.mark.parametrize("m,n,k", [(300, 18944, 64), (1300, 19200, 128), (2304, 18944, 72)])
@pytest.mark.parametrize("form", ["gelu_tanh", "capped", "gelu"])
def test_wide_layers_with_activations(m, n, k, form):
    """With as many blocks of features as SMs several token tiles share a block: the same bits as a launch per token tile."""
    x, w = _inputs(m, n if form == "gelu" else 2 * n, k)
    call = (lambda v: gemm.linear(v, w, gelu=True, tn=256)) if form == "gelu" else (lambda v: gemm.linear_swiglu(v, w, tn=128, act=form, cap=7.0))
    got = call(x)
    _native.assert_status_ok()
    for t in range(0, m, 256 if form == "gelu" else 128):
        assert torch.equal(got[t: t + 128], call(x[t: t + 128])), t


@pytest.mark.parametrize("m,k", [(300, 128), (512, 256), (2049, 128)])
def test_wide_mxfp8_layers(m, k):
    """The same for MXFP8 operands, plain and with the quantising epilogue (which keeps the other order with a ragged last tile)."""
    torch.manual_seed(m)
    n = 18944
    x, w = torch.randn(m, k, device="cuda").bfloat16(), _mx(n, k)
    got = gemm.linear_mx(mxfp8.quantize(x), w, tn=256)
    w2 = _mx(2 * n, k)
    q = gemm.linear_mx_swiglu_quant(mxfp8.quantize(x), w2)
    qe = mxfp8.unpack_sf_atoms(q.sf, q.data.shape[0], n // 32)
    _native.assert_status_ok()
    for t in range(0, m, 128):
        xs = mxfp8.quantize(x[t: t + 128])
        assert torch.equal(got[t: t + 128], gemm.linear_mx(xs, w, tn=256)), t
        part = gemm.linear_mx_swiglu_quant(xs, w2)
        rows = min(128, m - t)
        assert torch.equal(q.data[t: t + rows], part.data[:rows]), t
        assert torch.equal(qe[t: t + rows], mxfp8.unpack_sf_atoms(part.sf, part.data.shape[0], n // 32)[:rows]), t
