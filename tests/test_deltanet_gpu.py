"""Delta-Net kernels (conv + SiLU, recurrence + gated norm, sigmoid gate) and M-RoPE against their PyTorch references."""
import pytest
import torch

from gemm_b200 import _native
from gemm_b200.ops import deltanet as dn
from gemm_b200.ops import elementwise as ew
from gemm_b200.ops import gemm

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float().cpu() - b.float().cpu()).norm() / (b.float().cpu().norm() + 1e-12)).item()


def test_conv_silu_with_history():
    torch.manual_seed(1)
    ch, ck, wide = 512, 4, 768
    lens = [5, 1, 37]
    cu = torch.tensor([0, 5, 6, 43], dtype=torch.int32)
    slots = torch.tensor([2, 0, 3], dtype=torch.int32)
    x = torch.randn(43, wide).bfloat16()
    w = torch.randn(ch, ck)
    st = torch.randn(4, ck - 1, ch)
    st_ref, st_gpu = st.clone(), st.clone().cuda()
    ref = dn.conv_silu(x[:, :ch], w, st_ref, cu, slots)
    got = dn.conv_silu(x.cuda()[:, :ch], w.cuda(), st_gpu, cu.cuda(), slots.cuda())
    assert _rel(got, ref) < 1e-2
    assert _rel(st_gpu, st_ref) < 1e-6
    assert torch.equal(st_gpu[1].cpu(), st[1])            # a slot no sequence uses is untouched


@pytest.mark.parametrize("ch,ck,wide,off", [(512, 4, 768, 0), (510, 4, 513, 0), (1036, 2, 1040, 4), (257, 8, 300, 3), (64, 3, 64, 0)])
def test_conv_silu_tiles(ch, ck, wide, off):
    """Tiles of 32 tokens: sequences at and around their edges (empty and shorter than the window among them), more than 32 sequences, rows that are not
    8-byte aligned, other window lengths."""
    torch.manual_seed(5)
    lens = [31, 0, 32, 33, 1, 2, 64, 65, 0, 200] + [1] * 30 + [7, 40]
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32)
    slots = torch.randperm(len(lens) + 2)[: len(lens)].to(torch.int32)
    x = torch.randn(sum(lens), wide).bfloat16()
    w, st = torch.randn(ch, ck), torch.randn(len(lens) + 2, ck - 1, ch)
    st_gpu = st.clone().cuda()
    ref = dn.conv_silu(x[:, off: off + ch], w, st, cu, slots)
    got = dn.conv_silu(x.cuda()[:, off: off + ch], w.cuda(), st_gpu, cu.cuda(), slots.cuda())
    # the same f32 sums in the same order: the results differ by the sigmoid's rounding, at most one step of bf16
    assert (got.float().cpu() - ref.float()).abs().max() <= 2 ** -7 * ref.float().abs().max()
    assert _rel(got, ref) < 2 ** -9
    assert torch.equal(st_gpu.cpu(), st)


def test_conv_silu_taps_of_the_launch_before():
    """The taps may be the result of the kernel launched just before, which lets its successor start before it stores."""
    torch.manual_seed(7)
    ch, ck, k = 12288, 4, 512
    a, b = torch.randn(ch, k, device="cuda").bfloat16(), (torch.randn(ck, k, device="cuda") * k ** -0.5).bfloat16()
    x, st = torch.randn(8, ch, device="cuda").bfloat16(), torch.randn(1, ck - 1, ch, device="cuda")
    cu, slots = torch.tensor([0, 8], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    w = gemm.linear(a, b, out_dtype=torch.float32)
    torch.cuda.synchronize()
    want = dn.conv_silu(x, w.clone(), st.clone(), cu, slots)
    s2 = st.clone()
    torch.full((ch, ck), float("nan"), device="cuda")                                        # what the allocator hands out next
    torch.cuda.synchronize()
    assert torch.equal(dn.conv_silu(x, gemm.linear(a, b, out_dtype=torch.float32), s2, cu, slots), want)


@pytest.mark.parametrize("ds,ng,hv", [(64, 2, 4), (128, 2, 6)])
def test_deltanet_recurrence(ds, ng, hv):
    torch.manual_seed(2)
    lens = [9, 1, 20]
    cu = torch.tensor([0, 9, 10, 30], dtype=torch.int32)
    slots = torch.tensor([1, 2, 0], dtype=torch.int32)
    t = 30
    qkv = (torch.randn(t, (2 * ng + hv) * ds) * 0.5).bfloat16()
    z = torch.randn(t, hv * ds + 64).bfloat16()[:, : hv * ds]          # a column slice of a wider tensor
    ab = torch.randn(t, 2 * hv)
    a = -(torch.rand(hv) * 2 + 0.1)
    bias = torch.randn(hv) * 0.5
    nw = torch.rand(ds) + 0.5
    st = torch.randn(3, hv, ds, ds) * 0.1
    st_ref, st_gpu = st.clone(), st.clone().cuda()
    ref = dn.deltanet(qkv, z, ab, a, bias, nw, st_ref, cu, slots, ng, hv, ds, 1e-6)
    got = dn.deltanet(qkv.cuda(), z.cuda(), ab.cuda(), a.cuda(), bias.cuda(), nw.cuda(), st_gpu, cu.cuda(), slots.cuda(), ng, hv, ds, 1e-6)
    _native.assert_status_ok()
    assert _rel(got, ref) < 1e-2
    assert _rel(st_gpu, st_ref) < 1e-4


@pytest.mark.parametrize("lens", [[150, 64, 70, 200], [1000], [63, 65, 128, 129, 48]])
def test_deltanet_chunked_scan(lens):
    """Prefill-sized launches take the chunked scan (64 tokens per serial step, bf16 tiles, fp32 state): against the per-token
    fp32 reference and against the per-token kernel, including partial last chunks and states that are not zero."""
    torch.manual_seed(4)
    ds, ng, hv = 128, 2, 4
    n = len(lens)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    slots = torch.randperm(n + 1)[:n].to(torch.int32)
    t = sum(lens)
    qkv = torch.randn(t, (2 * ng + hv) * ds).bfloat16()
    z = torch.randn(t, hv * ds + 64).bfloat16()[:, : hv * ds]
    ab = torch.randn(t, 2 * hv)
    a = -(torch.rand(hv) * 2 + 0.1)
    bias = torch.randn(hv) * 0.5
    nw = torch.rand(ds) + 0.5
    st = torch.randn(n + 1, hv, ds, ds) * 0.1
    st_ref, st_gpu, st_tok = st.clone(), st.clone().cuda(), st.clone().cuda()
    assert dn.CHUNKED and t >= dn.CHUNKED_MIN_TOKENS * n
    ref = dn.deltanet(qkv, z, ab, a, bias, nw, st_ref, cu, slots, ng, hv, ds, 1e-6)
    args = (qkv.cuda(), z.cuda(), ab.cuda(), a.cuda(), bias.cuda(), nw.cuda())
    got = dn.deltanet(*args, st_gpu, cu.cuda(), slots.cuda(), ng, hv, ds, 1e-6)
    _native.assert_status_ok()
    dn.CHUNKED = False
    try:
        tok = dn.deltanet(*args, st_tok, cu.cuda(), slots.cuda(), ng, hv, ds, 1e-6)
    finally:
        dn.CHUNKED = True
    assert _rel(tok, ref) < 1e-2
    assert _rel(got, ref) < 2e-2, _rel(got, ref)
    assert _rel(st_gpu, st_ref) < 1e-2, _rel(st_gpu, st_ref)
    unused = [i for i in range(n + 1) if i not in slots.tolist()][0]
    assert torch.equal(st_gpu[unused].cpu(), st[unused])
    # per sequence, so that a wrong chunk of a short sequence cannot hide behind a long one
    for i in range(n):
        assert _rel(got[cu[i]:cu[i + 1]], ref[cu[i]:cu[i + 1]]) < 2e-2, (i, lens[i])


def test_deltanet_scan_with_one_and_two_ctas_per_head():
    """A launch whose heads fill the GPU scans with a CTA per head, a small one with two: the same numbers, bit for bit."""
    torch.manual_seed(6)
    ds, ng, hv, n = 128, 2, 4, 24                     # 192 CTAs in pairs: more than SMs
    lens = [48 + 7 * i for i in range(n)]
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    t = cu[-1]
    qkv, z, ab = torch.randn(t, (2 * ng + hv) * ds, device="cuda").bfloat16(), torch.randn(t, hv * ds, device="cuda").bfloat16(), torch.randn(t, 2 * hv, device="cuda")
    a, bias, nw = -(torch.rand(hv, device="cuda") * 2 + 0.1), torch.randn(hv, device="cuda") * 0.5, torch.rand(ds, device="cuda") + 0.5
    st = torch.randn(n, hv, ds, ds, device="cuda") * 0.1
    st1 = st.clone()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    got = dn.deltanet(qkv, z, ab, a, bias, nw, st, i32(cu), i32(list(range(n))), ng, hv, ds, 1e-6)
    for i in range(n):
        sl = slice(cu[i], cu[i + 1])
        one = dn.deltanet(qkv[sl], z[sl], ab[sl], a, bias, nw, st1, i32([0, lens[i]]), i32([i]), ng, hv, ds, 1e-6)
        assert torch.equal(one, got[sl]), i
    _native.assert_status_ok()
    assert torch.equal(st, st1)


def test_sigmoid_gate_mul():
    torch.manual_seed(3)
    x = torch.randn(19, 512).bfloat16()
    wide = torch.randn(19, 1536).bfloat16()
    ref = (x.float() * torch.sigmoid(wide[:, 1024:].float()))
    got = dn.gate_mul(x.clone().cuda(), wide.cuda()[:, 1024:])
    assert _rel(got, ref) < 1e-2


@pytest.mark.parametrize("d,rope_dim,sections", [(128, 64, [11, 11, 10, 0]), (128, 128, [24, 20, 20, 0]), (64, 64, [16, 8, 8, 0])])
def test_mrope_and_rope_table(d, rope_dim, sections):
    torch.manual_seed(4)
    t, hq, hkv = 21, 4, 2
    qkv = torch.randn(t, (hq + 2 * hkv) * d).bfloat16().cuda()
    pos = torch.randint(0, 3000, (t,), dtype=torch.int32).cuda()
    pos3 = torch.stack([pos, torch.randint(0, 50, (t,), dtype=torch.int32).cuda(), torch.randint(0, 50, (t,), dtype=torch.int32).cuda()]).contiguous()
    slots = torch.arange(t, dtype=torch.int32).cuda()
    qw, kw = (torch.rand(d) + 0.5).bfloat16().cuda(), (torch.rand(d) + 0.5).bfloat16().cuda()
    table = ew.rope_table(4096, rope_dim, 1e6, "cuda")
    for p3, sec in ((None, None), (pos3, sections)):
        kc = torch.zeros(t, hkv, d, dtype=torch.bfloat16, device="cuda")
        vc = torch.zeros_like(kc)
        q = ew.qk_norm_rope(qkv, pos, slots, qw, kw, kc, vc, hq, hkv, d, 1e6, 1e-6, 0.125, rope_dim, table=table, positions3=p3, sections=sec)
        rq, rk, rv = ew.qk_norm_rope_ref(qkv.cpu(), pos.cpu(), qw.cpu(), kw.cpu(), hq, hkv, d, 1e6, 1e-6, 0.125, rope_dim,
                                         p3.cpu() if p3 is not None else None, sec)
        assert _rel(q, rq) < 1e-2 and _rel(kc, rk) < 1e-2 and torch.equal(vc.cpu(), rv)
        # without the table the kernel computes the angles itself: same result
        kc2, vc2 = torch.zeros_like(kc), torch.zeros_like(vc)
        q2 = ew.qk_norm_rope(qkv, pos, slots, qw, kw, kc2, vc2, hq, hkv, d, 1e6, 1e-6, 0.125, rope_dim, positions3=p3, sections=sec)
        assert _rel(q2, rq) < 1e-2 and _rel(kc2, rk) < 1e-2
