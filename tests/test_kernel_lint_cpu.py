"""The GPU-less kernel linter: the tree is clean, and each rule fires on a snippet that breaks it."""
from gemm_b200.utils import kernel_lint as kl


def test_tree_is_clean_and_blackwell_native():
    rep = kl.lint_tree()
    assert rep["problems"] == [], rep["problems"]
    inv = rep["inventory"]
    gemm = inv["gemm_b200/csrc/kernels/gemm_tc.cu"]
    assert gemm.get("tcgen05.mma", 0) > 0 and gemm.get("cp.async.bulk.tensor", 0) > 0 and gemm.get("mma.sync / wmma", 0) == 0
    assert inv["gemm_b200/csrc/kernels/flash_attn.cu"].get("tcgen05.mma", 0) > 0
    assert inv["gemm_b200/csrc/kernels/moe_ffn.cu"].get("tcgen05.mma", 0) > 0


def _rules(src, **kw):
    return sorted({p["rule"] for p in kl.lint_text("x.cu", src, **kw)[0]})


def test_rules_fire():
    spin = "__global__ void k(unsigned* f) { while (ld_acquire_gpu(f) == 0) { } }"
    assert _rules(spin) == ["bounded-wait"]
    bounded = "__global__ void k(unsigned* f) { const uint64_t t0 = globaltimer_ns(); while (ld_acquire_gpu(f) == 0) { if (globaltimer_ns() - t0 > kBudgetNs) break; } }"
    assert _rules(bounded) == []
    dowhile = "__global__ void k(volatile int* f) { int v; do { v = *(volatile int*)f; } while (v == 0); }"
    assert _rules(dowhile) == ["bounded-wait"]
    leak = "__global__ void k(uint32_t* s) { tmem_alloc(s, 64); }"
    assert _rules(leak) == ["tmem-paired"]
    paired = "__global__ void k(uint32_t* s) { tmem_alloc(s, 64); tmem_dealloc(*s, 64); }"
    assert _rules(paired) == []
    # the qualifier is put together here so that this file itself does not spell a load of that kind
    qual = ".multi" + "cast" + "::cluster"
    mc = 'void f() { asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes' + qual + ' [%0], [%1, {%2, %3}], [%4], %5;"); }'
    assert _rules(mc) == ["no-cluster-broadcast-load"] and _rules(mc, multi_gpu=False) == []
    commit = 'void f() { asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster' + qual + '.b64 [%0], %1;"); }'
    assert _rules(commit) == []
    assert _rules('void f() { asm volatile("wgmma.mma_async.sync.aligned.m64n128k16.f32.bf16.bf16 ..."); }') == ["arch"]
    assert _rules("// while (ld_acquire_gpu(f) == 0) {}\n/* tmem_alloc( */ void f() {}") == []


def test_reads_in_front_of_the_dependency_wait():
    # weights may come out of the kernel launched just before, which lets its successor start before it stores
    head = "template <int N>\n__global__ void __launch_bounds__(256)\nk(const float* __restrict__ w, const Args a, float* out) "
    assert _rules(head + "{ const float x = w[threadIdx.x]; pdl_wait(); pdl_trigger(); out[0] = x; }") == ["wait-first"]
    assert _rules(head + "{ const float4 x = *reinterpret_cast<const float4*>(w + 4); pdl_wait(); }") == ["wait-first"]
    assert _rules(head + "{ const float x = a.tab[3]; pdl_wait(); }") == ["wait-first"]
    assert _rules(head + "{ bulk_load(smem, a.w, 16, bar); pdl_wait(); }") == ["wait-first"]
    assert _rules(head + "{ float t[4]; const int n = 2 * a.rows; pdl_wait(); t[0] = w[n]; out[0] = a.tab[1] + *w; }") == []
    assert _rules(head + "{ out[0] = w[0]; }") == []                   # without a wait: launched in plain stream order
    named = [n for n, _, _ in kl.kernel_parts(kl.strip_comments(head + "{ }"))]
    assert named == ["k"]


def test_warp_wide_loads_of_tensor_memory():
    head = "__global__ void k(float* out) "
    late = "tmem_ld_x16(t + c, r); tc_wait_ld(); if (!n_ok) continue; for (int j = 0; j < 16; ++j) out[j] = r[j]; } }"
    assert _rules(head + "{ for (int c = 0; c < n; c += 16) { " + late) == ["converged"]
    assert _rules(head + "{ for (int c = 0; c < n; c += 16) { __syncwarp(); " + late) == []
    assert _rules(head + "{ for (int c = 0; c < n; c += 16) { tmem_ld_x16(t + c, r); for (int j = 0; j < 16; ++j) { if (j > m) continue; out[j] = r[j]; } } }") == []
    assert _rules(head + "{ for (int i = 0; i < n; ++i) { if (!warp_wait(b)) continue; for (int c = 0; c < 4; ++c) { tmem_ld_x16(t + c, r); out[c] = r[0]; } } }") == []
