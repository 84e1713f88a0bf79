"""Which gate / up projections run on SM pairs (csrc/kernels/gemm_pair.cuh) and in which order wide layers walk their tiles (csrc/kernels/gemm_tc.cu): the host's
rules on both sides of each of their lines, for 148 SMs."""
import pytest

from gemm_b200 import _native


@pytest.mark.parametrize("m,n,k,pairs", [
    (65, 3072, 1024, False), (96, 3072, 1024, False), (97, 3072, 1024, True), (512, 3072, 1024, True),          # few tokens
    (80, 12288, 4096, False), (112, 10240, 2560, False), (129, 10240, 2560, True),                              # one tile of up to 128 tokens
    (320, 6144, 2048, False), (256, 8192, 2048, True), (512, 6144, 2048, True),                                 # a full round of single tiles
    (256, 2048, 4096, True), (256, 2048, 8192, False), (1300, 2048, 8192, True),                                # long k in one round
    (320, 12288, 4096, False), (384, 11008, 4096, False), (400, 11008, 4096, True), (512, 12288, 4096, True),   # rounds of either form
    (97, 25600, 5120, False), (256, 25600, 5120, True), (8300, 12288, 4096, True)])
def test_rule(m, n, k, pairs):
    assert bool(_native.cuda().gb_gemm_takes_pairs(n, k, m, 148)) == pairs


@pytest.mark.parametrize("n,m,tn,quant,group", [
    (18944, 2048, 256, 0, 8), (18816, 2048, 256, 0, 0),          # 148 and 147 blocks of features
    (18944, 257, 256, 0, 8), (18944, 256, 256, 0, 0),            # two token tiles, one
    (25600, 512, 128, 1, 8), (25600, 400, 128, 1, 0), (25600, 400, 128, 0, 8)])          # a ragged last tile: not with the quantising epilogue
def test_order_of_tiles(n, m, tn, quant, group):
    assert _native.cuda().gb_gemm_token_group(n, m, tn, quant, 148) == group
