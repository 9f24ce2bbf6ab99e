"""The forms that the default rules choose for quantized products on 148 SMs, without a GPU: a program linked against the library's objects asks
the rules themselves."""
import glob
import os
import subprocess

import pytest

from torchlette_b200 import _build
from torchlette_b200 import binding as B

ASK = """
#include <cstdio>
#include "tl_common.cuh"
int main() {
  long long m, n, k;
  int group, bf16, int4_out;
  while (std::scanf("%lld %lld %lld %d %d %d", &m, &n, &k, &group, &bf16, &int4_out) == 6) {
    tl_quant_desc q{};
    if (int4_out >= 0) {  // a receipt of an int4 product
      tl_ctx ctx;
      ctx.sm_count = 148;
      q.scheme = TL_SCHEME_INT4_GROUPED;
      q.group_size = group ? group : int(k);
      q.scales_dtype = TL_F16;
      tl_plan_receipt r;
      if (tl_plan_qmatmul(&ctx, m, n, k, bf16 ? TL_BF16 : TL_F16, int4_out, &q, nullptr, &r) != TL_OK) return 1;
      std::printf("%d %d %d\\n", r.choice.p0, r.choice.p1, r.choice.p2);
      continue;
    }
    q.scheme = TL_SCHEME_INT8_GROUPED;
    q.group_size = group ? group : int(k);
    q.scales_dtype = TL_F16;
    tl_variant v;
    if (bf16 == 2) {  // f32 activations, a small batch
      tl_qgemv_default_variant(nullptr, int(m), n, k, TL_F32, q, &v);
      std::printf("%d %d %d\\n", v.kernel, v.p0, v.p1);
      continue;
    }
    tl_qgemm_default_variant(nullptr, m, n, k, bf16 ? TL_BF16 : TL_F16, q, &v);
    std::printf("%d %d %d %d %d %d\\n", v.kernel, v.p0, v.p1, v.p2, v.p3, tl_dense_tc_choose(m, n, k, 148).parts);
  }
}
"""
FUSED, DEQUANT_DENSE = 0, 2


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    _build.build()
    d = tmp_path_factory.mktemp("rule")
    src, exe = d / "ask.cpp", d / "ask"
    src.write_text(ASK)
    cuda = os.path.dirname(os.path.dirname(_build.NVCC))
    subprocess.run(["g++", "-std=c++17", "-I", _build.CSRC, "-I", os.path.join(cuda, "include"), str(src), *glob.glob(os.path.join(_build.CSRC, "*.o")),
                    "-L", os.path.join(cuda, "lib64"), "-lcudart_static", "-ldl", "-lpthread", "-lrt", "-o", str(exe)], check=True)

    def ask(*shapes):
        text = "".join(" ".join(map(str, s if len(s) == 6 else s + (-1,))) + "\n" for s in shapes)
        return [tuple(map(int, line.split())) for line in subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True).stdout.splitlines()]
    return ask


# m, n, k, group, bf16: dequantize + dense cuts K in two to eight; the fused kernel, which the faster converters make the quicker one by up to
# an eighth, would sum over all of K or over more of it
@pytest.mark.parametrize("shape", [(1999, 793, 4992, 64, 0), (445, 2130, 11136, 16, 1), (470, 4160, 13824, 64, 0), (177, 909, 9344, 64, 0),
                                   (224, 4976, 13312, 128, 1), (510, 3832, 10032, 48, 0), (250, 791, 9216, 64, 1), (233, 513, 8320, 32, 0)])
def test_a_faster_fused_kernel_takes_no_longer_sums(rule, shape):
    kernel, *_, parts = rule(shape)[0]
    assert kernel == DEQUANT_DENSE and parts > 1


def test_tiles_of_192_tokens_keep_eight_converter_warps(rule):
    got = rule((180, 100352, 4096, 64, 0), (150, 151936, 1024, 64, 1), (333, 12288, 4096, 0, 0))
    assert [g[:5] for g in got[:2]] == [(FUSED, 192, 128, 3, 8)] * 2
    assert got[2][4] == 8


@pytest.mark.parametrize("n,k,group,m,fewer,warps", [(2400, 4096, 32, 16, (8, 2), 16), (4700, 12288, 64, 9, (8, 2), 16), (4096, 1536, 32, 12, (8, 2), 8),
                                                     (9500, 4096, 64, 16, (4, 1), 8), (9500, 1024, 128, 1, (4, 1), 8), (30000, 1024, 32, 16, (4, 1), 8)])
def test_an_int4_product_with_f32_output_keeps_its_short_sums(rule, n, k, group, m, fewer, warps):
    """The forms with fewer warps a tile, hence longer sums, are for 16-bit outputs."""
    wide, half, bf16 = (r[:2] for r in rule((m, n, k, group, 0, B.DTYPE_ID["f32"]), (m, n, k, group, 0, B.DTYPE_ID["f16"]), (m, n, k, group, 1, B.DTYPE_ID["bf16"])))
    assert half == bf16 == fewer and wide == (warps, 1)


@pytest.mark.parametrize("m,rows_a_warp,beyond", [(1, 1, (8, 2)), (2, 1, (8, 4)), (3, 2, (8, 4)), (4, 2, (4, 4)), (16, 2, (4, 4))])
def test_f32_activations_take_more_rows_a_warp_where_one_wave_ends(rule, m, rows_a_warp, beyond):
    """32 rows an SM: four CTAs of eight warps with a row each, or two with two."""
    simt = 1
    got = rule(*[(m, n, 4096, 64, 2) for n in (4200, 4736, 4737, 5328, 7103)])
    assert got[:2] == [(simt, 8, rows_a_warp)] * 2
    assert got[2:] == [(simt,) + beyond] * 3
