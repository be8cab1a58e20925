"""Tile widths of the bf16 GEMM on CTA pairs: one accumulator of 128 to 256 columns, two of together 352 to 512, in the three operand
layouts, with reductions around the batches at a wide tile's ends (three k-blocks of 64) and columns that end inside a tile, an
accumulator, a store box and a 16-byte piece, against fp64."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"
# (rows, columns, pairs): width with K-major B, width with MN-major B
PLANS = {(512, 1024, 1): (512, 512), (520, 840, 2): (448, 448), (264, 416, 1): (416, 416), (264, 352, 1): (352, 352), (1000, 1920, 4): (480, 480),
         (264, 200, 1): (224, 256), (264, 136, 1): (160, 256), (264, 120, 1): (128, 128), (776, 2040, 8): (512, 512), (520, 1400, 3): (352, 480)}


def _plan_source() -> str:
    text = (CUDA / "gemm_bf16.cu").read_text()
    i = text.index("struct Width {")
    return text[i:text.index("return best;", i)] + "return best;\n}\n"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_plan(tmp_path):
    """Every plan's accumulators are what the tensor core and the shared memory take, and the sizes below get the widths that
    they are there for."""
    checks = "".join(f"if (w({m}, {n}, 1536, {p}, {b}) != {ws[b]}) {{ printf(\"{m} {n} {p} {b}: %d\\n\", w({m}, {n}, 1536, {p}, {b})); return 1; }}\n"
                     for (m, n, p), ws in PLANS.items() for b in (0, 1))
    (tmp_path / "t.cc").write_text("#include <cstdio>\n#include <initializer_list>\nconstexpr int BM = 256, BN = 256, BK = 64;\n" + _plan_source() + """
int w(int m, int n, int k, int p, bool b) { Width x = plan_width(m, n, k, p, b); return x.cols[0] + x.cols[1]; }
int main() {
  for (int m = 1; m < 9000; m = m * 3 / 2 + 1)
    for (int n = 1; n < 30000; n = n * 4 / 3 + 1)
      for (int k = 1; k < 20000; k = k * 3 + 1)
        for (int p : {1, 3, 37, 74})
          for (int b = 0; b < 2; ++b) {
            const Width x = plan_width(m, n, k, p, b != 0);
            const int a = x.cols[0], c = x.cols[1];
            if (a % 32 || c % 32 || a < 128 || a > 256 || (c && (c < 160 || c > a))) { printf("%d %d %d %d %d: %d %d\\n", m, n, k, p, b, a, c); return 1; }
          }
""" + checks + """  puts("ok");
}
""")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,pairs", list(PLANS))
@pytest.mark.parametrize("K", [8, 64, 192, 200, 256, 384, 456, 1536])
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
def test_widths(M, N, pairs, K, layout):
    from roc_shmem_b200.ops.gemm import gemm_bf16, gemm_error_site
    a_mn, b_mn = layout == "tn", layout != "nt"
    torch.manual_seed(M + N + K)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda").to(torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda").to(torch.bfloat16)
    for cols in [N] if b_mn else [N, N - 1, N - 35]:
        buf = torch.full((M + 1, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
        bb = b if b_mn else b[:cols]
        for _ in range(2):                                   # the second call meets the first one's end
            gemm_bf16(a, bb, buf[:M, :cols], a_mn=a_mn, b_mn=b_mn, max_ctas=2 * pairs)
        torch.cuda.synchronize()
        assert gemm_error_site() == 0
        assert bool((buf[:, cols:] == 7).all()) and bool((buf[M] == 7).all())
        # bf16 result, and fp32 sums of K products in any order
        x, y = (a.double().t() if a_mn else a.double()), (bb.double() if b_mn else bb.double().t())
        ref = x @ y
        err = (buf[:M, :cols].double() - ref).abs()
        assert bool((err <= ref.abs() * 2 ** -8 + K * 2 ** -24 * (x.abs() @ y.abs())).all()), err.max().item()
