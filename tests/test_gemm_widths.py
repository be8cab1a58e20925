"""Tile widths of the bf16 GEMM on CTA pairs: one accumulator of 128 to 256 columns, two of together 352 to 512, in the three operand
layouts, with reductions around the batches at a wide tile's ends (three k-blocks of 64) and columns that end inside a tile, an
accumulator, a store box and a 16-byte piece, against fp64."""
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

CUDA = Path(__file__).resolve().parents[1] / "roc_shmem_b200" / "csrc" / "cuda"
# (rows, columns, pairs): width with K-major B, width with MN-major B
PLANS = {(512, 1024, 1): (512, 512), (520, 840, 2): (448, 448), (264, 416, 1): (416, 416), (264, 352, 1): (352, 352), (1000, 1920, 4): (480, 480),
         (264, 200, 1): (224, 256), (264, 136, 1): (160, 256), (264, 120, 1): (128, 256), (776, 2040, 8): (512, 512), (520, 1400, 3): (480, 480)}


# grouped products: (groups, capacity, columns, reduction, counts on the device): widths of the plain form, the gated one, the one
# that keeps activations, and the weight gradient's (its rows are the columns of the first operand, 1024 here)
GROUPED = {(2, 4096, 3840, 1536, True): (384, 384, 256, 512), (2, 1024, 256, 200, True): (128, 128, 128, 256), (3, 2048, 8192, 2048, True): (512, 512, 256, 512),
           (1, 1280, 7168, 8192, False): (512, 512, 512, 512), (1, 1280, 5888, 8192, False): (448, 512, 448, 384)}


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_plan(tmp_path):
    """Every plan's accumulators are what the tensor core and the shared memory take, and the sizes below get the widths that
    they are there for."""
    checks = "".join(f"if (w({m}, {n}, 1536, {p}, {b}) != {ws[b]}) {{ printf(\"{m} {n} {p} {b}: %d\\n\", w({m}, {n}, 1536, {p}, {b})); return 1; }}\n"
                     for (m, n, p), ws in PLANS.items() for b in (0, 1))
    for (g, cap, n, k, counted), ws in GROUPED.items():
        exact = "false" if counted else "true"
        mb = g * -(-((4 * cap + 4) // 5 if counted else cap) // 256)
        for args, width in zip((f"{mb}, {n}, {k}, 74, 64, false, {exact}", f"{mb}, {n}, {k}, 74, 128, false, {exact}",
                                f"{mb}, {n}, {k}, 74, 64, false, {exact}, 512, 8000", f"{4 * g}, {n}, {4 * cap // 5}, 74, 128, true"), ws):
            checks += f"{{ Width x = plan_width({args}); if (x.cols[0] + x.cols[1] != {width}) {{ printf(\"{args}: %d\\n\", x.cols[0] + x.cols[1]); return 1; }} }}\n"
    (tmp_path / "t.cc").write_text("#include <cstdio>\n#include <initializer_list>\n#include \"pair_plan.h\"\nusing namespace bshmem::gemm2;\n" + """
int w(int m, int n, int k, int p, bool b) { Width x = plan_width((m + 255) / 256, n, k, p, 32, b); return x.cols[0] + x.cols[1]; }
int main() {
  for (int m = 1; m < 9000; m = m * 3 / 2 + 1)
    for (int n = 1; n < 30000; n = n * 4 / 3 + 1)
      for (int k = 1; k < 20000; k = k * 3 + 1)
        for (int p : {1, 3, 37, 74})
          for (int b = 0; b < 6; ++b) {
            const int step = 32 << b / 2;
            const Width x = plan_width((m + 255) / 256, n, k, p, step, b & 1);
            const int a = x.cols[0], c = x.cols[1];
            if (a % step || c % step || a < 128 || a > 256 || (c && (c < 128 || c > a))) { printf("%d %d %d %d %d: %d %d\\n", m, n, k, p, b, a, c); return 1; }
          }
""" + checks + """  puts("ok");
}
""")
    exe = tmp_path / "t"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", str(CUDA), "-o", str(exe), str(tmp_path / "t.cc")], capture_output=True, text=True)
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


def _split(gu):
    """Interleaved pre-activations [R, 2F] (32 gate columns, 32 up columns, ...) as (gate, up), [R, F] each."""
    v = gu.view(gu.shape[0], gu.shape[1] // 64, 2, 32)
    return v[:, :, 0].reshape(gu.shape[0], -1), v[:, :, 1].reshape(gu.shape[0], -1)


@pytest.mark.gpu
@pytest.mark.parametrize("G,cap,N,K,counted", list(GROUPED))
def test_grouped_widths(G, cap, N, K, counted):
    """All forms on CTA pairs with counts that end inside tiles; the last tile of a group's columns reaches into the next group's weights,
    and nothing of that may be stored."""
    from roc_shmem_b200.ops.moe import grouped_gemm, grouped_gemm_act, grouped_gemm_swiglu_bwd, grouped_gemm_tn, moe_lib, zero_pad_rows
    torch.manual_seed(G + cap + N)
    bf, u = torch.bfloat16, 2.0 ** -8                       # u: one rounding to bf16; fp32 sums of K products: K / 2^24
    rows = [cap - 37 * (g + 1) if g != 1 else 1 for g in range(G)] if counted else [cap]
    cnt = torch.tensor(rows, dtype=torch.int32, device="cuda")
    new = lambda c: torch.full((G * cap, c), 7.0, dtype=bf, device="cuda")
    a, w = torch.randn(G * cap, K, device="cuda").to(bf), (torch.randn(G * N, K, device="cuda") * K ** -0.5).to(bf)
    plain, gated, gu, act, dgu = new(N), new(N // 2), new(N), new(N // 2), new(2 * N)
    some = cnt if counted else None
    pre = torch.randn(G * cap, 2 * N, device="cuda").to(bf)
    grouped_gemm(a, w, plain, G, rows=some)
    grouped_gemm(a, w, gated, G, rows=some, gated=True)
    grouped_gemm_act(a, w, gu, act, G, rows=some)
    grouped_gemm_swiglu_bwd(a, w, pre, dgu, G, rows=some)
    xt, yt = torch.randn(G * cap, 1024, device="cuda").to(bf), torch.randn(G * cap, N, device="cuda").to(bf)
    zero_pad_rows((xt, yt), G, cnt)
    dw = torch.full((G * 1024 + 1, N), 7.0, dtype=bf, device="cuda")
    grouped_gemm_tn(xt, yt, dw[:G * 1024], G, cnt)
    torch.cuda.synchronize()
    assert moe_lib().bshmem_moe_gemm_error_site(1) == 0 and bool((dw[G * 1024] == 7).all())
    for g, n in enumerate(rows):
        used, rest = slice(g * cap, g * cap + n), slice(g * cap + -(-n // 32) * 32, (g + 1) * cap)     # stored by 32 rows
        assert all(bool((t[rest] == 7).all()) for t in (plain, gated, gu, act, dgu))
        x, y = a[used].double(), w[g * N:(g + 1) * N].double().t()
        ref, sums = x @ y, K * 2 ** -24 * (x.abs() @ y.abs())
        for t in (plain, gu):
            assert bool(((t[used].double() - ref).abs() <= ref.abs() * u + sums).all())
        for t, start in ((act, gu[used].double()), (gated, ref)):     # from the rounded pre-activations, or from the sums
            gate, up = _split(start)
            h = gate * torch.sigmoid(gate) * up
            eg, eu = _split(sums if t is gated else torch.zeros_like(sums))
            # |silu'| <= 1.1; 2^-18: __expf
            tol = h.abs() * (u + 2 ** -18) + (1.1 * eg * (up.abs() + eu) + eu * (gate * torch.sigmoid(gate)).abs()) * (1 + u) + 1e-30
            assert bool(((t[used].double() - h).abs() <= tol).all())
        gate, up = _split(pre[used].double())
        s = torch.sigmoid(gate)
        dtol = ref.abs() * u + sums                          # the accumulator is rounded to bf16 on the way
        # the factor 1 + g (1 - s) cancels near its zero: its error is absolute, up to |g| 2^-18 (fp32 and __expf)
        fg, fu = up * s * (1 + gate * (1 - s)), gate * s
        fg_err, fu_err = up.abs() * s * (1 + gate.abs()) * 2 ** -18, fu.abs() * 2 ** -18
        for got, f, ferr in zip(_split(dgu[used].double()), (fg, fu), (fg_err, fu_err)):
            tol = (ref * f).abs() * u + (dtol * f.abs() + (ref.abs() + dtol) * ferr) * (1 + u) + 1e-30
            assert bool(((got - ref * f).abs() <= tol).all())
        x, y = xt[used].double().t(), yt[used].double()
        ref = x @ y
        assert bool(((dw[g * 1024:(g + 1) * 1024].double() - ref).abs() <= ref.abs() * u + n * 2 ** -24 * (x.abs() @ y.abs())).all())
