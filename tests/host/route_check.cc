// Host-side checks of the kernel library's pure decision code: the division constants used for
// tile coordinates, and which convolution descriptors take which route.  Prints one line per
// check ("ok <name>" / "FAIL <name> ...") and exits non-zero on any failure.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <random>
#include <string>

#include "contract_route.h"
#include "conv_route.h"
#include "tc_gemm.cuh"

static int failures = 0;
static void check(bool ok, const char* name) {
  std::printf("%s %s\n", ok ? "ok" : "FAIL", name);
  if (!ok) ++failures;
}

static uint32_t apply(uint32_t n, pmlb::FastDiv f) {
  return static_cast<uint32_t>((static_cast<unsigned long long>(n) * f.mul) >> f.shift);
}

static pmlb_conv_desc conv(int n, int h, int w, int c, int r, int s, int k, int stride, int pad, int epi = 0) {
  pmlb_conv_desc d = {};
  d.in_dtype = PMLB_BF16;
  d.out_dtype = PMLB_BF16;
  d.n = n; d.h = h; d.w = w; d.c = c; d.r = r; d.s = s; d.k = k;
  d.stride_h = d.stride_w = stride;
  d.pad_h = d.pad_w = pad;
  d.dil_h = d.dil_w = 1;
  d.p = (h + 2 * pad - r) / stride + 1;
  d.q = (w + 2 * pad - s) / stride + 1;
  d.epilogue = epi;
  return d;
}

// out[c] += a[a] * b[b], one letter per index variable, everything dense f32.
static pmlb::GenericParams contraction(const char* a, const char* b, const char* c, std::map<char, long long> ext) {
  pmlb::GenericParams p;
  std::memset(&p, 0, sizeof(p));
  p.agg = PMLB_AGG_SUM;
  p.combo = PMLB_COMBO_MUL;
  p.n_src = 2;
  p.direct = 1;
  p.out_elems = 1;
  std::map<char, int> var;
  for (const auto& e : ext) {
    var[e.first] = p.n_idx;
    p.range[p.n_idx++] = e.second;
  }
  auto fill = [&](pmlb::GAccess* t, const std::string& dims) {
    t->dtype = PMLB_F32;
    t->rank = static_cast<int>(dims.size());
    long long stride = 1;
    for (int d = t->rank - 1; d >= 0; --d) {
      t->sizes[d] = ext[dims[d]];
      t->strides[d] = stride;
      stride *= t->sizes[d];
      t->den[d] = 1;
      t->coef[d][var[dims[d]]] = 1;
    }
  };
  fill(&p.out, c);
  fill(&p.src[0], a);
  fill(&p.src[1], b);
  for (int d = 0; d < p.out.rank; ++d) {
    p.out_var[d] = var[c[d]];
    p.out_elems *= p.out.sizes[d];
  }
  return p;
}

int main() {
  // n / d for every small pair and for random pairs up to 2^31 - 1
  bool ok = true;
  for (uint32_t d = 1; d < 3000 && ok; ++d) {
    const pmlb::FastDiv f = pmlb::make_fastdiv(d);
    for (uint32_t n = 0; n < 12000; ++n) ok = ok && apply(n, f) == n / d;
  }
  check(ok, "fastdiv small");
  std::mt19937_64 g(7);
  ok = true;
  for (int i = 0; i < 4000000 && ok; ++i) {
    uint32_t d = static_cast<uint32_t>(g() & 0x7fffffffu) | 1u;
    if (i & 1) d = d % 100000u + 1u;
    const uint32_t n = static_cast<uint32_t>(g() & 0x7fffffffu);
    ok = apply(n, pmlb::make_fastdiv(d)) == n / d;
  }
  check(ok, "fastdiv random");
  const uint32_t edge[] = {1u, 2u, 3u, 0x40000000u, 0x40000001u, 0x7fffffffu};
  ok = true;
  for (uint32_t d : edge) {
    for (uint32_t n : {0u, 1u, d - 1u, d, d + 1u, 0x7ffffffeu, 0x7fffffffu}) {
      if (n <= 0x7fffffffu) ok = ok && apply(n, pmlb::make_fastdiv(d)) == n / d;
    }
  }
  check(ok, "fastdiv edges");

  // routes of ResNet-50's convolutions
  check(pmlb::conv_takes_s2d(conv(256, 224, 224, 3, 7, 7, 64, 2, 3, PMLB_EPI_BIAS | PMLB_EPI_RELU)), "7x7/2 on 3 channels: space to depth");
  check(!pmlb::conv_takes_s2d(conv(2, 33, 45, 4, 5, 5, 48, 2, 2)), "output width 23: not space to depth");
  check(pmlb::conv_takes_packed_rows(conv(2, 33, 45, 4, 5, 5, 48, 2, 2)), "... but packed rows");
  check(!pmlb::conv_takes_s2d(conv(2, 20, 20, 3, 3, 3, 64, 2, 1, PMLB_EPI_RESIDUAL)), "residual input: not space to depth");
  check(!pmlb::conv_takes_s2d(conv(2, 64, 64, 8, 3, 3, 64, 2, 1)), "8 channels: not space to depth");
  check(!pmlb::conv_takes_s2d(conv(1, 1024, 1024, 3, 7, 7, 64, 2, 3)), "1024-wide rows: tile buffers do not fit");
  check(pmlb::conv_takes_halo(conv(256, 56, 56, 64, 3, 3, 64, 1, 1)), "3x3 64 -> 64 at 56x56: halo rows");
  check(!pmlb::conv_takes_halo(conv(256, 28, 28, 128, 3, 3, 128, 1, 1)), "128 output channels: im2col");
  check(!pmlb::conv_takes_halo(conv(256, 56, 56, 64, 3, 3, 64, 2, 1)), "stride 2: im2col");
  check(!pmlb::conv_takes_halo(conv(4, 7, 7, 64, 3, 3, 64, 1, 1)), "7x7 image: too few real rows per tile");
  // shapes of the space-to-depth form
  {
    const pmlb::S2dShape g = pmlb::conv_s2d_shape(conv(256, 224, 224, 3, 7, 7, 64, 2, 3));
    check(g.pe_h == 4 && g.dh == 1 && g.r2 == 4 && g.s2 == 4 && g.h2 == 115 && g.wp == 128 && g.stage_px == 928,
          "7x7/2 pad 3 -> 4x4 taps, 115 rows of 128 pixels, 928 pixels per tile");
    const pmlb::S2dShape e = pmlb::conv_s2d_shape(conv(2, 20, 22, 2, 4, 2, 16, 2, 1));
    check(e.pe_h == 2 && e.dh == 1 && e.r2 == 3 && e.s2 == 2 && e.wp % 32 == 0 && e.stage_px % 32 == 0, "even filter, odd padding");
  }
  // contractions: which are matrix products, and which of these pay on the tensor cores (us: the tiles' estimate)
  {
    pmlb::ProductForm f;
    pmlb::LeanParams l;
    auto form = [&](const pmlb::GenericParams& p, long long b, long long m, long long n, long long k) {
      return pmlb::product_form(p, &f) && pmlb::lean_form(p, &l) && f.batch == b && f.m == m && f.n == n && f.k == k;
    };
    check(form(contraction("km", "kn", "mn", {{'k', 4096}, {'m', 512}, {'n', 512}}), 1, 512, 512, 4096) && f.am == 1 && f.ak == 512 &&
              pmlb::product_pays(f, true, 24.0),
          "weight gradient: product");
    check(form(contraction("ij", "ij", "ij", {{'i', 1024}, {'j', 1024}}), 1 << 20, 1, 1, 1) && !pmlb::product_pays(f, true, 1.0),
          "element-wise product: strided");
    check(form(contraction("yc", "c", "yc", {{'c', 128}, {'y', 100352}}), 128, 100352, 1, 1) && !pmlb::product_pays(f, true, 1.0),
          "scale per channel: strided");
    check(form(contraction("i", "j", "ij", {{'i', 4096}, {'j', 4096}}), 1, 4096, 4096, 1) && !pmlb::product_pays(f, true, 1.0),
          "outer product: strided");
    check(form(contraction("ik", "ik", "i", {{'i', 65536}, {'k', 64}}), 65536, 1, 1, 64) && !pmlb::product_pays(f, true, 2400.0) &&
              pmlb::product_pays(f, true, 10.0),
          "many short dot products: strided unless the estimate is small");
    check(form(contraction("km", "kn", "mn", {{'k', 15}, {'m', 512}, {'n', 512}}), 1, 512, 512, 15) && !pmlb::product_pays(f, false, 1.0),
          "fifteen terms: never on the tensor cores");
    check(form(contraction("km", "kn", "mn", {{'k', 16}, {'m', 128}, {'n', 128}}), 1, 128, 128, 16) && pmlb::product_pays(f, true, 5.5) &&
              !pmlb::product_pays(f, true, 6.0),
          "sixteen terms: by the estimate");
  }
  return failures == 0 ? 0 : 1;
}
