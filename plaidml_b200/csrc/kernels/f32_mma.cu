// fp32 products on the tensor cores: every operand element x is cut into three bf16 parts x = h + m + l of 8
// significant bits each, h towards zero (the largest finite values stay finite), m to nearest, l what is left (exact for
// 24 bits, |m| < 2^-7 and |l| <= 2^-16 of x's power of two, l of either sign), and a product is six of the nine part
// products: hh + (hm + mh + hl + lh + mm).  The two next ones, ml and lm, are 2^-22 of the product at most and cancel
// over a sum: with m cut towards zero as well they reached 2^-21 and all had the product's sign (4e-8 of every sum of
// positive terms).  Error of a single product against 64 bits, in norm: 3.0e-8 (5.1e-8 with m cut; plain f32 2.5e-8,
// three TF32 products 6.6e-8), of sums of 8 to 4096 terms 0.6 to 0.2 times that of plain f32 sums.  bf16 parts end at
// 2^-133: operands below 2^-110 lose what lies under 2^-134 (2^-16 of themselves at 2^-118).
// bf16 MMAs run at twice the TF32 rate, so six of them cost what three TF32 products cost, but three parts keep 24 bits
// (two TF32 parts 22), occupy 6 bytes of shared memory per element instead of 8, and bf16 operands may be MN-major, so a
// [k][n] B or a transposed A needs no transposition.
//
// One CTA computes a 128 x BN tile (or the part of its K range that falls to it, see below):
//   warps 0..15  loaders: fp32 from global memory into registers one operand tile ahead, cut into the three parts,
//                stored in the 128-byte swizzle the MMA reads.  No pre-pass writes and re-reads split copies, and
//                any row alignment is accepted.
//   warp 24      MMA issuer.  hh goes into an accumulator of its own; the five small products share a second one:
//                the tensor core truncates when it adds to its accumulator, an error per MMA of a fraction of the
//                accumulator's last place, and the small sums must not drown in it.  [h | m] of B lie side by side
//                in shared memory, so one MMA of width 2 BN does hh and hm with one read of A.
//   warps 16..23 after every kFlushBlocks k-blocks (256 terms) they add both accumulators to sums in registers with
//                round-to-nearest while the issuer goes on with the other accumulator pair: chains of 16 MMAs instead
//                of k / 8.  Error against 64 bits at 2048 terms: 2.0e-7, three TF32 products in one chain 1.4e-5.
//   all warps    the sums go through shared memory (free by then) to row-contiguous 16-byte stores with the epilogue.
//
// Few tiles and a long K: `split` CTAs of a cluster share a tile, each a contiguous run of k-blocks; every CTA then
// adds a 128 / split-row strip of all parts through distributed shared memory, in rank order.  No scratch memory, no
// atomics, no second launch; the result depends only on the shape.
//
// CTA pairs (256 x 256 tiles) have room for one accumulator pair only: their chains run over the pair's whole part of K.
//
// What bounds it: 64- and 128-wide tiles the loaders: per k-block of a 128-wide tile 64 KB of loads, 98 KB of stores and
// 16,384 elements to cut, ~2300 cycles where the MMAs take 1536.  Copies of an earlier form (eight loader warps, 1024 x
// 1024 x 4096, 90.6 us) with work left out: without the loads 71.5 us, without the stores 69.3, with two of the five MMAs
// 85.3.  Over 73 shapes 16 loader warps instead of eight took -12 to +5 % (median 0; 2047 x 2049 x 513 38.4 -> 34.2 us,
// 2048 x 4096 x 100 26.6 -> 27.9), then offsets that stay in registers and packed additions -9 to +6 % (median -1; 256 x
// 4096 x 4096 51.8 -> 49.3, 301 x 303 x 305 7.0 -> 7.4): problems of 6 to 12 us gave up to 0.4 us for it.
// CTA pairs: the rate the tensor pipe sustains under the power limit (six products of 2048 x 2048 x 1024 in 41 us:
// 1.27 PFLOP/s, 1.6 in the loop).  Small problems: ~6 us of launch, first loads, last sums and stores.
// Measured (graph replays), split copies by a pre-pass -> here: 1 x 1000 x 2048 35 -> 11.4 us, 300^3 12.9 -> 6.9, 1024^3
// 22.0 -> 18.1, 256 x 4096 x 4096 96 -> 49, 512 x 512 x 4096 62 -> 22, 1999 x 2001 x 1001 71 -> 49; convolutions 8 x 28 x
// 28 x 128 -> 128, 3x3 25.5 -> 20.0, 32 x 7 x 7 x 512 -> 512, 3x3 63 -> 45 (pairs, K in parts), 1 x 7 x 7 x 512 61 -> 15.
// Walking several tiles per CTA with the stores behind the next tile's loads was slower (1024^3 21.2 us against 19.2).
//
// inf / NaN: h is inf / NaN, x - h is NaN, so only hh is right; a sum whose hh part is not finite drops its small part.
#include "f32_mma.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "pmlb_kernels.h"
#include "dependent_launch.h"
#include "ptx.cuh"
#include "tc_gemm.cuh"

namespace pmlb {

namespace {

constexpr int kLoaderWarps = 16;
constexpr int kSumWarps = 8;
constexpr int kThreads = (kLoaderWarps + kSumWarps + 4) * 32;   // (whole warpgroups: the issuer's has three idle warps)
// Registers per thread: 896 threads start with 72 (64,512 in all).  The loaders go down to 64 and the issuer's warpgroup
// to 40, which frees 8,192; the sums go up to 96, which takes 6,144.
constexpr int kIssuerRegs = 40, kLoaderRegs = 64, kSumRegs = 96;
constexpr int kIssuerWarp = kLoaderWarps + kSumWarps;
constexpr int kBlockK = 64;            // k-block: 64 terms = 128-byte bf16 rows
constexpr int kFlushBlocks = 4;        // k-blocks per accumulator chain
constexpr int kPartA = 128 * 128;      // bytes of one part of an A tile

enum : int { kRowsK = 0, kRowsMn = 1, kRowsConv = 2 };   // operand layouts: k contiguous, m / n contiguous, im2col

struct F32MmaParams {
  int m, n, k;
  int tiles_n, tiles_per_batch;
  int num_kb;
  int split;                    // CTAs that share a tile's K range
  int one_order;                // 64-wide tiles: the small products in one accumulator, in the order of 128-wide ones
  const float* a;
  const float* b;
  long long lda, ldb, a_batch, b_batch;
  // convolution
  int c, h, w, p, q, s, stride_h, stride_w, pad_h, pad_w, dil_h, dil_w;
  FastDiv fd_c, fd_s, fd_pq, fd_q;
  float* out;
  long long ldc, out_batch;
  int out_vec;                  // output (and residual) rows start on 16-byte boundaries
  int epi_flags;
  const float* bias;
  const float* residual;
  long long ldr, res_batch;
  float* rowmax;
  int* status;
};

// BN: columns of a tile.  64, 128: one CTA per 128-row tile.  256: a CTA pair per 256-row tile, each CTA with its 128
// rows of A and half of B's columns.
template <int BN>
struct F32Cfg {
  static constexpr bool kPair = BN == 256;
  static constexpr int kColsB = kPair ? BN / 2 : BN;   // columns of B that a CTA holds
  static constexpr int kPartB = kColsB * 128;
  static constexpr int kStageBytes = 3 * (kPartA + kPartB);
  static constexpr int kStages = BN == 64 ? 3 : 2;
  static constexpr int kSmem = kStages * kStageBytes + 1024 + 256;
  // hh, then the small products (BN == 64: these in two accumulators side by side, so that the middle part of A also
  // meets [h | m] in one MMA).  Pairs: one accumulator pair fills TMEM, so their chains run over all of K.
  static constexpr int kAccCols = kPair ? 512 : 256;
};

// 32 lanes x 8 (16) columns of 32-bit accumulators.
__device__ __forceinline__ void tmem_ld_8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}

__device__ __forceinline__ void tmem_ld_16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ uint32_t upper_halves(float lo, float hi) {
  return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
}

// Two floats cut to bf16, x in the lower half.  Not upper_halves: NaN stays NaN also where its payload is in the bits that
// are cut off.
__device__ __forceinline__ uint32_t cut_to_bf16(float x, float y) {
  uint32_t r;
  asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
  return r;
}

__device__ __forceinline__ uint32_t round_to_bf16(float x, float y) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
  return r;
}

// (a, b) + (c, d) in one instruction.
__device__ __forceinline__ float2 add2(float a, float b, float c, float d) {
  float2 r;
  asm("{\n\t"
      ".reg .b64 x, y;\n\t"
      "mov.b64 x, {%2, %3};\n\t"
      "mov.b64 y, {%4, %5};\n\t"
      "add.rn.f32x2 x, x, y;\n\t"
      "mov.b64 {%0, %1}, x;\n\t"
      "}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a), "f"(b), "f"(c), "f"(d));
  return r;
}

__device__ __forceinline__ float2 sub2(float a, float b, float c, float d) {
  float2 r;
  asm("{\n\t"
      ".reg .b64 x, y;\n\t"
      "mov.b64 x, {%2, %3};\n\t"
      "mov.b64 y, {%4, %5};\n\t"
      "sub.rn.f32x2 x, x, y;\n\t"
      "mov.b64 {%0, %1}, x;\n\t"
      "}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a), "f"(b), "f"(c), "f"(d));
  return r;
}

// What is left of two floats without their upper halves (exact; NaN for inf).
__device__ __forceinline__ float2 rest_of(float x, float y) {
  // the upper half with its sign turned: one logic operation
  return add2(x, y, __uint_as_float((__float_as_uint(x) & 0xffff0000u) ^ 0x80000000u), __uint_as_float((__float_as_uint(y) & 0xffff0000u) ^ 0x80000000u));
}

__device__ __forceinline__ void st_shared_v2(uint32_t addr, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}

__device__ __forceinline__ void st_shared_b32(uint32_t addr, uint32_t x) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(x) : "memory");
}

// Cuts two elements into the three parts.  One conversion per part, as cheap as taking upper halves (1024^3 17.7 us both).
struct Parts {
  uint32_t h, m, l;
};
__device__ __forceinline__ Parts cut(float x, float y) {
  Parts c;
  c.h = cut_to_bf16(x, y);
  const float2 r = rest_of(x, y);
  c.m = round_to_bf16(r.x, r.y);
  const float2 l = sub2(r.x, r.y, __uint_as_float(c.m << 16), __uint_as_float(c.m & 0xffff0000u));
  c.l = upper_halves(l.x, l.y);
  return c;
}

// Stores 8 (4) bytes of each part of consecutive elements.
__device__ __forceinline__ void store_parts(uint32_t addr, uint32_t part_bytes, const float (&v)[4]) {
  const Parts a = cut(v[0], v[1]), b = cut(v[2], v[3]);
  st_shared_v2(addr, a.h, b.h);
  st_shared_v2(addr + part_bytes, a.m, b.m);
  st_shared_v2(addr + 2 * part_bytes, a.l, b.l);
}

__device__ __forceinline__ void store_parts(uint32_t addr, uint32_t part_bytes, const float (&v)[2]) {
  const Parts a = cut(v[0], v[1]);
  st_shared_b32(addr, a.h);
  st_shared_b32(addr + part_bytes, a.m);
  st_shared_b32(addr + 2 * part_bytes, a.l);
}

// One loader thread's share of an operand tile of ROWS rows (m or n) x 64 terms.  `origin`: row 0 of the tile, term 0
// of the problem; `rows`: rows that exist.  VEC: groups of four elements, 16-byte aligned.  Else groups of two, so that
// a warp's element loads still cover whole lines (four consecutive elements per lane would touch five lines per load).
template <int LAYOUT, int ROWS, bool VEC>
struct TileLoader {
  static constexpr int kGroup = VEC || LAYOUT == kRowsConv ? 4 : 2;
  static constexpr int kGroups = ROWS * kBlockK / (kLoaderWarps * 32 * kGroup);
  // m / n contiguous: groups along the row dimension, and the terms that one pass of the loaders covers
  enum : int { kMnGroups = ROWS / kGroup, kMnStep = kLoaderWarps * 32 / kMnGroups };
  // k contiguous: groups along k, and the rows of one pass
  enum : int { kKGroups = kBlockK / kGroup, kKStep = kLoaderWarps * 32 / kKGroups };
  float v[kGroups][kGroup];
  const float* origin;
  long long ld;
  int rows, k_end;
  bool plain;                 // whole k-blocks need no tests: see place()
  uint32_t at[kGroups];       // byte offset of each group from the k-block's first element (rows layouts only)
  // convolution: first tap's position and the image's offset of each of this thread's rows
  int base[LAYOUT == kRowsConv ? kGroups : 1];
  int yx[LAYOUT == kRowsConv ? kGroups : 1];

  // The first `valid` elements of group i, zeros behind them.
  __device__ __forceinline__ void fetch(int i, const float* q, int valid) {
#pragma unroll
    for (int e = 0; e < kGroup; ++e) v[i][e] = 0.f;
    if constexpr (VEC) {
      if (valid >= kGroup) {
        const float4 u = __ldg(reinterpret_cast<const float4*>(q));
        v[i][0] = u.x, v[i][1] = u.y, v[i][2] = u.z, v[i][3] = u.w;
        return;
      }
    }
#pragma unroll
    for (int e = 0; e < kGroup; ++e) {
      if (e < valid) v[i][e] = __ldg(q + e);
    }
  }
  // All of group i or none of it: one predicated load (or one per element).
  __device__ __forceinline__ void fetch_if(int i, const float* q, bool exists) {
#pragma unroll
    for (int e = 0; e < kGroup; ++e) v[i][e] = 0.f;
    if constexpr (VEC) {
      if (exists) {
        const float4 u = __ldg(reinterpret_cast<const float4*>(q));
        v[i][0] = u.x, v[i][1] = u.y, v[i][2] = u.z, v[i][3] = u.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < kGroup; ++e) {
        if (exists) v[i][e] = __ldg(q + e);
      }
    }
  }

  // After origin, ld, rows and k_end are set.  A thread's groups keep their places in every k-block, so a load is one
  // instruction: the block's address is the same for all threads, the offset never changes.  Groups of rows that do not
  // exist read the first group instead: what they bring reaches only results that are not stored.
  __device__ __forceinline__ void place(int tid) {
    plain = rows > 0 && ld < (1 << 23) && (LAYOUT == kRowsK || rows % kGroup == 0);
#pragma unroll
    for (int i = 0; i < kGroups; ++i) {
      const int row = LAYOUT == kRowsK ? tid / kKGroups + kKStep * i : (tid % kMnGroups) * kGroup;
      const int term = LAYOUT == kRowsK ? (tid % kKGroups) * kGroup : tid / kMnGroups + kMnStep * i;
      const uint32_t r = row < rows ? row : 0;
      at[i] = 4u * (LAYOUT == kRowsK ? r * static_cast<uint32_t>(ld) + term : term * static_cast<uint32_t>(ld) + r);
    }
  }

  __device__ __forceinline__ void load(int k0, const F32MmaParams& p, int tid) {
    if constexpr (LAYOUT == kRowsConv) {
      const int k = k0 + (tid % kKGroups) * kGroup;
      const int tap = fast_div(k, p.fd_c);
      const int ch = k - tap * p.c;
      const int fr = fast_div(tap, p.fd_s);
      const int dy = fr * p.dil_h, dx = (tap - fr * p.s) * p.dil_w;
      const int off = (dy * p.w + dx) * p.c + ch;
      const bool live = k < k_end;
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        const int y = (yx[i] >> 16) + dy, x = static_cast<int>(static_cast<short>(yx[i])) + dx;
        const bool in = live && static_cast<unsigned>(y) < static_cast<unsigned>(p.h) && static_cast<unsigned>(x) < static_cast<unsigned>(p.w);
        fetch_if(i, origin + base[i] + off, in);
      }
    } else if (plain && k0 + kBlockK <= k_end) {
      const char* block = reinterpret_cast<const char*>(origin + (LAYOUT == kRowsK ? k0 : k0 * ld));
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        if constexpr (VEC) {
          const float4 u = __ldg(reinterpret_cast<const float4*>(block + at[i]));
          v[i][0] = u.x, v[i][1] = u.y, v[i][2] = u.z, v[i][3] = u.w;
        } else {
#pragma unroll
          for (int e = 0; e < kGroup; ++e) v[i][e] = __ldg(reinterpret_cast<const float*>(block + at[i]) + e);
        }
      }
    } else if constexpr (LAYOUT == kRowsK) {
      const int k = k0 + (tid % kKGroups) * kGroup;
      const int r0 = tid / kKGroups;
      const float* q = origin + static_cast<long long>(r0) * ld + k;
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        fetch(i, q, r0 + kKStep * i < rows ? k_end - k : 0);
        q += kKStep * ld;
      }
    } else {
      const int mn = (tid % kMnGroups) * kGroup;
      const int kk = k0 + tid / kMnGroups;
      const float* q = origin + static_cast<long long>(kk) * ld + mn;
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        fetch(i, q, kk + kMnStep * i < k_end ? rows - mn : 0);
        q += kMnStep * ld;
      }
    }
  }

  // Cuts the elements into their three parts and stores them (kGroup * 2 bytes of each part per group).
  __device__ __forceinline__ void store(uint32_t tile, uint32_t part_bytes, int tid) const {
    if constexpr (LAYOUT == kRowsMn) {
      const int mn = (tid % kMnGroups) * kGroup;
      const int k = tid / kMnGroups;
      const uint32_t col = static_cast<uint32_t>(mn >> 6) * 8192u + static_cast<uint32_t>(mn & 7) * 2u;
      const uint32_t chunk = static_cast<uint32_t>(mn & 63) >> 3;
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        const uint32_t kk = static_cast<uint32_t>(k + kMnStep * i);
        store_parts(tile + col + kk * 128u + ((chunk ^ (kk & 7u)) << 4), part_bytes, v[i]);
      }
    } else {
      const uint32_t k = static_cast<uint32_t>(tid % kKGroups) * kGroup;
      const uint32_t r0 = static_cast<uint32_t>(tid / kKGroups);
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        const uint32_t r = r0 + kKStep * i;
        store_parts(tile + r * 128u + (((k >> 3) ^ (r & 7u)) << 4) + (k & 7u) * 2u, part_bytes, v[i]);
      }
    }
  }
};

__device__ __forceinline__ float atomic_max_f32(float* addr, float v) {
  // (order-preserving integer views of the two signs; the target starts at -inf)
  if (__float_as_int(v) >= 0) return __int_as_float(atomicMax(reinterpret_cast<int*>(addr), __float_as_int(v)));
  return __uint_as_float(atomicMin(reinterpret_cast<unsigned int*>(addr), __float_as_uint(v)));
}

// Arrive on a barrier of the cluster, this thread's (warp's) shared-memory stores before it.
__device__ __forceinline__ void mbar_arrive_release_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(cluster_addr)
               : "memory");
  return v;
}

// All threads of all CTAs of the cluster.  Not the .aligned form: the issuer's elected lane and lanes without columns to
// store arrive on their own, and an aligned arrive executed twice by one warp would release the barrier early.
__device__ __forceinline__ void cluster_sync_each_thread() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// tcgen05 instruction descriptor: bf16 operands, f32 accumulators, 128 (pair: 256) rows.
__host__ __device__ constexpr uint32_t mma_desc(int n, bool a_mn, bool b_mn, int m = 128) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u) |
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// The barrier between set-up and roles, one copy per role: each role has work of its own before it (loads on their way,
// TMEM), and a shared copy would make the compiler keep all of that within one role's registers.
template <int ROLE, bool PAIR>
__device__ __forceinline__ void setup_done() {
  if constexpr (PAIR) {   // (the other CTA's barriers must exist before anything is sent to them)
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;  // role %0" ::"n"(ROLE) : "memory");
  } else {
    asm volatile("bar.sync 0, %0;  // role %1" ::"n"(kThreads), "n"(ROLE) : "memory");
  }
}

// Accumulators' hh sums with their small products; those of inf / NaN operands are NaN and dropped.
template <int N>
__device__ __forceinline__ void both_parts(const uint32_t (&hh)[N], const uint32_t (&small)[N], float (&v)[N]) {
  bool nan = false;
#pragma unroll
  for (int e = 0; e < N; e += 2) {
    const float2 t = add2(__uint_as_float(hh[e]), __uint_as_float(hh[e + 1]), __uint_as_float(small[e]), __uint_as_float(small[e + 1]));
    v[e] = t.x, v[e + 1] = t.y;
    nan = nan || t.x != t.x || t.y != t.y;
  }
  if (nan) {
#pragma unroll
    for (int e = 0; e < N; ++e) {
      if (!(fabsf(__uint_as_float(hh[e])) < INFINITY)) v[e] = __uint_as_float(hh[e]);
    }
  }
}

// Bias, residual, ReLU and the store of `n` <= 4 consecutive results of row i from column j on.
__device__ __forceinline__ void finish(const F32MmaParams& p, int batch, int i, int j, float (&o)[4], int n) {
  if (p.epi_flags & kEpiBias) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e < n) o[e] += __ldg(p.bias + j + e);
    }
  }
  if (p.epi_flags & kEpiResidual) {
    const float* res = p.residual + batch * p.res_batch + static_cast<long long>(i) * p.ldr + j;
    if (p.out_vec && n >= 4) {
      const float4 u = __ldg(reinterpret_cast<const float4*>(res));
      o[0] += u.x, o[1] += u.y, o[2] += u.z, o[3] += u.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (e < n) o[e] += __ldg(res + e);
      }
    }
  }
  if (p.epi_flags & kEpiRelu) {
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = relu_keep_nan(o[e]);
  }
  float* dst = p.out + batch * p.out_batch + static_cast<long long>(i) * p.ldc + j;
  if (p.out_vec && n >= 4) {
    *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e < n) dst[e] = o[e];
    }
  }
}

// Contractions come from a kernel that adds plain f32 products, and keep its results where three bf16 parts cannot
// stand for an operand: infinity times a subnormal below 2^-133 (whose parts are 0: NaN), and rows of operands below
// 2^-110.  Such results are recognised by what they are (NaN, or not zero and below 2^-100) and added again, term by
// term, by the thread that stored them, after everything else.  The others pay the comparison: 0.1 to 0.3 us of a launch
// (64 x 64 x 64 4.65 -> 4.87 us, 1000 x 999 x 301 11.7 -> 11.8, 512 x 512 x 4096 21.5 -> 21.4).
__device__ __forceinline__ bool parts_fail(float v) { return !(fabsf(v) >= 0x1p-100f) & (v != 0.f); }

// CONTRACT: the launch of a contraction.
template <int BN, int AL, int BL, bool VEC, bool CONTRACT>
__global__ void __launch_bounds__(kThreads, 1) f32_mma_kernel(const __grid_constant__ F32MmaParams p) {
  using Cfg = F32Cfg<BN>;
  constexpr bool PAIR = Cfg::kPair;
  constexpr int BR = Cfg::kColsB;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u;
  const uint32_t bar0 = ring + Cfg::kStages * Cfg::kStageBytes;
  uint8_t* tail = smem_raw + (bar0 - raw);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (4 + s); };
  auto tfull_bar = [&](int a) { return bar0 + 8u * (8 + a); };
  auto tempty_bar = [&](int a) { return bar0 + 8u * (10 + a); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail + 96);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 100);   // flag, code, wait limit
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == kLoaderWarps * 32) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      mbar_init(full_bar(s), PAIR ? 2 * kLoaderWarps : kLoaderWarps);   // (pairs: both CTAs' loaders, at the first CTA)
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), kSumWarps);
    }
    abort_flag[0] = 0;
    abort_flag[1] = 0;
    abort_flag[2] = 0;
    fence_mbar_init();
  }
  // this CTA's tile and its run of k-blocks
  // (the CTAs of a tile are one cluster: `split` parts of K, of a pair each where the tile is a pair's)
  const int share = PAIR ? 2 * p.split : p.split;
  const int unit = static_cast<int>(blockIdx.x) / share;
  const int cluster_rank = static_cast<int>(blockIdx.x) - unit * share;
  const int rank = PAIR ? cluster_rank >> 1 : cluster_rank;   // part of K
  const int side = PAIR ? cluster_rank & 1 : 0;               // CTA of the pair
  const uint32_t first_cta = static_cast<uint32_t>(cluster_rank & ~1);
  const int batch = unit / p.tiles_per_batch;
  const int tile = unit - batch * p.tiles_per_batch;
  const int tm = tile / p.tiles_n;
  const int m0 = PAIR ? tm * 256 + side * 128 : tm * 128;
  const int n0 = (tile - tm * p.tiles_n) * BN;
  const int kb_begin = static_cast<int>(static_cast<long long>(p.num_kb) * rank / p.split);
  const int kb_end = static_cast<int>(static_cast<long long>(p.num_kb) * (rank + 1) / p.split);
  const int blocks = kb_end - kb_begin;

  if (warp < kLoaderWarps) {
    // ------------------------------------------------------------ loaders
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLoaderRegs));
    const int tid = threadIdx.x;
    TileLoader<AL, 128, VEC> la;
    TileLoader<BL, BR, VEC> lb;
    la.k_end = lb.k_end = p.k;
    la.ld = p.lda;
    lb.ld = p.ldb;
    const int nb0 = PAIR ? n0 + side * BR : n0;    // first column of B this CTA loads
    la.rows = min(128, p.m - m0);
    lb.rows = min(BR, p.n - nb0);
    if constexpr (AL == kRowsConv) {
      la.origin = p.a;
#pragma unroll
      for (int i = 0; i < la.kGroups; ++i) {
        const int row = m0 + tid / la.kKGroups + la.kKStep * i;
        if (row < p.m) {
          const int img = fast_div(row, p.fd_pq);
          const int px = row - img * p.p * p.q;
          const int oy = fast_div(px, p.fd_q);
          const int y = oy * p.stride_h - p.pad_h, x = (px - oy * p.q) * p.stride_w - p.pad_w;
          la.base[i] = ((img * p.h + y) * p.w + x) * p.c;
          la.yx[i] = static_cast<int>((static_cast<uint32_t>(y) << 16) | (static_cast<uint32_t>(x) & 0xffffu));
        } else {
          la.base[i] = 0;
          la.yx[i] = static_cast<int>(0x80008000u);   // far outside the image
        }
      }
    } else {
      la.origin = p.a + batch * p.a_batch + (AL == kRowsMn ? static_cast<long long>(m0) : static_cast<long long>(m0) * p.lda);
    }
    lb.origin = p.b + batch * p.b_batch + (BL == kRowsMn ? static_cast<long long>(nb0) : static_cast<long long>(nb0) * p.ldb);
    if constexpr (AL != kRowsConv) la.place(tid);
    lb.place(tid);
    grid_dependency_wait();
    grid_launch_dependents();
    // (the first loads are on their way while the barriers and TMEM are set up)
    la.load(kb_begin * kBlockK, p, tid);
    lb.load(kb_begin * kBlockK, p, tid);
    setup_done<0, PAIR>();
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb_begin; kb < kb_end; ++kb) {
      if (!mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag)) {
        if (lane == 0 && abort_flag[1] == 0) abort_flag[1] = 1;
        break;
      }
      const uint32_t sa = ring + static_cast<uint32_t>(stage) * Cfg::kStageBytes;
      la.store(sa, kPartA, tid);
      if (kb + 1 < kb_end) la.load((kb + 1) * kBlockK, p, tid);
      lb.store(sa + 3 * kPartA, Cfg::kPartB, tid);
      if (kb + 1 < kb_end) lb.load((kb + 1) * kBlockK, p, tid);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) {
          mbar_arrive_release_cluster(mapa_rank(full_bar(stage), first_cta));
        } else {
          mbar_arrive(full_bar(stage));
        }
      }
      if (++stage == Cfg::kStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else if (warp >= kIssuerWarp) {
    // ------------------------------------------------------------ MMA issuer
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssuerRegs));
    if (warp == kIssuerWarp) {
      if constexpr (PAIR) {
        tmem_alloc_pair(smem_u32(tmem_slot), 512);
        tmem_relinquish_pair();
      } else {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
      }
      tc_fence_before_sync();
    }
    setup_done<1, PAIR>();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const bool leader = elect_one();
    constexpr bool A_MN = AL == kRowsMn, B_MN = BL == kRowsMn;
    const uint64_t desc_a0 = make_smem_desc_sw128(0, A_MN ? 8192 : 16, 1024);
    const uint64_t desc_b0 = make_smem_desc_sw128(0, B_MN ? 8192 : 16, 1024);
    constexpr uint32_t kStepA = A_MN ? 128u : 2u, kStepB = B_MN ? 128u : 2u;   // 16 terms, in 16-byte units
    constexpr uint32_t id1 = mma_desc(BN, A_MN, B_MN, PAIR ? 256 : 128);
    constexpr uint32_t id2 = mma_desc(PAIR ? BN : 2 * BN, A_MN, B_MN), id3 = mma_desc(3 * 64, A_MN, B_MN);
    int stage = 0;
    uint32_t phase = 0;
    const bool issues = warp == kIssuerWarp && (!PAIR || side == 0);
    for (int i = 0; i < blocks && issues; ++i) {
      const bool first = PAIR ? i == 0 : i % kFlushBlocks == 0;
      const bool last = i == blocks - 1 || (!PAIR && i % kFlushBlocks == kFlushBlocks - 1);
      const int chain = PAIR ? 0 : i / kFlushBlocks;
      const int acc = chain & 1;
      if (!PAIR && first && !mbar_wait_warp(tempty_bar(acc), ((chain >> 1) & 1) ^ 1u, abort_flag)) {
        if (leader && abort_flag[1] == 0) abort_flag[1] = 2;
        break;
      }
      if (!mbar_wait_warp<PAIR>(full_bar(stage), phase, abort_flag)) {
        if (leader && abort_flag[1] == 0) abort_flag[1] = 3;
        break;
      }
      tc_fence_after_sync();
      if (leader) {
        const uint32_t sa = ring + static_cast<uint32_t>(stage) * Cfg::kStageBytes, sb = sa + 3 * kPartA;
        // (a descriptor takes the offset in this CTA's shared memory: in a cluster the address carries the CTA's rank above it)
        const uint64_t ah = desc_a0 | ((sa & 0x3FFFFu) >> 4), bh = desc_b0 | ((sb & 0x3FFFFu) >> 4);
        constexpr uint64_t pa = kPartA >> 4, pb = Cfg::kPartB >> 4;
        const uint32_t d = tmem_base + static_cast<uint32_t>(acc * Cfg::kAccCols);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint64_t a = ah + kStepA * j, b = bh + kStepB * j;
          const uint32_t go = (first && j == 0) ? 0u : 1u;
          if constexpr (PAIR) {
            tc_mma_pair<kMmaF16>(d, a, b, id1, go);                   // h * h
            tc_mma_pair<kMmaF16>(d + BN, a, b + pb, id1, go);         // h * m
            tc_mma_pair<kMmaF16>(d + BN, a, b + 2 * pb, id1, 1u);     // h * l
            tc_mma_pair<kMmaF16>(d + BN, a + pa, b, id1, 1u);         // m * h
            tc_mma_pair<kMmaF16>(d + BN, a + pa, b + pb, id1, 1u);    // m * m
            tc_mma_pair<kMmaF16>(d + BN, a + 2 * pa, b, id1, 1u);     // l * h
          } else if (BN == 128 || (!CONTRACT && p.one_order)) {
            tc_mma<kMmaF16>(d, a, b, id2, go);                        // h * [h | m]
            tc_mma<kMmaF16>(d + BN, a + pa, b, id1, 1u);              // m * h
            tc_mma<kMmaF16>(d + BN, a + pa, b + pb, id1, 1u);         // m * m
            tc_mma<kMmaF16>(d + BN, a, b + 2 * pb, id1, 1u);          // h * l
            tc_mma<kMmaF16>(d + BN, a + 2 * pa, b, id1, 1u);          // l * h
          } else {
            tc_mma<kMmaF16>(d, a, b, id3, go);                        // h * [h | m | l]
            tc_mma<kMmaF16>(d + BN, a + pa, b, id2, 1u);              // m * [h | m]
            tc_mma<kMmaF16>(d + BN, a + 2 * pa, b, id1, 1u);          // l * h
          }
        }
        if constexpr (PAIR) {
          tc_commit_pair(empty_bar(stage), static_cast<uint16_t>(3u << first_cta));   // the stage is free in both CTAs
          if (last) tc_commit_pair(tfull_bar(acc), static_cast<uint16_t>(3u << first_cta));
        } else {
          tc_commit(empty_bar(stage));
          if (last) tc_commit(tfull_bar(acc));
        }
      }
      if (++stage == Cfg::kStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else {
    // ------------------------------------------------------------ sums
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSumRegs));
    setup_done<2, PAIR>();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const int q = warp & 3;                       // TMEM lane quarter this warp may read
    const int half = (warp - kLoaderWarps) >> 2;  // columns [half * BN / 2, ...) of the tile
    constexpr int kCols = BN / 2;
    const uint32_t t_half = tmem_base + static_cast<uint32_t>(half * kCols) + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t row = static_cast<uint32_t>(q * 32 + lane);
    // The ring is free once the last MMAs have completed.  It then takes the sums, 128 rows of BN floats, 16-byte
    // pieces of a row permuted by the row number so that lanes (rows) spread over the banks.
    auto put = [&](int j, float x, float y, float z, float w) {
      const uint32_t piece = static_cast<uint32_t>(half * kCols + j) >> 2;
      st_shared_v4(ring + row * (BN * 4u) + ((piece ^ (row & 15u)) << 4),
                   make_uint4(__float_as_uint(x), __float_as_uint(y), __float_as_uint(z), __float_as_uint(w)));
    };
    if constexpr (PAIR) {
      if (!mbar_wait_warp(tfull_bar(0), 0, abort_flag)) {
        if (lane == 0 && abort_flag[1] == 0) abort_flag[1] = 4;
      } else {
        tc_fence_after_sync();
#pragma unroll 2
        for (int j = 0; j < kCols; j += 16) {
          uint32_t hh[16], small[16];
          tmem_ld_16(t_half + j, hh);
          tmem_ld_16(t_half + BN + j, small);
          tmem_ld_wait();
          float v[16];
          both_parts(hh, small, v);
#pragma unroll
          for (int e = 0; e < 16; e += 4) put(j + e, v[e], v[e + 1], v[e + 2], v[e + 3]);
        }
      }
    } else {
      float sum[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) sum[j] = 0.f;
      bool ok = true;
      for (int kb = 0, chain = 0; kb < blocks; kb += kFlushBlocks, ++chain) {
        const int acc = chain & 1;
        if (!mbar_wait_warp(tfull_bar(acc), (chain >> 1) & 1, abort_flag)) {
          if (lane == 0 && abort_flag[1] == 0) abort_flag[1] = 4;
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t t = t_half + static_cast<uint32_t>(acc * Cfg::kAccCols);
        // (eight columns at a time: the sums, the values in flight and the loop fit 96 registers)
#pragma unroll
        for (int j = 0; j < kCols; j += 8) {
          uint32_t hh[8], small[8];
          tmem_ld_8(t + j, hh);
          tmem_ld_8(t + BN + j, small);
          if constexpr (BN == 64) {
            uint32_t small2[8];
            tmem_ld_8(t + 2 * BN + j, small2);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
              // (a third accumulator that was not used holds anything)
              const bool third = CONTRACT || !p.one_order;
              const float2 t = add2(__uint_as_float(small[e]), __uint_as_float(small[e + 1]), third ? __uint_as_float(small2[e]) : 0.f,
                                    third ? __uint_as_float(small2[e + 1]) : 0.f);
              small[e] = __float_as_uint(t.x), small[e + 1] = __float_as_uint(t.y);
            }
          } else {
            tmem_ld_wait();
          }
          float v[8];
          both_parts(hh, small, v);
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const float2 t = add2(sum[j + e], sum[j + e + 1], v[e], v[e + 1]);
            sum[j + e] = t.x, sum[j + e + 1] = t.y;
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar(acc));
      }
      if (ok) {
#pragma unroll
        for (int j = 0; j < kCols; j += 4) put(j, sum[j], sum[j + 1], sum[j + 2], sum[j + 3]);
      }
    }
  }

  // ---------------------------------------------------------------- parts of the tile -> output
  __syncwarp();
  tc_fence_before_sync();
  const int strips = p.split;   // row strips that the CTAs of a tile (of a pair's side) add up and store
  if (strips > 1) {
    cluster_sync_each_thread();
  } else {
    __syncthreads();
  }
  const bool failed = abort_flag[0] != 0;
  grid_dependency_wait();   // (long past for the loaders; the other warps have not touched global memory yet)
  bool again = false;
  if (!failed && warp < kIssuerWarp) {
    constexpr int kPieces = BN / 4;                 // 16-byte pieces per row
    const int strip = (128 + strips - 1) / strips;
    const int strip_begin = strips > 1 ? rank * strip : 0;
    const int strip_end = min(128, strip_begin + strip);
    // (whole warps: the row maxima are shuffled)
    for (int t = threadIdx.x; t < (strip * kPieces + 31) / 32 * 32; t += kIssuerWarp * 32) {
      const int row = min(strip_begin + t / kPieces, 127);
      const bool mine = strip_begin + t / kPieces < strip_end;
      const int piece = t % kPieces;
      const uint32_t at = ring + static_cast<uint32_t>(row) * (BN * 4u) + ((static_cast<uint32_t>(piece) ^ (static_cast<uint32_t>(row) & 15u)) << 4);
      float o[4] = {0.f, 0.f, 0.f, 0.f};
      if (strips > 1) {
        for (int r = 0; r < strips; ++r) {
          const float4 u = ld_cluster_v4(mapa_rank(at, static_cast<uint32_t>(PAIR ? 2 * r + side : r)));
          o[0] += u.x, o[1] += u.y, o[2] += u.z, o[3] += u.w;
        }
      } else {
        const uint4 u = ld_shared_v4(at);
        o[0] = __uint_as_float(u.x), o[1] = __uint_as_float(u.y), o[2] = __uint_as_float(u.z), o[3] = __uint_as_float(u.w);
      }
      const int i = m0 + row, j = n0 + piece * 4;
      const int valid = mine && i < p.m ? p.n - j : 0;   // columns of this piece that exist
      if (p.epi_flags & kEpiRowMax) {
        float best = -INFINITY;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (e < valid) best = fmaxf(best, o[e]);
        }
        // (a row is kPieces consecutive threads: half a warp, a warp or two)
#pragma unroll
        for (int d = (kPieces < 32 ? kPieces : 32) / 2; d > 0; d >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, d));
        if (piece % 32 == 0 && mine && i < p.m) atomic_max_f32(p.rowmax + static_cast<long long>(batch) * p.m + i, best);
        if (p.out == nullptr) continue;
      }
      if constexpr (CONTRACT) {
#pragma unroll
        for (int e = 0; e < 4; ++e) again |= parts_fail(o[e]);
      }
      if (valid > 0) finish(p, batch, i, j, o, valid);
    }
  }
  if (failed) {
    if (threadIdx.x == 0) atomicCAS(p.status, 0, abort_flag[1] != 0 ? abort_flag[1] : 9);
    // give MMAs still in flight a bounded time before TMEM and shared memory go away
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 2000000ull) __nanosleep(2000);
  }
  if (PAIR || strips > 1) {
    cluster_sync_each_thread();   // no CTA of the cluster leaves while another may still read its part (or send to it)
  } else {
    __syncthreads();
  }
  if (warp == kIssuerWarp) {
    __syncwarp();
    tc_fence_after_sync();
    if constexpr (PAIR) {
      tmem_dealloc_pair(*tmem_slot, 512);
    } else {
      tmem_dealloc(*tmem_slot, 512);
    }
  }
  if (CONTRACT && __builtin_expect(again, 0)) {
    constexpr int kPieces = BN / 4;
    const int strip = (128 + strips - 1) / strips;
    const int strip_begin = strips > 1 ? rank * strip : 0;
    const int strip_end = min(128, strip_begin + strip);
    const long long step_a = AL == kRowsMn ? p.lda : 1, step_b = BL == kRowsMn ? p.ldb : 1, step_j = BL == kRowsMn ? 1 : p.ldb;
#pragma unroll 1
    for (int t = threadIdx.x; t < strip * kPieces; t += kIssuerWarp * 32) {
      const int i = m0 + strip_begin + t / kPieces, j = n0 + t % kPieces * 4;
      if (strip_begin + t / kPieces >= strip_end || i >= p.m) break;   // (rows only grow)
      const int cols = min(4, p.n - j);
      float* dst = p.out + batch * p.out_batch + static_cast<long long>(i) * p.ldc + j;
      bool any = false;
#pragma unroll
      for (int e = 0; e < 4; ++e) any |= e < cols && parts_fail(dst[e]);
      if (!any) continue;
      const float* a = p.a + batch * p.a_batch + (AL == kRowsMn ? static_cast<long long>(i) : i * p.lda);
      const float* b = p.b + batch * p.b_batch + j * step_j;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      bool number = true;   // (NaN stays)
#pragma unroll 1
      for (int k = 0; k < p.k && number; ++k) {
        const float x = __ldg(a);
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] = __fadd_rn(sum[e], __fmul_rn(x, __ldg(b + (e < cols ? e : 0) * step_j)));
        number = sum[0] == sum[0] || sum[1] == sum[1] || sum[2] == sum[2] || sum[3] == sum[3];
        a += step_a, b += step_b;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (e < cols && parts_fail(dst[e])) dst[e] = sum[e];
      }
    }
  }
}

template <class In>
__global__ void __launch_bounds__(256) filter_to_f32_kernel(const In* in, float* out, long long n) {
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (i < n) out[i] = static_cast<float>(in[i]);
}

// Zero until a launch gives up waiting.  Handed out in turn: two plans 1024 apart share one, and either may then report it.
constexpr unsigned kStatusWords = 1024;
__device__ int g_status_words[kStatusWords];

using KernelPtr = void (*)(const F32MmaParams);

// The shared-memory limit is an attribute per device.
template <int BN, int AL, int BL, bool VEC, bool CONTRACT = false>
KernelPtr instance(int dev) {
  static std::atomic<uint64_t> done{0};
  const uint64_t bit = 1ull << (dev & 63);
  if (dev >= 64 || (done.load(std::memory_order_acquire) & bit) == 0) {
    if (cudaFuncSetAttribute(f32_mma_kernel<BN, AL, BL, VEC, CONTRACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, F32Cfg<BN>::kSmem) == cudaSuccess) {
      done.fetch_or(bit, std::memory_order_release);
    }
  }
  return f32_mma_kernel<BN, AL, BL, VEC, CONTRACT>;
}

// Clusters of `split` CTAs that the device holds at once (a GPC holds whole clusters only).
int resident_clusters(int dev, int split) {
  static std::mutex mutex;
  static int known[64][9];   // per device and split, 0 = not asked yet
  if (dev < 0 || dev >= 64) return 1;
  std::lock_guard<std::mutex> lock(mutex);
  if (known[dev][split] == 0) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(split);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = F32Cfg<64>::kSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = split;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, instance<64, kRowsK, kRowsMn, true>(dev), &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = 1;
    }
    known[dev][split] = n;
  }
  return known[dev][split];
}

constexpr long long kMaxTiles = 0x0fffffff;   // (times eight CTAs: the grid's limit)

struct Choice {
  int bn = 0, split = 0;
  double cycles = 0;
};

// Tile width and K split: the pair with the smallest estimated time, in cycles per wave of resident tiles.  Measured
// (B200, 1.9 GHz): a k-block takes 1700 cycles with 64-wide and 2400 with 128-wide tiles (the loaders) and 3750 on a CTA
// pair for four times the 128-wide tile's work on two SMs (the rate the tensor pipe sustains); rows that are not 16-byte aligned cost a
// third more loads.  Everything around the loop: 8800, 11500 and 18000 cycles, and 1500 + 150 per CTA of a K split.
// (Clusters are counted with the 64-wide kernel: every kernel here leaves room for one CTA per SM.)
Choice choose_tiles(int m, int n, int num_kb, int batch, bool vec, int bn_override, int split_override, bool pairs, int dev, int sms) {
  Choice best;
  for (int bn = 64; bn <= (pairs ? 256 : 128); bn *= 2) {
    if (bn_override != 0 && bn != bn_override) continue;
    const int rows = bn == 256 ? 256 : 128;
    const long long tiles = (m + rows - 1ll) / rows * ((n + bn - 1ll) / bn) * batch;
    if (tiles > kMaxTiles) continue;
    for (int split = 1; split <= (bn == 256 ? 4 : 8); ++split) {
      if (split_override != 0 ? split != split_override : split > num_kb) continue;
      const int share = bn == 256 ? 2 * split : split;
      const long long room = share == 1 ? sms : resident_clusters(dev, share);
      const long long waves = (tiles + room - 1) / room;
      const double block = (bn == 256 ? 3750.0 : (bn == 128 ? 2400.0 : 1700.0)) * (vec ? 1.0 : 1.33);
      const double around = (bn == 256 ? 18000.0 : (bn == 128 ? 11500.0 : 8800.0)) + (split > 1 ? 1500.0 + 150.0 * split : 0.0);
      const double cycles = static_cast<double>(waves) * ((num_kb + split - 1) / split * block + around);
      if (best.bn == 0 || cycles < best.cycles) {
        best.bn = bn;
        best.split = split;
        best.cycles = cycles;
      }
    }
  }
  return best;
}

// A has its columns contiguous in contractions only.
template <int BN, bool VEC>
KernelPtr choose(int al, int bl, int dev) {
  if (al == kRowsConv) return instance<BN, kRowsConv, kRowsMn, VEC>(dev);
  return bl == kRowsK ? instance<BN, kRowsK, kRowsK, VEC>(dev) : instance<BN, kRowsK, kRowsMn, VEC>(dev);
}

template <int BN, bool VEC>
KernelPtr choose_contraction(int al, int bl, int dev) {
  if (al == kRowsK) return bl == kRowsK ? instance<BN, kRowsK, kRowsK, VEC, true>(dev) : instance<BN, kRowsK, kRowsMn, VEC, true>(dev);
  return bl == kRowsK ? instance<BN, kRowsMn, kRowsK, VEC, true>(dev) : instance<BN, kRowsMn, kRowsMn, VEC, true>(dev);
}

template <bool VEC>
KernelPtr choose(int bn, bool contraction, int al, int bl, int dev) {
  if (contraction) return bn == 128 ? choose_contraction<128, VEC>(al, bl, dev) : choose_contraction<64, VEC>(al, bl, dev);
  if (bn == 256) return choose<256, VEC>(al, bl, dev);
  return bn == 128 ? choose<128, VEC>(al, bl, dev) : choose<64, VEC>(al, bl, dev);
}

}  // namespace

bool f32_mma_takes_conv(const ConvGeom& g) {
  // 16-byte groups of channels; positions and element offsets inside the kernel's 16- and 32-bit fields
  const long long in_elems = static_cast<long long>(g.n) * g.h * g.w * g.c;
  const long long reach_h = static_cast<long long>(g.p) * g.stride_h + static_cast<long long>(g.r) * g.dil_h + g.pad_h;
  const long long reach_w = static_cast<long long>(g.q) * g.stride_w + static_cast<long long>(g.s) * g.dil_w + g.pad_w;
  return g.c % 4 == 0 && in_elems < (1ll << 30) && reach_h < 16384 && reach_w < 16384 && g.h < 16384 && g.w < 16384 &&
         static_cast<long long>(g.n) * g.p * g.q < (1ll << 30) && static_cast<long long>(g.r) * g.s * g.c < (1ll << 30);
}

F32MmaTiles f32_mma_tiles(const F32MmaShape& s) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // A sum's order follows from the tile kind and the split.  64- and 128-wide tiles can share one, pairs and parts cannot.
  const Choice c = choose_tiles(s.m, s.n, (s.k + kBlockK - 1) / kBlockK, s.batch, s.aligned_in, s.tile_n, s.whole_k ? 1 : 0,
                                !s.short_chains && !s.whole_k, dev, sms);
  F32MmaTiles t;
  t.bn = c.bn, t.split = c.split, t.us = c.cycles / 1900.0, t.one_order = s.whole_k;
  return t;
}

// Both estimates in microseconds.  The pre-pass route (B200, graph replays): 9 us of launches and set-up, 12 bytes per
// element at 5.2 TB/s, then 0.58 (128-wide tiles) or 0.38 us (64-wide) per 32 terms of each wave of a persistent grid
// that stores one tile while it computes the next, a third more where rows are not 16-byte aligned.  It wins where a
// launch has several waves of tiles and each of them few terms, because this file's kernel stores a tile before its SM
// starts the next: 4096 x 4096 x 256 46 against 71 us, 100352 x 64 x 576 72 against 93 us; it loses on few tiles, long
// K, odd rows and strided 1x1 convolutions: 64 x 4096 x 4096 94 against 29 us, 1999 x 2001 x 1001 70 against 55 us.
bool f32_mma_faster(const F32MmaShape& s, F32MmaTiles* tiles) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  *tiles = f32_mma_tiles(s);
  if (tiles->bn == 0) return false;
  if (s.whole_k) return true;   // (the pre-pass adds in another order)
  const Choice any = choose_tiles(s.m, s.n, (s.k + kBlockK - 1) / kBlockK, s.batch, s.aligned_in, 0, 0, true, dev, sms);
  const double here = any.cycles / 1900.0 * (s.conv ? (any.bn == 256 ? 1.05 : 1.2) : 1.0);   // (gathering pixels costs more)
  const double tiles_m = (s.m + 127) / 128;
  auto prepass = [&](int bn, double block_us) {
    const double waves = std::max(1.0, tiles_m * ((s.n + bn - 1) / bn) * s.batch / sms);
    return 9.0 + static_cast<double>(s.elems) * 12.0 / 5.2e6 + waves * s.k / 32.0 * block_us * (s.aligned_out ? 1.0 : 1.33);
  };
  const double there = std::min(prepass(128, 0.58), prepass(64, 0.38));
  return here <= 0.95 * there;
}

int* f32_mma_status_word() {
  static std::atomic<unsigned> next{0};
  void* words = nullptr;
  if (cudaGetSymbolAddress(&words, g_status_words) != cudaSuccess) return nullptr;
  return static_cast<int*>(words) + next.fetch_add(1, std::memory_order_relaxed) % kStatusWords;
}

int f32_mma_launch(const F32MmaLaunch& L, cudaStream_t stream, std::string* err) {
  F32MmaParams p{};
  p.m = L.m, p.n = L.n, p.k = L.k;
  p.a = L.a, p.b = L.b;
  p.lda = L.lda, p.ldb = L.ldb, p.a_batch = L.a_batch, p.b_batch = L.b_batch;
  p.out = L.out, p.ldc = L.ldc, p.out_batch = L.out_batch;
  p.epi_flags = L.epi_flags;
  p.bias = L.bias, p.residual = L.residual, p.ldr = L.ldr, p.res_batch = L.res_batch;
  p.rowmax = L.rowmax;
  p.status = L.status;
  p.num_kb = (L.k + kBlockK - 1) / kBlockK;
  auto aligned = [](const void* ptr, long long ld, long long batch) {
    return reinterpret_cast<uintptr_t>(ptr) % 16 == 0 && ld % 4 == 0 && batch % 4 == 0;
  };
  const bool vec = aligned(L.a, L.conv ? 0 : L.lda, L.a_batch) && aligned(L.b, L.ldb, L.b_batch);
  p.out_vec = aligned(L.out, L.ldc, L.out_batch) && (!L.residual || aligned(L.residual, L.ldr, L.res_batch));
  int al = L.a_mn ? kRowsMn : kRowsK;
  if (L.conv) {
    const ConvGeom& g = *L.conv;
    al = kRowsConv;
    p.c = g.c, p.h = g.h, p.w = g.w, p.p = g.p, p.q = g.q, p.s = g.s;
    p.stride_h = g.stride_h, p.stride_w = g.stride_w, p.pad_h = g.pad_h, p.pad_w = g.pad_w, p.dil_h = g.dil_h, p.dil_w = g.dil_w;
    p.fd_c = make_fastdiv(g.c);
    p.fd_s = make_fastdiv(g.s);
    p.fd_pq = make_fastdiv(g.p * g.q);
    p.fd_q = make_fastdiv(g.q);
  }
  int dev = 0;
  cudaGetDevice(&dev);
  const int best_bn = L.tiles.bn;
  p.split = L.tiles.split;
  p.one_order = L.tiles.one_order;
  p.tiles_n = (L.n + best_bn - 1) / best_bn;
  const int tile_rows = best_bn == 256 ? 256 : 128, share = best_bn == 256 ? 2 * p.split : p.split;
  const long long per_batch = static_cast<long long>((L.m + tile_rows - 1) / tile_rows) * p.tiles_n;
  const long long units = per_batch * L.batch;
  if (units > kMaxTiles) {
    *err = "too many tiles";
    return PMLB_ERR_UNSUPPORTED;
  }
  p.tiles_per_batch = static_cast<int>(per_batch);
  const long long grid = units * share;
  const int bl = L.b_mn ? kRowsMn : kRowsK;
  if (L.contraction ? best_bn == 256 : L.a_mn) {
    *err = "no such tiles";
    return PMLB_ERR_UNSUPPORTED;
  }
  const KernelPtr kernel = vec ? choose<true>(best_bn, L.contraction, al, bl, dev) : choose<false>(best_bn, L.contraction, al, bl, dev);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = best_bn == 256 ? F32Cfg<256>::kSmem : (best_bn == 128 ? F32Cfg<128>::kSmem : F32Cfg<64>::kSmem);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0] = dependent_launch_attribute();
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = share;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = share > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
  if (e != cudaSuccess) {
    *err = std::string("fp32 tensor-core launch: ") + cudaGetErrorString(e);
    return PMLB_ERR_CUDA;
  }
  return 0;
}

cudaError_t launch_filter_to_f32(const void* in, int in_dtype, float* out, long long elems, cudaStream_t stream) {
  const unsigned grid = static_cast<unsigned>((elems + 255) / 256);
  if (in_dtype == PMLB_F32) return cudaMemcpyAsync(out, in, elems * sizeof(float), cudaMemcpyDeviceToDevice, stream);
  if (in_dtype == PMLB_BF16) {
    filter_to_f32_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(in), out, elems);
  } else {
    filter_to_f32_kernel<<<grid, 256, 0, stream>>>(static_cast<const __half*>(in), out, elems);
  }
  return cudaGetLastError();
}

}  // namespace pmlb
