// FP64 density assembly and grid matrix elements on the tensor cores.
//
// GB300 issues 2 FP64 FMAs per clock and SM, and the pair kernels of
// lcp_kernels_pair.cu keep that pipe 95 % busy: 16.9 ms (density) and 19.9 ms
// (matrix elements) on the 64-atom 96^3 cell, where the kernels below take 1.6
// ms each.  The tensor cores do 4,096 FP16 multiply-adds per clock and SM
// with FP32 accumulation, which is exact for integers below 2^24.  So each FP64
// operand is put on a fixed-point grid of 56 bits,
//
//   x = t 2^-55 2^E,  |x| < 2^E,  t = sum_i d_i 256^(7-i),  |d_i| <= 128,
//
// whose seven base-256 digits are exact FP16 values (the splitting of Ozaki, Ogita,
// Oishi and Rump, Numer. Algorithms 59, 2012, on fixed grids), and a contraction of two
// operands is the 28 digit products d_i d_j' with i + j <= 8, each group of
// equal weight (i + j = d + 1) in its own FP32 accumulator a_d.  Over 64 terms
// |a_d| <= d 2^20 < 2^24, so every sum is exact in the matrix elements; in the
// density, over segments of 256 rows, a_1 to a_4 are, for any values (kDSeg).
// The dropped groups are below 2^-62 of the scales' product.  What is
// rounded: each operand once to 2^-56 of its row's (column's, point's) largest
// value, the assembled sum once to 2^-55 of the scales' product, and the FP64
// additions that follow.  An FP64 FMA chain rounds every partial sum to 2^-53
// of itself.  Against 113-bit sums over the same tables, on cells of 2 to 6
// atoms and 4 to 18 orbitals, the errors over the result's norm are 1.3e-16 to
// 2.1e-16 in H (pair kernels 2.0e-16 to 3.7e-16) and 1.3e-16 to 1.5e-16 in rho
// (1.4e-16 to 2.8e-16).
//
// What a value on a grid loses is what lies below 2^-56 of the grid's scale, where
// an FP64 product keeps 53 bits of its own whatever its neighbours hold:
//   phi   elements: the row's largest in the brick; density, force: the point's
//         largest row;
//   V     2^-62 of the brick's largest where an orbital is (f64_vprep_kernel lists
//         the bricks where it spans too much for that);
//   D     density: its column's largest over all pairs of the cell
//         (f64_btop_kernel lists the bricks that this would cost more than 12 bits);
//         force: its row's.
// The listed ("odd") bricks are summed directly in FP64, and so are those with
// values that are not finite.  Elements of H far below the largest, where two
// orbitals' tails meet, carry fewer digits of their own than the pair kernels'
// (99th percentile of the elements' relative errors 3e-14 to 2e-13, against 1e-14).
//
// The split is integer work: the mantissa shifted to the scale's grid, rounded,
// biased by 128 in every byte, and each byte turned into FP16 by placing it
// under the exponent of 1024 and subtracting 1152 (two digits per instruction).
// FP16 rather than BF16 because a byte fits FP16's eleven-bit integers without
// a sign trick; the tensor rate is the same.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "lcp_bounds.cuh"
#include "lcp_device.h"
#include "lcp_tc.cuh"

namespace lcp {

namespace {

constexpr int kDig = 7;       // digits per operand
constexpr int kWin = 32;      // columns of a window (7 * 32 TMEM columns per buffer)
constexpr int kBadExp = 4095; // scale of a column or brick that holds Inf or NaN
constexpr uint32_t kBufCols = 256;

// |x| as a 53-bit integer m and a biased exponent e: |x| = m 2^(e - 1075) (subnormals too).
__device__ __forceinline__ uint64_t mantissa(double x, int& e) {
  const uint32_t hi = (uint32_t)__double2hiint(x);
  const int f = (int)((hi >> 20) & 0x7ffu);
  e = max(f, 1);
  return ((uint64_t)((hi & 0xfffffu) | (f > 0 ? 0x100000u : 0u)) << 32) | (uint32_t)__double2loint(x);
}

// t + sum_k 128 * 256^k of x on the grid of exponent E (biased; |x| < 2^(E - 1023)):
// rounded to nearest, ties away from zero.
__device__ __forceinline__ uint64_t fx_biased(double x, int E) {
  int e;
  const uint64_t m = mantissa(x, e) << 4;
  const uint64_t t = ((m >> min((uint32_t)(E - e), 63u)) + 1) >> 1;
  const uint64_t s = (uint64_t)(int64_t)(__double2hiint(x) >> 31);
  return (t ^ s) - s + kF64Bias;
}

// FP16 pairs of the seven digits of two values (d[0]: the leading digits).
__device__ __forceinline__ uint32_t half_digits(uint32_t biased) {  // 0x64bb64bb: 1024 + byte
  const uint32_t k = 0x64806480u;                                   // 1152
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&biased), *reinterpret_cast<const __half2*>(&k));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void digit_pairs(uint64_t x, uint64_t y, uint32_t* d) {
  const uint32_t xl = (uint32_t)x, xh = (uint32_t)(x >> 32), yl = (uint32_t)y, yh = (uint32_t)(y >> 32);
  const uint32_t k = 0x64646464u;
  const uint32_t z0 = __byte_perm(xl, yl, 0x5140);  // bytes 0 and 1 of x and y interleaved
  const uint32_t z1 = __byte_perm(xl, yl, 0x7362);  // 2 and 3
  const uint32_t z2 = __byte_perm(xh, yh, 0x5140);  // 4 and 5
  // the leading digit keeps the carry byte: 128 + 128 = 256 is possible
  d[0] = half_digits(__byte_perm(xh, yh, 0x7632) | 0x64006400u);
  d[1] = half_digits(__byte_perm(z2, k, 0x4342));
  d[2] = half_digits(__byte_perm(z2, k, 0x4140));
  d[3] = half_digits(__byte_perm(z1, k, 0x4342));
  d[4] = half_digits(__byte_perm(z1, k, 0x4140));
  d[5] = half_digits(__byte_perm(z0, k, 0x4342));
  d[6] = half_digits(__byte_perm(z0, k, 0x4140));
}

// The digits of eight values into seven 16-byte pieces, `step` bytes apart.
__device__ __forceinline__ void store_digits(uint8_t* dst, uint32_t step, const uint64_t* t) {
  uint32_t d[4][kDig];
#pragma unroll
  for (int q = 0; q < 4; ++q) digit_pairs(t[2 * q], t[2 * q + 1], d[q]);
#pragma unroll
  for (int i = 0; i < kDig; ++i)
    *reinterpret_cast<uint4*>(dst + i * step) = make_uint4(d[0][i], d[1][i], d[2][i], d[3][i]);
}

// Biased exponent bound of the magnitude whose high word is h: |x| < 2^(E - 1023).
__device__ __forceinline__ int exp_bound(uint32_t h) {
  const int e = (int)(h >> 20);
  return e == 0x7ff ? kBadExp : e + 1;
}

constexpr uint32_t idesc_f16_f32(int M, int N, int a_mn, int b_mn) {  // FP16 operands, FP32 accumulator
  return (1u << 4) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}

// The seven accumulators of four columns from `col` on, lanes of `quarter`.
__device__ __forceinline__ void tmem_ld4_nowait(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void load_acc(uint32_t tmem, uint32_t quarter, uint32_t col, uint32_t (&y)[kDig][4]) {
#pragma unroll
  for (int i = 0; i < kDig; ++i) tmem_ld4_nowait(tc::tmem_addr(tmem, quarter * 32, col + i * kWin), y[i]);
  tc::tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < kDig; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) asm volatile("" : "+r"(y[i][j]));  // no use before the wait
}

// Eight consecutive slots of row `row` of a 32-row table chunk staged in
// shared memory; piece: the 2 KB of that slot group ([4 pairs][32 rows][2]).
__device__ __forceinline__ void read_piece(const uint8_t* piece, int row, uint64_t* t) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(piece + i * 512 + row * 16);
    t[2 * i] = w.x;
    t[2 * i + 1] = w.y;
  }
}

// Table pieces of kRawBytes on their way into a ring of shared-memory slots
// (bulk copies), issued by the MMA warp: once the digits of a slot's piece have
// arrived as operands, it holds the next one.  (A barrier on which the split
// warps gave a slot back after loading from it let a refilled slot be read: an
// arrival does not wait for loads whose values are only used after it.  Giving
// it back after the digits had the issuing split warp wait for the others.)
constexpr uint32_t kRawBytes = 16384;
template <int SLOTS>
struct RawRing {
  uint8_t* buf;
  uint64_t* full;
  uint32_t slot = 0, issued = 0;
  __device__ __forceinline__ void issue(const uint8_t* src) {  // the whole warp
    if (tc::elect_one()) {
      tc::mbar_arrive_expect_tx(&full[slot], kRawBytes);
      tc::bulk_g2s(buf + slot * kRawBytes, src, kRawBytes, &full[slot]);
    }
    __syncwarp();
    ++issued;
    if (++slot == SLOTS) slot = 0;
  }
  // the last copies have landed (before the shared memory goes away)
  __device__ __forceinline__ void drain() {
    for (uint32_t i = 0; i < SLOTS && i < issued; ++i) {
      const uint32_t n = issued - 1 - i;
      tc::mbar_wait(&full[n % SLOTS], (n / SLOTS) & 1, 1u << 22);
    }
  }
};

__device__ __forceinline__ F64Row load_meta(const F64Row* p) {
  const uint2 w = __ldg(reinterpret_cast<const uint2*>(p));
  return F64Row{w.x, w.y};
}
__device__ __forceinline__ int row_no(uint32_t info) { return (int)(info & 63u); }
__device__ __forceinline__ int row_exp(uint32_t info) { return (int)(info >> 6); }  // matrix elements
__device__ __forceinline__ int row_col(uint32_t info) { return (int)(info >> 6); }  // density: column of D

__device__ __forceinline__ F64Brick load_brick(const F64Brick* p) {
  const uint4 w = __ldg(reinterpret_cast<const uint4*>(p));
  return F64Brick{w.x, w.y, w.z, w.w};
}

// A CTA's bricks with rows, in order; AHEAD: each one is loaded a brick ahead
// (four registers).
template <bool AHEAD>
struct BrickIterT {
  int k, nb;
  F64Brick b, n;
  __device__ __forceinline__ int R() const { return (int)(b.size & 0xffffu); }
  __device__ __forceinline__ int m() const { return (int)(b.size >> 16); }
  __device__ __forceinline__ bool valid() const { return k < nb; }
  __device__ __forceinline__ void settle(const F64Bricks& B) {
    for (; k < nb; k += gridDim.x) {
      b = AHEAD ? n : load_brick(B.bricks + k);
      if (AHEAD && k + (int)gridDim.x < nb) n = load_brick(B.bricks + k + gridDim.x);
      if (R() > 0) return;
    }
  }
  __device__ __forceinline__ void start(const F64Bricks& B) {
    k = blockIdx.x;
    nb = (int)B.nbricks;
    if (AHEAD && k < nb) n = load_brick(B.bricks + k);
    settle(B);
  }
  __device__ __forceinline__ void next(const F64Bricks& B) {
    k += gridDim.x;
    settle(B);
  }
};
using BrickIter = BrickIterT<true>;

// The next of the units that warps take one by one.
__device__ __forceinline__ int64_t claim_unit(unsigned long long* next, int lane) {
  unsigned long long u = 0;
  if (lane == 0) u = atomicAdd(next, 1ull);
  return (int64_t)__shfl_sync(0xffffffffu, u, 0);
}

int device_sms() {
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace

// ==========================================================================
// Scales and tables of a tiling.
// ==========================================================================
namespace {

// Rows and scales, one warp per image (lane = orbital): each row's exponent
// bound over the brick's points, or each point's over all rows, and behind those
// the bricks where a phi is not finite; with cover, the slots that the images hold,
// none of such a brick.
__global__ void __launch_bounds__(256) f64_scales_kernel(F64Bricks b, F64Source f, const int32_t* __restrict__ row0,
                                                         F64Row* __restrict__ rows, int32_t* __restrict__ ptexp,
                                                         uint64_t* __restrict__ cover) {
  __shared__ uint32_t s_cover[2];
  __shared__ int s_bad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int64_t hb = blockIdx.x; hb < b.nbricks; hb += gridDim.x) {
    const int64_t i0 = f.img_off[hb];
    const int m = (int)(f.img_off[hb + 1] - i0);
    if (cover) {
      __syncthreads();
      if (threadIdx.x == 0) s_cover[0] = s_cover[1] = 0, s_bad = 0;
      __syncthreads();
    }
    for (int i = warp; i < m; i += nw) {
      const int a = f.img_atom[i0 + i], no = f.numorbs[a];
      const double* src = f.phi + f.phi_off[a] + lane;
      const int32_t* sl = f.slot + (i0 + i) * b.P;
      uint32_t mx = 0;
#pragma unroll 8
      for (int p = 0; p < b.P; ++p) {
        const int k = sl[p];
        const uint32_t h = (k >= 0 && lane < no) ? (uint32_t)__double2hiint(__ldg(src + (int64_t)k * no)) & 0x7fffffffu : 0u;
        mx = max(mx, h);
        if (k >= 0 && ptexp) {
          const uint32_t pm = __reduce_max_sync(0xffffffffu, h);
          if (lane == 0) {
            atomicMax(ptexp + hb * b.P + p, exp_bound(pm));
            if (exp_bound(pm) >= kBadExp) ptexp[b.nbricks * b.P + hb] = 1;  // bad
          }
        }
      }
      if (lane < no)
        rows[(int64_t)b.bricks[hb].row + row0[i0 + i] + lane] =
            F64Row{(uint32_t)no | ((ptexp ? (uint32_t)(a * 32 + lane) : (uint32_t)exp_bound(mx)) << 6),
                   ((uint32_t)i << 8) | (uint32_t)lane};
      if (cover) {
        if (lane < no && exp_bound(mx) >= kBadExp) s_bad = 1;
        for (int h = 0; h < 2; ++h) {
          const uint32_t in = __ballot_sync(0xffffffffu, sl[h * 32 + lane] >= 0);
          if (lane == 0) atomicOr(&s_cover[h], in);
        }
      }
    }
    if (cover) {
      __syncthreads();
      if (threadIdx.x == 0) cover[hb] = s_bad ? 0 : ((uint64_t)s_cover[1] << 32) | s_cover[0];
    }
  }
}

// phi of every row at every slot on its scale's grid: lane = row of a chunk,
// two slots per store (the phi rows of a point are contiguous over its lanes).
__global__ void __launch_bounds__(256) f64_table_kernel(F64Bricks b, F64Source f, uint64_t* __restrict__ table) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int64_t hb = blockIdx.x; hb < b.nbricks; hb += gridDim.x) {
    const F64Brick br = load_brick(b.bricks + hb);
    const int R = (int)(br.size & 0xffffu);
    const int64_t i0 = f.img_off[hb];
    for (int c = 0; c * 32 < R; ++c) {
      const int r = c * 32 + lane;
      F64Row m{};
      const double* src = f.phi;
      const int32_t* sl = f.slot;
      if (r < R) {
        m = load_meta(b.rows + br.row + r);
        const int64_t im = i0 + (m.img_orb >> 8);
        src = f.phi + f.phi_off[f.img_atom[im]] + (m.img_orb & 255u);
        sl = f.slot + im * b.P;
      }
      const int no = row_no(m.info), e = row_exp(m.info);
      for (int w = warp; w < b.P / 2; w += nw) {
        const int p = 2 * w;
        uint64_t t[2] = {kF64Bias, kF64Bias};
        if (r < R) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int k = __ldg(sl + p + q);
            if (k >= 0) t[q] = fx_biased(__ldg(src + (int64_t)k * no), b.P == 128 ? __ldg(b.ptexp + hb * b.P + p + q) : e);
          }
        }
        reinterpret_cast<ulonglong2*>(table + (int64_t)(br.chunk + c) * 32 * b.P)[w * 32 + lane] = make_ulonglong2(t[0], t[1]);
      }
    }
  }
}

}  // namespace

// ==========================================================================
// Matrix elements.  Per brick of 64 points, over its R packed rows,
//
//   G[r][c] = sum_p phi_r(p) V(p) phi_c(p),   r <= c  (G is symmetric),
//
// as tiles of 128 rows x windows of 32 columns: A holds the V-weighted rows
// (split once per tile), B a window's plain columns, both K-major.  64 points
// because the seven digit planes of A take 112 KB of shared memory at that K;
// packed rows because 13 orbitals in 16-row blocks would waste a third of the
// products, and 4- and 18-orbital atoms more.
//
// A pair's bricks (over a thousand for a self pair) are summed by FP64 atomic
// adds into one of eight copies of H, the brick's number mod 8, which
// f64_finish_kernel adds up: with one copy the matrix was 2.5 to 4 times
// further from the exact one than the pair kernels' (8e-16 against 3e-16 of
// its norm, one rounding per brick instead of one per 512 points).  Exact sums
// in two 64-bit integers (5e-17) cost a second atomic per element, 14 clocks
// per warp and SM each, and the adds are what the epilogue waits for most.
//
// A step is one window.  Since only r <= c counts, window w of a tile needs
// the tile's row blocks up to its own: the first four steps split their chunk
// twice, as the window's B and, V-weighted, as row block w of A, and no step
// waits for a whole A tile.  (Rows of A left from an earlier tile only feed
// results with r > c, which nobody reads.)
//
// Roles (640 threads, one CTA per SM, persistent over bricks; warp w runs on
// scheduler w % 4, and the epilogue warps of one quarter of the TMEM lanes
// have to sit on one scheduler.  The first quarter holds the lowest rows,
// which count in every window, the last one the fewest, so the schedulers get
// 4, 3, 2 and 2 epilogue warps and the split warps fill the others):
//   epilogue: a warp takes its share of a window's eight column groups: the
//             seven accumulators as integers, assembled in 64 bits, one FP64
//             atomic add into the pair's accumulated block (lanes are
//             consecutive orbitals of one image: consecutive addresses);
//   MMA:      4 K steps x 7 MMAs, digit i of A against digits 1 .. 8-i of B
//             stacked along N (N = 32 (8 - i)), so that every product lands
//             in the accumulator of its weight;
//   split:    8 warps, one k group (8 points) each, lane = row of the chunk.
// Every wait is bounded; a timeout sets *status and stops all roles.
// ==========================================================================
namespace {

constexpr int kHP = 64;
constexpr int kHEpi = 11, kHConv = 8;
constexpr int kHThreads = 32 * (kHEpi + 1 + kHConv);
constexpr uint32_t kHADigit = 128 * kHP * 2;           // 16 KB: [k group][128 rows][16 B]
constexpr uint32_t kHBLbo = kDig * kWin * 16;          // 3,584 B per k group: [digit][32 columns][16 B]
constexpr uint32_t kHBStage = (kHP / 8) * kHBLbo;      // 28 KB
constexpr int kHRaw = 3;                               // table chunks in shared memory
constexpr size_t kHSmemBytes = kDig * (size_t)kHADigit + 2 * (size_t)kHBStage + kHRaw * (size_t)kRawBytes;  // 216 KB
static_assert(kRawBytes == 32 * kHP * 8, "a raw slot is a chunk");

// sum a_d 256^(7-d) / 256 for |a_d| <= d 2^20 (64 products of each kind, |digit| <= 128), rounded;
// below 2^61.  a_1 .. a_4 lie within 2^22, where adding 1.5 2^23 leaves the
// integer in the low bits; a_7 only counts in units of 256.  Conversions run
// at a quarter of the rate of these additions.
__device__ __forceinline__ int64_t assemble_bounded(uint32_t u1, uint32_t u2, uint32_t u3, uint32_t u4, uint32_t u5,
                                                    uint32_t u6, uint32_t u7) {
  constexpr float M = 12582912.0f;
  constexpr int K = 0x4B400000;  // bits of M
  const int b1 = __float_as_int(__fadd_rn(__uint_as_float(u1), M)), b2 = __float_as_int(__fadd_rn(__uint_as_float(u2), M)),
            b3 = __float_as_int(__fadd_rn(__uint_as_float(u3), M)), b4 = __float_as_int(__fadd_rn(__uint_as_float(u4), M));
  const float f7 = __fadd_rn(__fmaf_rn(__uint_as_float(u7), 0.00390625f, M), -M);
  const int i6 = __float2int_rn(__fadd_rn(__uint_as_float(u6), f7)), i5 = __float2int_rn(__uint_as_float(u5));
  const int p23 = (int)((uint32_t)b2 * 256u + (uint32_t)b3 - (uint32_t)K * 257u);
  const int p45 = (int)((uint32_t)b4 * 256u + (uint32_t)i5 - (uint32_t)K * 256u);
  int64_t S = (int64_t)p45 * 256 + i6;
  S += (int64_t)p23 * (1 << 24);
  return S + (int64_t)((uint64_t)(uint32_t)((b1 - K) * 256) << 32);
}

// Steps of a CTA in order: brick, row tile r0, window c0 >= r0.
struct StepIter : BrickIter {
  int r0, c0;
  __device__ __forceinline__ void begin(const F64Bricks& B) {
    r0 = c0 = 0;
    start(B);
  }
  __device__ __forceinline__ void step(const F64Bricks& B) {
    c0 += kWin;
    if (c0 < R()) return;
    r0 += 128;
    c0 = r0;
    if (r0 < R()) return;
    r0 = c0 = 0;
    next(B);
  }
};

struct F64HamArgs {
  F64Bricks b;
  F64Source f;
  F64HamWork w;
  const double* vpot;
  const int32_t* nodd;
  unsigned long long* next;  // unit of the odd bricks' elements
  int64_t hsize;
  int* status;
};

// V of every slot that an image holds, in brick order, rounded to a multiple of
// 2^-62 of the brick's bound (zero at the other slots, whatever V holds there), and the bounds.
//
// One scale serves all of a brick's pairs, and a pair may hold only those of its
// points where V is small: what V spans, its elements lose.  So the bricks where
// V spans more than the kernel should lose are listed as odd and summed directly
// (their V is zero here): V is not finite; some V but zero lies 2^16 below the
// largest; or an eighth of the points 2^8.  A sign change of a smooth V does
// neither: the potentials of SCF steps on cells of 2 to 64 atoms, with and without
// vacuum, list 0 to 0.06 % of the bricks (up to 0.4 % in the transverse channels
// of non-collinear spin, which are all sign changes).  A line at 2^12 would list
// 0.5 % (10 %), one at 2^8 of a single point 8 % (59 %).
__global__ void __launch_bounds__(kHP) f64_vprep_kernel(F64Bricks b, const double* __restrict__ vpot,
                                                        int64_t* __restrict__ vb, int32_t* __restrict__ vexp,
                                                        int32_t* __restrict__ odd, int32_t* __restrict__ nodd) {
  __shared__ uint32_t s[2];
  __shared__ int far[2];
  const int p = threadIdx.x;
  for (int64_t k = blockIdx.x; k < b.nbricks; k += gridDim.x) {
    const uint64_t cover = __ldg(b.cover + k);
    const int64_t gi = p < b.npts && ((cover >> p) & 1u) ? brick_point_index(k, p, b.bdim, b.nb, b.ngrid) : -1;
    const double v = gi >= 0 ? vpot[gi] : 0.0;
    const uint32_t mine = (uint32_t)__double2hiint(v) & 0x7fffffffu, h = __reduce_max_sync(0xffffffffu, mine);
    if ((p & 31) == 0) s[p >> 5] = h;
    __syncthreads();
    const int E = exp_bound(max(s[0], s[1]));
    const int below = v != 0.0 ? E - 1 - (int)(mine >> 20) : 0;
    const int n = __popc(__ballot_sync(0xffffffffu, below > 8)), any = __any_sync(0xffffffffu, below > 16);
    if ((p & 31) == 0) far[p >> 5] = any ? kHP : n;
    __syncthreads();
    const bool is_odd = E >= kBadExp || 8 * (far[0] + far[1]) > __popcll(cover) ||
                        (cover == 0 && (load_brick(b.bricks + k).size & 0xffffu) > 0);
    int e;
    const uint64_t m = mantissa(v, e) << 10;
    const int64_t t = (int64_t)(((m >> min((uint32_t)(E - e - 1), 63u)) + 1) >> 1);
    vb[k * kHP + p] = is_odd ? 0 : (v < 0.0 ? -t : t);
    if (p == 0) {
      vexp[k] = is_odd ? 1 : E;
      if (is_odd) odd[atomicAdd(nodd, 1)] = (int32_t)k;
    }
  }
}

// The odd bricks' elements as FP64 sums over the points that both images hold,
// as the pair kernels take them.  A warp claims 32 elements of an image pair at a
// time: the blocks that run out of bricks early do most of it.  One odd brick of
// a 2-atom cell's 216 takes 16 us (20 with the units dealt evenly), one of a
// 64-atom cell's 13,824 nothing that shows; if every one of those is odd, 45 ms
// (pair kernels 20).
__device__ __forceinline__ void odd_elements(const F64HamArgs& A, int nodd) {
  constexpr int kParts = 8, kAhead = 8;  // units of an image pair; points whose loads are in flight
  const F64Bricks& B = A.b;
  const F64Source& f = A.f;
  const int lane = threadIdx.x & 31;
  int64_t unit = claim_unit(A.next, lane), base = 0;  // base: the first unit of a brick
  for (int q0 = 0; q0 < nodd; q0 += 32) {
    const int kl = q0 + lane < nodd ? A.w.odd[q0 + lane] : -1;
    const int ml = kl >= 0 ? (int)(load_brick(B.bricks + kl).size >> 16) : 0;
    for (int q = 0; q < min(32, nodd - q0); ++q) {
      const int k = __shfl_sync(0xffffffffu, kl, q), m = __shfl_sync(0xffffffffu, ml, q);
      const int64_t end = base + (int64_t)m * (m + 1) / 2 * kParts;
      for (; unit < end; unit = claim_unit(A.next, lane)) {
        // pair (s, t), s <= t, is number t (t + 1) / 2 + s
        const int part = (int)((unit - base) % kParts), st = (int)((unit - base) / kParts);
        int t = (int)((sqrtf(8.0f * (float)st + 1.0f) - 1.0f) * 0.5f);
        while (t * (t + 1) / 2 > st) --t;
        while ((t + 1) * (t + 2) / 2 <= st) ++t;
        const int s = st - t * (t + 1) / 2;
        const int32_t off = B.tab[(int64_t)load_brick(B.bricks + k).tab + s * m + t];
        if (off < 0) continue;
        const int64_t i0 = f.img_off[k];
        const int as = f.img_atom[i0 + s], at = f.img_atom[i0 + t], noi = f.numorbs[as], noj = f.numorbs[at];
        if (part * 32 >= noi * noj) continue;
        const double *ps = f.phi + f.phi_off[as], *pt = f.phi + f.phi_off[at];
        double* acc = A.w.acc + (k & (kF64Copies - 1)) * A.hsize + off;
        int ks[2], kt[2];
        double v[2];
        uint32_t in[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int p = h * 32 + lane;
          ks[h] = f.slot[(i0 + s) * kHP + p];
          kt[h] = f.slot[(i0 + t) * kHP + p];
          const bool both = ks[h] >= 0 && kt[h] >= 0;
          v[h] = both ? A.vpot[brick_point_index(k, p, B.bdim, B.nb, B.ngrid)] : 0.0;
          in[h] = __ballot_sync(0xffffffffu, both);
        }
        for (int e0 = part * 32; e0 < noi * noj; e0 += 32 * kParts) {
          const int e = e0 + lane;
          const bool on = e < noi * noj;
          const int b = on ? e / noi : 0, a = on ? e - b * noi : 0;
          double sum = 0.0;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            for (uint32_t left = in[h]; left;) {
              double x[kAhead], y[kAhead];
              int n = 0, p[kAhead];
#pragma unroll
              for (int j = 0; j < kAhead; ++j) {  // past the last point: that point again, not added
                p[j] = j > 0 ? p[j - 1] : 0;
                if (left) {
                  p[j] = __ffs(left) - 1;
                  left &= left - 1;
                  ++n;
                }
                x[j] = __ldg(ps + (int64_t)__shfl_sync(0xffffffffu, ks[h], p[j]) * noi + a);
                y[j] = __ldg(pt + (int64_t)__shfl_sync(0xffffffffu, kt[h], p[j]) * noj + b);
              }
#pragma unroll
              for (int j = 0; j < kAhead; ++j) {
                const double w = __shfl_sync(0xffffffffu, v[h], p[j]);
                if (j < n) sum = fma(x[j] * w, y[j], sum);
              }
            }
          }
          if (on && (s < t || a <= b) && bounds_ok((int64_t)off + e, A.hsize, 20)) atomicAdd(acc + e, sum);
        }
      }
      base = end;
    }
  }
}

__global__ void __launch_bounds__(kHThreads, 1) f64_hamiltonian_kernel(const __grid_constant__ F64HamArgs args) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t afree_bar, bready_bar[2], bempty_bar[2], tfull_bar[2], tempty_bar[2], drain_bar;
  __shared__ uint64_t rawfull_bar[kHRaw];
  __shared__ uint32_t tslot;
  __shared__ int nodd;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sched = warp & 3, rank = warp >> 2;
  const int nepi = sched == 0 ? 4 : (sched == 1 ? 3 : 2);  // epilogue warps on this scheduler
  const bool is_mma = warp == 16;
  const F64Bricks& B = args.b;
  uint8_t* sA = smem;
  uint8_t* sB = smem + kDig * kHADigit;
  if (is_mma) tc::tmem_alloc(&tslot, 512);
  if (tid == 0) {
    tc::mbar_init(&afree_bar, 1);
    for (int s = 0; s < kHRaw; ++s) tc::mbar_init(&rawfull_bar[s], 1);
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(&bready_bar[s], kHConv);
      tc::mbar_init(&bempty_bar[s], 1);
      tc::mbar_init(&tfull_bar[s], 1);
      tc::mbar_init(&tempty_bar[s], kHEpi);
    }
    tc::mbar_init(&drain_bar, 1);
    tc::fence_mbar_init();
    abort_flag = 0;
    nodd = *args.nodd;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tslot;
  auto give_up = [&]() {
    if (!abort_flag) atomicExch(args.status, LCP_ETIMEDOUT);
    abort_flag = 1;
  };

  if (rank < nepi) {
    // ------------------------------------------------------------ epilogue
    const uint32_t quarter = (uint32_t)sched;
    uint32_t it = 0;
    BrickIter x;
    for (x.start(B); x.valid() && !abort_flag; x.next(B)) {
      const int R = x.R(), m = x.m();
      const F64Row* rows = B.rows + x.b.row;
      const int32_t* tab = B.tab + x.b.tab;
      const int ve = __ldg(args.w.vexp + x.k);
      double* acc0 = args.w.acc + (x.k & (kF64Copies - 1)) * args.hsize;
      for (int r0 = 0; r0 < R && !abort_flag; r0 += 128) {
        const int rq = r0 + (int)quarter * 32, r = rq + lane;
        F64Row mr{};
        if (r < R) mr = load_meta(rows + r);
        const int s_img = (int)(mr.img_orb >> 8), a = (int)(mr.img_orb & 255u), noi = row_no(mr.info);
        const int r_eff = r < R ? r : 1 << 30;
        const int ea = row_exp(mr.info) + ve - 1023 - 54 - 2046;
        // scales beyond these take scalbn below (phi outside 2^-423 .. 2^177, V
        // above 2^377, V phi below 2^-446); rows of zeros have S = 0
        const auto odd_exp = [](int e) { return e > 1 && (e < 600 || e > 1200); };
        const bool slow_r = __any_sync(0xffffffffu, ve > 1400 ||
                                                        (r < R && (odd_exp(row_exp(mr.info)) ||
                                                                   (row_exp(mr.info) > 1 && row_exp(mr.info) + ve < 1600))));
        double* acc = acc0 + a;
        for (int c0 = r0; c0 < R && !abort_flag; c0 += kWin, ++it) {
          const uint32_t buf = it & 1;
          // the window's columns: lane l keeps column c0 + l for the shuffles below
          F64Row mc{};
          if (c0 + lane < R) mc = load_meta(rows + c0 + lane);
          const bool slow = slow_r || __any_sync(0xffffffffu, c0 + lane < R && odd_exp(row_exp(mc.info)));
          // block offsets of a column group, loaded a group ahead (columns past R: entry t = 0)
          const int32_t* trow = tab + (int64_t)s_img * m;
          auto ask = [&](int cb, int32_t (&o)[4]) {
#pragma unroll
            for (int j = 0; j < 4; ++j) o[j] = __ldg(trow + (__shfl_sync(0xffffffffu, mc.img_orb, cb + j) >> 8));
          };
          int32_t next[4];
          ask(rank * 4, next);
          if (!tc::mbar_wait_warp(&tfull_bar[buf], (it >> 1) & 1, &abort_flag)) {
            give_up();
            break;
          }
          tc::fence_after_sync();
          if (rq < R && rq <= c0) {  // rows of this warp that count in this window
#pragma unroll 1
            for (int cb = rank * 4; cb < kWin; cb += nepi * 4) {
              if (c0 + cb >= R) break;
              int32_t offs[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) offs[j] = next[j];
              ask((cb + nepi * 4) & (kWin - 1), next);
              uint32_t y[kDig][4];
              load_acc(tmem, quarter, buf * kBufCols + cb, y);
              // no branch before the adds: the four columns' chains interleave
              // (with one, each column took 550 clocks of its own latency); one
              // conversion on the FP64 pipe costs less than the dozen integer
              // instructions that normalise S
              double v[4];
              int64_t S[4];
              int ex[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint32_t io = __shfl_sync(0xffffffffu, mc.img_orb, cb + j);
                ex[j] = ea + row_exp(__shfl_sync(0xffffffffu, mc.info, cb + j));
                S[j] = assemble_bounded(y[0][j], y[1][j], y[2][j], y[3][j], y[4][j], y[5][j], y[6][j]);
                // columns past R have S = 0
                const bool counts = r_eff <= c0 + cb + j && offs[j] >= 0 && S[j] != 0;
                offs[j] = counts ? offs[j] + (int)(io & 255u) * noi : -1;
                v[j] = (double)S[j];
              }
              if (!slow) {  // S 2^-54 2^(ea - 1023) 2^(eb - 1023): no under- or overflow
#pragma unroll
                for (int j = 0; j < 4; ++j)
                  v[j] = __hiloint2double(__double2hiint(v[j]) + (ex[j] << 20), __double2loint(v[j]));
              } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                  v[j] = scalbn(v[j], ex[j]);
              }
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (offs[j] >= 0 && bounds_ok((int64_t)offs[j] + a, args.hsize, 20)) atomicAdd(acc + offs[j], v[j]);
            }
          }
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&tempty_bar[buf]);
        }
      }
    }
  } else if (is_mma) {
    // ------------------------------------------------------------ MMA issuer, table producer
    uint32_t it = 0;
    StepIter ahead;  // kHRaw steps ahead
    ahead.begin(B);
    RawRing<kHRaw> ring{smem + kDig * kHADigit + 2 * kHBStage, rawfull_bar};
    auto fetch = [&]() {
      if (!ahead.valid()) return;
      ring.issue(reinterpret_cast<const uint8_t*>(B.table + (int64_t)(ahead.b.chunk + ahead.c0 / 32) * 32 * kHP));
      ahead.step(B);
    };
    for (int i = 0; i < kHRaw; ++i) fetch();
    BrickIter x;
    for (x.start(B); x.valid() && !abort_flag; x.next(B)) {
      const int R = x.R();
      for (int r0 = 0; r0 < R && !abort_flag; r0 += 128) {
        for (int c0 = r0; c0 < R; c0 += kWin, ++it) {
          const uint32_t buf = it & 1, use = it >> 1;
          if (use > 0 && !tc::mbar_wait_warp(&tempty_bar[buf], (use - 1) & 1, &abort_flag)) {
            give_up();
            break;
          }
          if (!tc::mbar_wait_warp(&bready_bar[buf], use & 1, &abort_flag)) {
            give_up();
            break;
          }
          tc::fence_after_sync();
          const uint32_t a0 = tc::smem_u32(sA), b0 = tc::smem_u32(sB + buf * kHBStage), d0 = tmem + buf * kBufCols;
#pragma unroll
          for (int ks = 0; ks < kHP / 16; ++ks) {
            const uint64_t db = tc::smem_desc(b0 + ks * 2 * kHBLbo, kHBLbo, 128);
#pragma unroll
            for (int i = 0; i < kDig; ++i) {
              const uint64_t da = tc::smem_desc(a0 + i * kHADigit + ks * 4096, 2048, 128);
              // digit 0 writes all seven accumulators first
              if (tc::elect_one())
                tc::mma_f16kind(d0 + kWin * i, da, db, idesc_f16_f32(128, kWin * (kDig - i), 0, 0),
                             (ks > 0 || i > 0) ? 1u : 0u);
            }
          }
          if (tc::elect_one()) {
            tc::mma_commit(&bempty_bar[buf]);
            tc::mma_commit(&tfull_bar[buf]);
            if (c0 + kWin >= R) tc::mma_commit(&afree_bar);  // the tile's A may be overwritten
          }
          __syncwarp();
          fetch();  // into this step's slot: its B is split
        }
      }
    }
    if (tc::elect_one()) {
      tc::mma_commit(&drain_bar);
      if (!tc::mbar_wait(&drain_bar, 0, 1u << 24)) give_up();
    }
    __syncwarp();
    ring.drain();
  } else {
    // ------------------------------------------------------------ split
    const int kg = sched == 1 ? rank - 3 : (sched == 2 ? rank : rank + 3);  // 0..7
    uint32_t it = 0, tile = 0, rslot = 0, rpar = 0;
    uint8_t* raw = smem + kDig * kHADigit + 2 * kHBStage;
    StepIter x;
    x.begin(B);
    while (x.valid() && !abort_flag) {
      const int k = x.k;
      const int r0 = x.r0, c0 = x.c0;
      x.step(B);
      longlong2 v[4];
      if (c0 < r0 + 128) {
        const longlong2* vb = reinterpret_cast<const longlong2*>(args.w.vb + (int64_t)k * kHP + kg * 8);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = __ldg(vb + i);
      }
      uint64_t t[8];
      if (!tc::mbar_wait_warp(&rawfull_bar[rslot], rpar, &abort_flag)) {
        give_up();
        break;
      }
      read_piece(raw + rslot * kRawBytes + kg * 2048, lane, t);
      if (++rslot == kHRaw) {
        rslot = 0;
        rpar ^= 1;
      }
      const uint32_t buf = it & 1, use = it >> 1;
      if (use > 0 && !tc::mbar_wait_warp(&bempty_bar[buf], (use - 1) & 1, &abort_flag)) {
        give_up();
        break;
      }
      store_digits(sB + buf * kHBStage + kg * kHBLbo + lane * 16, kWin * 16, t);
      if (c0 < r0 + 128) {  // also row block (c0 - r0) / 32 of A
        if (c0 == r0) {
          if (tile > 0 && !tc::mbar_wait_warp(&afree_bar, (tile - 1) & 1, &abort_flag)) {
            give_up();
            break;
          }
          ++tile;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // t V 2^-62, rounded: V is a multiple of 2^-62 of its bound
          t[2 * i] = (uint64_t)((__mul64hi((int64_t)(t[2 * i] - kF64Bias) * 8, v[i].x) + 1) >> 1) + kF64Bias;
          t[2 * i + 1] = (uint64_t)((__mul64hi((int64_t)(t[2 * i + 1] - kF64Bias) * 8, v[i].y) + 1) >> 1) + kF64Bias;
        }
        store_digits(sA + kg * 2048 + (c0 - r0 + lane) * 16, kHADigit, t);
      }
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bready_bar[buf]);
      __syncwarp();
      ++it;
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (is_mma) tc::tmem_dealloc(tmem, 512);
  if (nodd > 0) odd_elements(args, nodd);
}

// The accumulated blocks (the later of a pair's two blocks, [b][a]), their
// copies added in a fixed order, times gridvol, in both orientations; a self
// pair holds a <= b only.
__global__ void f64_finish_kernel(DevPairs pr, const int32_t* __restrict__ numorbs, const double* __restrict__ acc,
                                  int64_t hsize, double gridvol, double* __restrict__ H) {
  for (int64_t q = blockIdx.x; q < pr.nu; q += gridDim.x) {
    const int noi = numorbs[pr.atom[q]], noj = numorbs[pr.jatom[q]];
    const int64_t bp = pr.boff_p[q], bq = pr.boff_q[q];
    const bool self = pr.self[q] != 0;
    for (int e = threadIdx.x; e < noi * noj; e += blockDim.x) {
      const int b = e / noi, a = e - b * noi;
      if (self && a > b) continue;
      double c[kF64Copies];
#pragma unroll
      for (int i = 0; i < kF64Copies; ++i) c[i] = acc[i * hsize + bq + e];
#pragma unroll
      for (int w = kF64Copies / 2; w > 0; w /= 2)
#pragma unroll
        for (int i = 0; i < w; ++i) c[i] += c[i + w];
      const double v = c[0] * gridvol;
      H[bq + e] = v;
      H[bp + (int64_t)a * noj + b] = v;
    }
  }
}

}  // namespace

// ==========================================================================
// Density and force term.  Per brick of 128 points, over its R packed rows,
//
//   rho(p) = sum_c phi_c(p) X[p][c],  X[p][c] = sum_{r <= c} phi_r(p) Ds[r][c],
//   Ds[r][c] = D_rc + D_cr (r < c),  D_rr (r = c),
//
// (src/Matrix/Set_Density_Grid.jl:268-304), and for the force term
// (src/Force.jl:405-566, 3344-3394) over the rows of all images,
//
//   F[image of c] += w V(p) grad phi_c(p) Y[p][c],  Y[p][c] = sum_r phi_r(p) D_cr.
//
// M = the points, windows of 32 columns, K the packed rows in chunks of 32
// (density: only the rows up to the window).  A (phi, scaled per point) is MN-major,
// so that a lane splits one row at eight points; B (Ds, scaled per column) is
// K-major.
//
// Roles (768 threads, one CTA per SM, persistent over bricks):
//   warps 0-7    epilogue: lane = point, half a window each: X assembled in 64
//                bits, times phi_c(p) into a 128-bit sum (FP64 products took
//                128 clocks per column and warp of this GPU's FP64 pipe);
//   warp 8       MMA issuer: per chunk 2 K steps x 7 MMAs; then the bulk copies
//                of the table's chunk after next;
//   warps 9-16   split A: two of a chunk's sixteen pieces (8 points x 32 rows) each;
//   warps 17-23  split B: its four pieces (8 rows x 32 columns) in turn; the
//                entries' addresses come from the pair tables, two pieces ahead.
// Every split warp has its next chunk's loads in flight while it splits one:
// without that a chunk took 5,000 clocks, whatever the arithmetic.  With four
// warps on B, B set the pace (2,900 clocks a chunk); with one of the A warps
// issuing the copies, that warp did.  Seven warps on B and the copies on the MMA
// warp took the 64-atom 96^3 cell from 1.79 to 1.53 ms (1.60 since rows come in
// segments and columns of any size keep their digits); the integer pipe is the
// busiest unit now (2.5 of 4 instructions a clock issued).
//
// The force term's epilogue holds Y's column as one FP64 value times the
// gradients at its point, read from the point-major tables through the
// brick's slots; the three sums of an image are kept over its columns, and
// reduced over the points when the columns pass to the next image.  The sums
// are added in a fixed order (no atomics).  A random 16-atom 13-orbital cell
// took 5.30 ms with the pair kernel, bound by the FP64 pipe, and takes 1.13 ms.
// ==========================================================================
namespace {

constexpr int kDP = 128;
constexpr int kDEpi = 8, kDConvA = 8, kDConvB = 7, kDConv = kDConvA + kDConvB;
constexpr int kDPiecesB = 4;  // of a chunk's B (8 rows each), taken in turn by the kDConvB warps
constexpr int kDThreads = 32 * (kDEpi + 1 + kDConv);
static_assert(kF64ForceParts == kDEpi * 3, "three sums per image and epilogue warp");
constexpr int kDChunk = 32;
// Rows that one accumulator sums.  |a_d| <= d 2^14 a row, and above 2^24 an MMA
// step truncates; over 256 rows a_1 to a_4 are exact for any digits.  a_5 loses
// 2^-46 of the scales' product a step only if its five digit products average more
// than 0.8 of their largest over a segment; a_6 and a_7 2^-54 and less.  More rows
// of a window are further segments, each with its own buffer and turn of the
// epilogue, which adds up X phi anyway.  (Without segments a_2 is truncated from
// 512 rows on: with 830 that count at a point and large leading digits rho was off
// by 3e-10.)  192 rows would make a_5 exact for any digits too, at 3 % of a step;
// 256 are all that most bricks of cells of 13-orbital atoms have (two segments take
// 0.8 % of the step of a 20-atom 18-orbital cell, 330 rows).  The force term takes
// 320: a_4 then loses 2^-38 a step only if its four products average 0.8 of their
// largest, the leading digits among them, which takes phi of one size in all rows
// (4- to 18-orbital cells: their sum is 11 to 53 times the largest).  A second segment
// of a few rows repeats its epilogue with the gradients: at 256 rows the bricks of
// 260 of a 16-atom cell made the kernel 12 % slower.
template <bool FORCE>
constexpr int kDSeg = FORCE ? 320 : 256;
static_assert(kDSeg<false> % kDChunk == 0 && kDSeg<true> % kDChunk == 0, "segments are whole chunks");
constexpr uint32_t kDStages = 2;
constexpr uint32_t kDEmpty = 4;  // barriers of the chunks' releases, chunk n's at n % 4
static_assert(kDConvB <= 2 * kDPiecesB && kDEmpty >= 2 * kDStages, "a split warp passes over one chunk at most");
constexpr int kDRaw = 4;                                      // half chunks of the table in shared memory
constexpr uint32_t kDADigit = kDP * kDChunk * 2;             // 8 KB: [point group][32 rows][16 B]
constexpr uint32_t kDBLbo = kDig * kWin * 16;
constexpr uint32_t kDBBytes = (kDChunk / 8) * kDBLbo;        // 14 KB
constexpr uint32_t kDStageBytes = kDig * kDADigit + kDBBytes;  // 70 KB
constexpr size_t kDSmemBytes = kDStages * (size_t)kDStageBytes + kDRaw * (size_t)kRawBytes;  // 204 KB
static_assert(2 * kRawBytes == 32 * kDP * 8, "a raw slot is half a chunk");

// sum a_d 256^(7-d) / 256, rounded, over a segment: the sum is below 2^63.
__device__ __forceinline__ int64_t assemble(uint32_t u1, uint32_t u2, uint32_t u3, uint32_t u4, uint32_t u5, uint32_t u6,
                                            uint32_t u7) {
  constexpr float M = 12582912.0f;
  const float f7 = __fadd_rn(__fmaf_rn(__uint_as_float(u7), 0.00390625f, M), -M);
  const int i6 = __float2int_rn(__fadd_rn(__uint_as_float(u6), f7));
  const int a1 = __float2int_rn(__uint_as_float(u1)), a2 = __float2int_rn(__uint_as_float(u2)),
            a3 = __float2int_rn(__uint_as_float(u3)), a4 = __float2int_rn(__uint_as_float(u4)),
            a5 = __float2int_rn(__uint_as_float(u5));
  int64_t S = (int64_t)a5 * 256 + i6;
  S += (int64_t)a4 * 65536;
  S += (int64_t)a3 * (1 << 24);
  return S + (int64_t)((uint64_t)(uint32_t)(a1 * 256 + a2) << 32);
}

struct F64DensArgs {
  F64Bricks b;
  const uint64_t* dfix;
  const uint32_t* cmax;  // [natom * 32] high word of max |Ds| of a column
  const int32_t* btop;   // [nbricks] exponent bound of the largest column of a brick; -1: odd
  double* rho;
  // density: of the odd bricks
  F64Source src;
  const double* dm;
  const int32_t* odd;
  const int32_t* nodd;
  unsigned long long* next;
  F64Force f;            // force term only
  int* status;
};

// Ds per ordered pair and the largest magnitude of each column (orbital b of
// the neighbour atom) and of each atom's own block (smax), one block per pair.
__global__ void __launch_bounds__(128) f64_dsym_kernel(F64Pairs pr, const double* __restrict__ dm,
                                                       double* __restrict__ dsym, uint32_t* __restrict__ cmax,
                                                       uint32_t* __restrict__ smax) {
  __shared__ uint32_t mx[32];
  for (int64_t p = blockIdx.x; p < pr.npairs; p += gridDim.x) {
    const int i = pr.atom[p], j = pr.jatom[p];
    const int noi = pr.numorbs[i], noj = pr.numorbs[j];
    const int q = pr.partner[p];
    const int64_t bp = pr.boff[p], bq = pr.boff[q];
    if (threadIdx.x < 32) mx[threadIdx.x] = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < noi * noj; e += blockDim.x) {
      const int a = e / noj, b = e - a * noj;
      double v = dm[bp + e];
      if (q != p || a != b) v += dm[bq + (int64_t)b * noi + a];
      dsym[bp + e] = v;
      atomicMax(&mx[b], (uint32_t)__double2hiint(v) & 0x7fffffffu);
    }
    __syncthreads();
    if (threadIdx.x < noj) atomicMax(cmax + (int64_t)j * 32 + threadIdx.x, mx[threadIdx.x]);
    if (threadIdx.x < 32 && p == pr.first[i]) {  // the self pair
      const uint32_t h = __reduce_max_sync(0xffffffffu, mx[threadIdx.x]);
      if (threadIdx.x == 0) smax[i] = h;
    }
    __syncthreads();
  }
}

// Exponent bound of the largest column scale among a brick's rows (one warp per
// brick).  Odd, and summed directly: bricks where a column is not finite (an
// element of D reaches only the points that its two atoms hold), or lies further
// below the largest than the sum reaches (2^-120 and not zero), or where a phi is
// not finite; and bricks whose pairs hold only entries more than 2^12 below their
// column's scale, which is the largest of all pairs.  The last is looked into only
// for columns that far above their atom's own block, whose pair is in every brick
// of the atom: for a D of occupied orbitals, |D_rc|^2 <= D_rr D_cc, that takes an
// atom 2^24 emptier than its neighbour.
__global__ void __launch_bounds__(256) f64_btop_kernel(F64Bricks b, const double* __restrict__ dsym,
                                                       const uint32_t* __restrict__ cmax,
                                                       const uint32_t* __restrict__ smax, int32_t* __restrict__ btop,
                                                       int32_t* __restrict__ odd, int32_t* __restrict__ nodd) {
  constexpr int kSpan = 12;
  const int lane = threadIdx.x & 31;
  for (int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; k < b.nbricks;
       k += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const F64Brick br = load_brick(b.bricks + k);
    const int R = (int)(br.size & 0xffffu), m = (int)(br.size >> 16);
    const F64Row* rows = b.rows + br.row;
    auto above = [&](int r, uint32_t& h) {  // the row's column lies far above its atom's own block
      const int c = row_col(load_meta(rows + r).info);
      h = __ldg(cmax + c);
      return exp_bound(h) > exp_bound(__ldg(smax + (c >> 5))) + kSpan;
    };
    int top = 1, low = kBadExp;
    bool any = false;
    for (int r = lane; r < R; r += 32) {
      uint32_t h;
      any |= above(r, h);
      top = max(top, exp_bound(h));
      if (h > 0) low = min(low, exp_bound(h));
    }
    top = __reduce_max_sync(0xffffffffu, top);
    low = __reduce_min_sync(0xffffffffu, low);
    bool is_odd = top >= kBadExp || top - low > 120 || __ldg(b.bad + k) != 0;
    if (!is_odd && __any_sync(0xffffffffu, any)) {
      for (int c = 0; c < R && !is_odd; ++c) {
        uint32_t h, most = 0;
        if (!above(c, h)) continue;
        const F64Row mc = load_meta(rows + c);
        const int t = (int)(mc.img_orb >> 8), noj = row_no(mc.info);
        for (int r = lane; r <= c; r += 32) {  // the entries of the column
          const uint32_t io = load_meta(rows + r).img_orb;
          const int32_t off = __ldg(b.tab + br.tab + (int64_t)(io >> 8) * m + t);
          if (off >= 0)
            most = max(most, (uint32_t)__double2hiint(__ldg(dsym + off + (int)(io & 255u) * noj + (int)(mc.img_orb & 255u))) & 0x7fffffffu);
        }
        most = __reduce_max_sync(0xffffffffu, most);
        is_odd = most > 0 && exp_bound(h) > exp_bound(most) + kSpan;
      }
    }
    if (lane == 0) {
      btop[k] = is_odd ? -1 : top;
      if (is_odd) odd[atomicAdd(nodd, 1)] = (int32_t)k;
    }
  }
}

// The density at the odd bricks' points: the pairs of images that hold a point, a
// warp to a point, as FP64 sums.
__device__ __forceinline__ void odd_points(const F64DensArgs& A, int nodd) {
  const F64Bricks& B = A.b;
  const F64Source& f = A.src;
  const int lane = threadIdx.x & 31;
  for (int64_t unit = claim_unit(A.next, lane); unit < (int64_t)nodd * 128; unit = claim_unit(A.next, lane)) {
    const int k = A.odd[unit >> 7], p = (int)(unit & 127);
    const int64_t gi = p < B.npts ? brick_point_index(k, p, B.bdim, B.nb, B.ngrid) : -1;
    if (gi < 0) continue;
    const F64Brick br = load_brick(B.bricks + k);
    const int m = (int)(br.size >> 16);
    const int64_t i0 = f.img_off[k];
    double sum = 0.0;
    for (int s = 0; s < m; ++s) {
      const int ks = f.slot[(i0 + s) * 128 + p];
      if (ks < 0) continue;
      const int as = f.img_atom[i0 + s], noi = f.numorbs[as];
      const double* ps = f.phi + f.phi_off[as] + (int64_t)ks * noi;
      for (int t = 0; t < m; ++t) {
        const int kt = f.slot[(i0 + t) * 128 + p];
        const int32_t off = kt >= 0 ? B.tab[(int64_t)br.tab + s * m + t] : -1;
        if (off < 0) continue;
        const int at = f.img_atom[i0 + t], noj = f.numorbs[at];
        const double* pt = f.phi + f.phi_off[at] + (int64_t)kt * noj;
        for (int e = lane; e < noi * noj; e += 32) {
          const int a = e / noj, b = e - a * noj;
          sum = fma(__ldg(ps + a) * __ldg(A.dm + off + e), __ldg(pt + b), sum);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o /= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && bounds_ok(gi, (int64_t)B.ngrid[0] * B.ngrid[1] * B.ngrid[2], 21)) A.rho[gi] = sum;
  }
}

// Force term: the largest magnitude of every row of D over its pairs (the
// columns of the product: orbital a of the pair's first atom), one block per pair.
__global__ void __launch_bounds__(128) f64_drow_kernel(F64Pairs pr, const double* __restrict__ dm,
                                                       uint32_t* __restrict__ cmax) {
  __shared__ uint32_t mx[32];
  for (int64_t p = blockIdx.x; p < pr.npairs; p += gridDim.x) {
    const int i = pr.atom[p], noi = pr.numorbs[i], noj = pr.numorbs[pr.jatom[p]];
    const int64_t bp = pr.boff[p];
    if (threadIdx.x < 32) mx[threadIdx.x] = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < noi * noj; e += blockDim.x)
      atomicMax(&mx[e / noj], (uint32_t)__double2hiint(dm[bp + e]) & 0x7fffffffu);
    __syncthreads();
    if (threadIdx.x < noi) atomicMax(cmax + (int64_t)i * 32 + threadIdx.x, mx[threadIdx.x]);
    __syncthreads();
  }
}
__global__ void __launch_bounds__(128) f64_drowfix_kernel(F64Pairs pr, const double* __restrict__ dm,
                                                          const uint32_t* __restrict__ cmax,
                                                          uint64_t* __restrict__ dfix) {
  for (int64_t p = blockIdx.x; p < pr.npairs; p += gridDim.x) {
    const int i = pr.atom[p], noj = pr.numorbs[pr.jatom[p]], n = pr.numorbs[i] * noj;
    const int64_t bp = pr.boff[p];
    for (int e = threadIdx.x; e < n; e += blockDim.x)
      dfix[bp + e] = fx_biased(dm[bp + e], exp_bound(__ldg(cmax + (int64_t)i * 32 + e / noj)));
  }
}

// The images' partial sums by atom: block (atom, slice) adds its slice of the
// images in a fixed order, then force[atom] (+)= gridvol times the slices' sum.
// (One block per atom over all images took 111 us for 16 atoms and 21,000 images.)
__global__ void __launch_bounds__(256) f64_force_slices_kernel(int64_t nimg, const int32_t* __restrict__ img_atom,
                                                               const double* __restrict__ part,
                                                               double* __restrict__ slices) {
  __shared__ double red[3][256];
  const int atom = blockIdx.x;
  const int64_t per = (nimg + kF64ForceSlices - 1) / kF64ForceSlices, i0 = blockIdx.y * per, i1 = min(i0 + per, nimg);
  double v[3] = {0, 0, 0};
  for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x)
    if (img_atom[i] == atom)
      for (int w = 0; w < kDEpi; ++w)
        for (int e = 0; e < 3; ++e) v[e] += part[(i * kDEpi + w) * 3 + e];
  for (int e = 0; e < 3; ++e) red[e][threadIdx.x] = v[e];
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int e = 0; e < 3; ++e) red[e][threadIdx.x] += red[e][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x < 3) slices[((int64_t)blockIdx.y * gridDim.x + atom) * 3 + threadIdx.x] = red[threadIdx.x][0];
}
__global__ void f64_force_sum_kernel(int n, const double* __restrict__ slices, double gridvol, int add,
                                     double* __restrict__ force) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double v = 0.0;
  for (int s = 0; s < kF64ForceSlices; ++s) v += slices[(int64_t)s * n + k];
  force[k] = v * gridvol + (add ? force[k] : 0.0);
}

// Ds on the grids of its columns' scales.
__global__ void __launch_bounds__(128) f64_dfix_kernel(F64Pairs pr, const double* __restrict__ dsym,
                                                       const uint32_t* __restrict__ cmax, uint64_t* __restrict__ dfix) {
  for (int64_t p = blockIdx.x; p < pr.npairs; p += gridDim.x) {
    const int j = pr.jatom[p], noj = pr.numorbs[j], n = pr.numorbs[pr.atom[p]] * noj;
    const int64_t bp = pr.boff[p];
    for (int e = threadIdx.x; e < n; e += blockDim.x)
      dfix[bp + e] = fx_biased(dsym[bp + e], exp_bound(__ldg(cmax + (int64_t)j * 32 + e % noj)));
  }
}

// Chunks of a CTA in order: brick, window c0, row chunk r0 (density: r0 <= c0; force: every chunk).
template <bool FORCE>
__device__ __forceinline__ int last_chunk(int c0, int R) {
  return FORCE ? (R - 1) & ~(kDChunk - 1) : c0;
}
// The segment of rows after r0 of window c0, or the next window's first.
template <bool FORCE>
__device__ __forceinline__ void next_segment(int& c0, int& r0, int R) {
  r0 += kDSeg<FORCE>;
  if (r0 > last_chunk<FORCE>(c0, R)) {
    r0 = 0;
    c0 += kWin;
  }
}
template <bool FORCE, bool AHEAD>
struct ChunkIter : BrickIterT<AHEAD> {
  int c0, r0;
  __device__ __forceinline__ void begin(const F64Bricks& B) {
    c0 = r0 = 0;
    this->start(B);
  }
  __device__ __forceinline__ void step(const F64Bricks& B) {
    r0 += kDChunk;
    if (r0 <= last_chunk<FORCE>(c0, this->R())) return;
    r0 = 0;
    c0 += kWin;
    if (c0 < this->R()) return;
    c0 = 0;
    this->next(B);
  }
};

// Eight rows of a chunk's B for one column per lane, in three steps whose
// loads depend on one another, each a chunk ahead of the next: the rows and
// the column (ask_b), the pair tables' block offsets (locate_b), the entries
// (gather_b).  The L1 that the shared memory leaves is too small to hold any
// of them, so every load takes its time in L2.  No branches around the loads
// (entry 0 where there is nothing), so that they are in flight together.
// Density: Ds of row and column at tab[s][t] + a_row noj + b_col, rows up to the
// column; force: D of (column's atom, row's atom) at tab[t][s] + a_col noj + b_row.
// Nothing here uses a value that it has just loaded: loads of all three steps
// are in flight together (with the entries' selection beside their loads a
// piece took three latencies in turn).
struct BAsk {
  F64Row col, row;  // the column's; of row lane % 8
  uint32_t mask;    // rows that count
  uint32_t tab;
  int m;
  bool ok;
};
struct BPiece {
  uint32_t rio, mask;  // img_orb (and orbital count << 24) of row lane % 8
  int b, noj;          // the column's orbital and its atom's orbitals
  int32_t off[8];
  bool ok;
};
template <bool FORCE>
__device__ __forceinline__ void ask_b(const F64Bricks& B, const ChunkIter<FORCE, false>& x, int g, int lane, BAsk& q) {
  q.ok = x.valid();
  if (!q.ok) return;
  const int c = x.c0 + lane, rh = x.r0 + 8 * g, R = x.R();
  q.tab = x.b.tab;
  q.m = x.m();
  q.col = load_meta(B.rows + x.b.row + min(c, R - 1));
  q.row = load_meta(B.rows + x.b.row + min(rh + (lane & 7), R - 1));
  const int n = (FORCE ? R : c + 1) - rh;  // rows of this piece that count
  q.mask = c < R && n > 0 ? (n >= 8 ? 255u : (1u << n) - 1u) : 0u;
}
template <bool FORCE>
__device__ __forceinline__ void locate_b(const F64Bricks& B, const BAsk& a, BPiece& q) {
  q.ok = a.ok;
  if (!a.ok) return;
  q.rio = a.row.img_orb | ((uint32_t)row_no(a.row.info) << 24);
  q.mask = a.mask;
  q.b = (int)(a.col.img_orb & 255u);
  q.noj = row_no(a.col.info);
  const int t = (int)(a.col.img_orb >> 8);
  const int32_t* tab = B.tab + a.tab + (FORCE ? t * a.m : t);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    q.off[i] = __ldg(tab + (int)((__shfl_sync(0xffffffffu, q.rio, i) >> 8) & 0xffffu) * (FORCE ? 1 : a.m));
}
template <bool FORCE>
__device__ __forceinline__ void gather_b(const uint64_t* __restrict__ dfix, const BPiece& q, uint64_t* t, uint32_t& ok) {
  ok = 0;
  if (!q.ok) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t io = __shfl_sync(0xffffffffu, q.rio, i);
    const int a = (int)(io & 255u);
    const bool y = ((q.mask >> i) & 1u) && q.off[i] >= 0;
    ok |= (y ? 1u : 0u) << i;
    t[i] = __ldg(dfix + (y ? q.off[i] + (FORCE ? q.b * (int)(io >> 24) + a : a * q.noj + q.b) : 0));
  }
}

// Bits by which a brick of R rows aligns its columns' products: the sum of X phi
// over the columns is at most sum_c sum_{r <= c} |phi_r phi_c| < (R^2 + R) / 2 in
// units of the scales' product, and the 128-bit sum holds 2^18-base of them.
// (Seven for any R wrapped the sum from 90 to 130 rows of like size and sign on.)
__device__ __forceinline__ int align_bits(int R) {
  int base = 7;
  while ((R * R + R) / 2 >= 1 << (18 - base)) --base;
  return base;  // 7 to 63 rows, 3 at 200, -1 at 1,000
}

// The 192-bit integer w2:w1:w0 >> n, 0 <= n < 192 (n the same in a warp).
__device__ __forceinline__ void shift_down(uint64_t& w0, uint64_t& w1, int64_t& w2, int n) {
  for (; n >= 64; n -= 64) {
    w0 = w1;
    w1 = (uint64_t)w2;
    w2 >>= 63;
  }
  w0 = (w0 >> n) | (w1 << 1) << (63 - n);
  w1 = (w1 >> n) | ((uint64_t)w2 << 1) << (63 - n);
  w2 >>= n;
}

// The sums of three values over the warp: of the first in lane 0, of the
// second in lane 8, of the third in lane 16 (six additions, not fifteen).
__device__ __forceinline__ double warp_sum3(double v0, double v1, double v2, int lane) {
  const bool up = lane & 16, odd = lane & 8;
  const double x = __shfl_xor_sync(0xffffffffu, up ? v0 : v2, 16), y = __shfl_xor_sync(0xffffffffu, v1, 16);
  const double a = (up ? v2 : v0) + x, b = v1 + y;
  double t = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o /= 2) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

template <bool FORCE>
__global__ void __launch_bounds__(kDThreads, 1) f64_points_kernel(const __grid_constant__ F64DensArgs args) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar[kDStages], empty_bar[kDEmpty], tfull_bar[2], tempty_bar[2], drain_bar;
  __shared__ uint64_t rawfull_bar[kDRaw];
  __shared__ uint64_t s_low[FORCE ? 1 : 32 * kDEpi];  // the low word of the points' sums
  __shared__ uint32_t tslot;
  __shared__ int nodd;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const F64Bricks& B = args.b;
  if (warp == kDEpi) tc::tmem_alloc(&tslot, 512);
  if (tid == 0) {
    for (int s = 0; s < kDRaw; ++s) tc::mbar_init(&rawfull_bar[s], 1);
    for (uint32_t s = 0; s < kDStages; ++s) tc::mbar_init(&full_bar[s], kDConvA + kDPiecesB);
    for (uint32_t s = 0; s < kDEmpty; ++s) tc::mbar_init(&empty_bar[s], 1);
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(&tfull_bar[s], 1);
      tc::mbar_init(&tempty_bar[s], kDEpi);
    }
    tc::mbar_init(&drain_bar, 1);
    tc::fence_mbar_init();
    abort_flag = 0;
    nodd = FORCE ? 0 : *args.nodd;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tslot;
  auto give_up = [&]() {
    if (!abort_flag) atomicExch(args.status, LCP_ETIMEDOUT);
    abort_flag = 1;
  };

  if (warp < kDEpi) {
    // ------------------------------------------------------------ epilogue
    const uint32_t quarter = warp & 3, half = warp >> 2;
    const int p = (int)quarter * 32 + lane;
    uint32_t win = 0;
    if constexpr (FORCE) {
      const F64Force& F = args.f;
      BrickIter x;
      for (x.start(B); x.valid() && !abort_flag; x.next(B)) {
        const int R = x.R();
        const int64_t i0 = __ldg(F.img_off + x.k);
        const int64_t gi = p < B.npts ? brick_point_index(x.k, p, B.bdim, B.nb, B.ngrid) : -1;
        const double vp = gi >= 0 ? F.w * __ldg(F.vpot + gi) : 0.0;
        const int et = __ldg(B.ptexp + (int64_t)x.k * kDP + p);
        const int ep = et >= kBadExp ? kBadExp : et - 2 * 1023 - 54;  // a phi there is not finite: no column is
        int cur = -1, asked = -1, k = -1;  // image of the sums, image whose point is k
        int64_t base = 0;
        double f0 = 0.0, f1 = 0.0, f2 = 0.0;
        bool in = false;  // the point lies in the sphere of cur
        auto flush = [&]() {  // this warp's sums of image cur, added in the order of its windows
          const double s = in ? vp : 0.0;  // outside, whatever V holds there
          const double t = warp_sum3(f0 * s, f1 * s, f2 * s, lane);
          if ((lane & 7) == 0 && lane < 24) F.part[((i0 + cur) * kDEpi + warp) * 3 + (lane >> 3)] += t;
          f0 = f1 = f2 = 0.0;
          in = false;
        };
        for (int c0 = 0, r0 = 0; c0 < R && !abort_flag; ++win) {  // segment r0 of window c0
          const uint32_t buf = win & 1;
          F64Row mc{};
          int ce = 1;
          if (c0 + lane < R) {
            mc = load_meta(B.rows + x.b.row + c0 + lane);
            ce = exp_bound(__ldg(args.cmax + row_col(mc.info)));
          }
          if (!tc::mbar_wait_warp(&tfull_bar[buf], (win >> 1) & 1, &abort_flag)) {
            give_up();
            break;
          }
          tc::fence_after_sync();
#pragma unroll 1
          for (int q = 0; q < 4; ++q) {
            const int cb = (int)half * 16 + q * 4;
            if (c0 + cb >= R) break;
            double d[4][3];
            bool has[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // the gradients of the four columns
              const uint32_t io = __shfl_sync(0xffffffffu, mc.img_orb, cb + j);
              const int no = row_no(__shfl_sync(0xffffffffu, mc.info, cb + j)), img = (int)(io >> 8);
              d[j][0] = d[j][1] = d[j][2] = 0.0;
              has[j] = false;
              if (c0 + cb + j < R) {  // uniform over the warp
                if (img != asked) {
                  asked = img;
                  k = __ldg(F.slot + (i0 + img) * kDP + p);
                  base = __ldg(F.phi_off + __ldg(F.img_atom + i0 + img));
                }
                has[j] = k >= 0;
                if (has[j]) {
                  const int64_t at = base + (int64_t)k * no + (int)(io & 255u);
#pragma unroll
                  for (int e = 0; e < 3; ++e) d[j][e] = __ldg(F.dphi[e] + at);
                }
              }
            }
            uint32_t y[kDig][4];
            load_acc(tmem, quarter, buf * kBufCols + cb, y);
            double v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int ec = __shfl_sync(0xffffffffu, ce, cb + j), e = ec + ep;
              const int64_t S = assemble(y[0][j], y[1][j], y[2][j], y[3][j], y[4][j], y[5][j], y[6][j]);
              v[j] = (double)S;  // times 2^e
              if (e >= kBadExp || ec >= kBadExp) v[j] = has[j] ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
              else if (e > -800 && e < 800 && S != 0)
                v[j] = __hiloint2double(__double2hiint(v[j]) + (e << 20), __double2loint(v[j]));
              else v[j] = scalbn(v[j], e);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int img = (int)(__shfl_sync(0xffffffffu, mc.img_orb, cb + j) >> 8);
              if (c0 + cb + j < R) {
                if (img != cur) {
                  if (cur >= 0) flush();
                  cur = img;
                }
                in |= has[j];
                f0 = fma(v[j], d[j][0], f0);
                f1 = fma(v[j], d[j][1], f1);
                f2 = fma(v[j], d[j][2], f2);
              }
            }
          }
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&tempty_bar[buf]);
          next_segment<FORCE>(c0, r0, R);
        }
        if (abort_flag) break;
        if (cur >= 0) flush();
      }
    } else {
      BrickIter x;
      for (x.start(B); x.valid() && !abort_flag; x.next(B)) {
        const int R = x.R();
        const uint64_t* mine = B.table + (int64_t)x.b.chunk * 32 * kDP + (p >> 3) * 256 + ((p & 7) >> 1) * 64 + (p & 1);
        // S, a multiple of 2^-54 of the scales' product, is a segment's part of X.  The sum
        // of X phi is a 128-bit integer in units 2^-54 2^-(55 + base) of the scales'
        // product with the brick's largest column scale (phi shifted up by base less
        // what the column's scale lies below it, beyond that the product down, into 64
        // more bits below: a column 2^-120 of the largest keeps 52 bits of its own)
        uint64_t slo = 0;
        s_low[tid] = 0;  // not in registers: the kernel has none left, and few windows need it
        const int base = align_bits(R);
        int64_t shi = 0;
        const int etop = __ldg(args.btop + x.k);
        for (int c0 = 0, r0 = 0; c0 < R && !abort_flag; ++win) {  // segment r0 of window c0
          const uint32_t buf = win & 1;
          // lane l keeps how far column c0 + l's scale lies below the brick's
          // largest, for the shuffles below
          int ce = 0;
          if (c0 + lane < R)
            ce = etop - exp_bound(__ldg(args.cmax + row_col(load_meta(B.rows + x.b.row + c0 + lane).info)));
          const bool far = __any_sync(0xffffffffu, ce > base);
          const uint32_t up = 1u << min(max(base - ce, 0), 7);
          const uint64_t* phi = mine + (int64_t)(c0 / 32) * 32 * kDP;
          uint64_t ph[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) ph[j] = __ldg(phi + (half * 16 + j) * 2);  // rows past R are zero in the table
          if (!tc::mbar_wait_warp(&tfull_bar[buf], (win >> 1) & 1, &abort_flag)) {
            give_up();
            break;
          }
          tc::fence_after_sync();
#pragma unroll 1
          for (int q = 0; q < 4; ++q) {
            const int cb = (int)half * 16 + q * 4;
            if (c0 + cb >= R) break;
            uint32_t y[kDig][4];
            load_acc(tmem, quarter, buf * kBufCols + cb, y);
            // no branches: the four columns' chains interleave (with them, each
            // column took 650 clocks of its own latency), and multiplications for
            // shifts: the integer pipe is the busiest one
            int64_t S[4], tp[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int64_t t = (int64_t)(ph[j] - kF64Bias);
              const uint32_t m = __shfl_sync(0xffffffffu, up, cb + j);
              tp[j] = (int64_t)((uint64_t)(uint32_t)t * m + ((uint64_t)((uint32_t)(t >> 32) * m) << 32));
              S[j] = assemble(y[0][j], y[1][j], y[2][j], y[3][j], y[4][j], y[5][j], y[6][j]);
            }
            if (far) {  // columns far below the brick's largest
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int d = __shfl_sync(0xffffffffu, ce, cb + j), n = min(max(d - base, 0), 191);
                // S tp >> n = (S >> n) tp + ((S mod 2^n) tp >> n): the second part here
                const int64_t x = n < 64 ? S[j] & ((1ll << n) - 1) : S[j];
                S[j] = n < 64 ? S[j] >> n : 0;
                uint64_t w0 = 0, w1 = (uint64_t)x * (uint64_t)tp[j];
                int64_t w2 = __mul64hi(x, tp[j]);
                shift_down(w0, w1, w2, n);
                const uint64_t low = s_low[tid] + w0, c = low < w0 ? 1 : 0;
                s_low[tid] = low;
                slo += w1;
                shi += w2 + (slo < w1 ? 1 : 0);
                slo += c;
                shi += slo < c ? 1 : 0;
              }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint64_t lo = (uint64_t)S[j] * (uint64_t)tp[j];
              slo += lo;
              shi += __mul64hi(S[j], tp[j]) + (slo < lo ? 1 : 0);
            }
            if (q < 3) {
#pragma unroll
              for (int j = 0; j < 4; ++j) ph[j] = __ldg(phi + (cb + 4 + j) * 2);
            }
          }
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&tempty_bar[buf]);
          next_segment<FORCE>(c0, r0, R);
        }
        if (abort_flag) break;
        const int64_t gi = p < B.npts ? brick_point_index(x.k, p, B.bdim, B.nb, B.ngrid) : -1;
        uint64_t sx = s_low[tid];
        const bool neg = shi < 0;
        if (neg) {
          sx = ~sx + 1;
          slo = ~slo + (sx == 0 ? 1 : 0);
          shi = ~shi + (sx == 0 && slo == 0 ? 1 : 0);
        }
        double acc = fma((double)shi, 0x1p64, fma((double)sx, 0x1p-64, (double)slo));
        if (neg) acc = -acc;
        // two halves onto a zeroed point: the same sum in either order (odd bricks: odd_points)
        if (gi >= 0 && etop >= 0 && bounds_ok(gi, (int64_t)B.ngrid[0] * B.ngrid[1] * B.ngrid[2], 21))
          atomicAdd(args.rho + gi, scalbn(acc, 2 * (B.ptexp[(int64_t)x.k * kDP + p] - 1023) + etop - 1023 - 109 - base));
      }
    }
  } else if (warp == kDEpi) {
    // ------------------------------------------------------------ MMA issuer, table producer
    uint32_t st = 0, par = 0, win = 0, chunk = 0;
    ChunkIter<FORCE, true> ahead;  // kDRaw / 2 chunks ahead
    ahead.begin(B);
    RawRing<kDRaw> ring{smem + kDStages * kDStageBytes, rawfull_bar};
    auto fetch = [&]() {
      if (!ahead.valid()) return;
      const uint8_t* src = reinterpret_cast<const uint8_t*>(B.table + (int64_t)(ahead.b.chunk + ahead.r0 / 32) * 32 * kDP);
      ring.issue(src);
      ring.issue(src + kRawBytes);
      ahead.step(B);
    };
    for (int i = 0; i < kDRaw / 2; ++i) fetch();
    BrickIter x;
    for (x.start(B); x.valid() && !abort_flag; x.next(B)) {
      const int R = x.R();
      for (int c0 = 0; c0 < R && !abort_flag; c0 += kWin) {
        const int last = last_chunk<FORCE>(c0, R);
        for (int s0 = 0; s0 <= last && !abort_flag; s0 += kDSeg<FORCE>, ++win) {
          const uint32_t buf = win & 1;
          if (win >= 2 && !tc::mbar_wait_warp(&tempty_bar[buf], ((win >> 1) - 1) & 1, &abort_flag)) {
            give_up();
            break;
          }
          const uint32_t d0 = tmem + buf * kBufCols;
          const int end = min(s0 + kDSeg<FORCE> - kDChunk, last);
          for (int r0 = s0; r0 <= end; r0 += kDChunk) {
            if (!tc::mbar_wait_warp(&full_bar[st], par, &abort_flag)) {
              give_up();
              break;
            }
            tc::fence_after_sync();
            const uint32_t a0 = tc::smem_u32(smem + st * kDStageBytes), b0 = a0 + kDig * kDADigit;
#pragma unroll
            for (int ks = 0; ks < kDChunk / 16; ++ks) {
              const uint64_t db = tc::smem_desc(b0 + ks * 2 * kDBLbo, kDBLbo, 128);
#pragma unroll
              for (int i = 0; i < kDig; ++i) {
                const uint64_t da = tc::smem_desc(a0 + i * kDADigit + ks * 256, 128, 512);
                if (tc::elect_one())
                  tc::mma_f16kind(d0 + kWin * i, da, db, idesc_f16_f32(128, kWin * (kDig - i), 1, 0),
                               (r0 > s0 || ks > 0 || i > 0) ? 1u : 0u);
              }
            }
            if (tc::elect_one()) {
              tc::mma_commit(&empty_bar[chunk % kDEmpty]);
              if (r0 == end) tc::mma_commit(&tfull_bar[buf]);
            }
            __syncwarp();
            fetch();  // into this chunk's slots: its A is split
            ++chunk;
            if (++st == kDStages) {
              st = 0;
              par ^= 1;
            }
          }
        }
      }
    }
    if (tc::elect_one()) {
      tc::mma_commit(&drain_bar);
      if (!tc::mbar_wait(&drain_bar, 0, 1u << 24)) give_up();
    }
    __syncwarp();
    ring.drain();
  } else {
    // ------------------------------------------------------------ split
    const int cw = warp - kDEpi - 1;
    // chunk n's stage n % kDStages is free once chunk n - kDStages has been released
    auto stage_free = [&](uint32_t n) {
      const uint32_t u = n - kDStages;
      return n < kDStages || tc::mbar_wait_warp(&empty_bar[u % kDEmpty], (u / kDEmpty) & 1, &abort_flag);
    };
    uint8_t* raw = smem + kDStages * kDStageBytes;
    if (cw < kDConvA) {
      ChunkIter<FORCE, true> x;
      x.begin(B);
      uint32_t n = 0, rslot = 0, rpar = 0;
      for (; x.valid() && !abort_flag; ++n) {
        x.step(B);
        const uint32_t st = n % kDStages;
        bool ok = true;
        uint8_t* sA = smem + st * kDStageBytes;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          ok = ok && tc::mbar_wait_warp(&rawfull_bar[rslot], rpar, &abort_flag);
          if (ok) {
            uint64_t t[8];
            read_piece(raw + rslot * kRawBytes + cw * 2048, lane, t);
            if (++rslot == kDRaw) {
              rslot = 0;
              rpar ^= 1;
            }
            if (h == 0) ok = stage_free(n);
            if (ok) store_digits(sA + (cw + 8 * h) * 512 + lane * 16, kDADigit, t);
          }
        }
        if (!ok) {
          give_up();
          break;
        }
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&full_bar[st]);
        __syncwarp();
      }
    } else {
      // Piece i of the CTA's sequence is piece i % 4 of chunk i / 4; this warp's are
      // kDConvB apart.  It passes chunks over, and a barrier's parity tells a phase
      // from its neighbours only: hence more release barriers than stages.  The
      // warp's last piece waited for a release at most two chunks before the one
      // it waits for next, so the phase before that is past.
      int ga = cw - kDConvA;   // piece to ask for next, counted from x's chunk
      uint32_t piece = ga;     // the piece in t
      ChunkIter<FORCE, false> x;
      x.begin(B);
      auto ask_next = [&](BAsk& ask) {
        for (; ga >= kDPiecesB; ga -= kDPiecesB)
          if (x.valid()) x.step(B);
        ask_b<FORCE>(B, x, ga, lane, ask);
        ga += kDConvB;
      };
      uint64_t t[8];
      uint32_t rows;  // entries of t that there are
      BAsk ask;
      BPiece q;
      ask_next(ask);
      bool now = ask.ok;  // there is a piece in t
      locate_b<FORCE>(B, ask, q);
      ask_next(ask);
      gather_b<FORCE>(args.dfix, q, t, rows);
      locate_b<FORCE>(B, ask, q);
      ask_next(ask);
      for (; now && !abort_flag; piece += kDConvB) {
        const uint32_t c = piece / kDPiecesB, st = c % kDStages;
        if (!stage_free(c)) {
          give_up();
          break;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = (rows >> i) & 1u ? t[i] : kF64Bias;
        store_digits(smem + st * kDStageBytes + kDig * kDADigit + piece % kDPiecesB * kDBLbo + lane * 16, kWin * 16, t);
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&full_bar[st]);
        __syncwarp();
        now = q.ok;
        gather_b<FORCE>(args.dfix, q, t, rows);
        locate_b<FORCE>(B, ask, q);
        ask_next(ask);
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == kDEpi) tc::tmem_dealloc(tmem, 512);
  if constexpr (!FORCE) {
    if (nodd > 0) odd_points(args, nodd);
  }
}

}  // namespace

cudaError_t launch_f64_table(const F64Bricks& b, const F64Source& f, const int32_t* row0, F64Row* rows, int32_t* ptexp,
                             uint64_t* cover, uint64_t* table, cudaStream_t st) {
  const unsigned blocks = (unsigned)std::min<int64_t>(b.nbricks, 152 * 32);
  f64_scales_kernel<<<blocks, 256, 0, st>>>(b, f, row0, rows, ptexp, cover);
  LCP_CUDA_TRY(cudaGetLastError());
  f64_table_kernel<<<blocks, 256, 0, st>>>(b, f, table);
  return cudaGetLastError();
}

cudaError_t launch_f64_density(const F64Bricks& b, const F64Source& f, const F64Pairs& pr, const double* dm,
                               const F64DensWork& w, double* rho, int* status, cudaStream_t st) {
  const int64_t nn = (int64_t)b.ngrid[0] * b.ngrid[1] * b.ngrid[2];
  LCP_CUDA_TRY(cudaMemsetAsync(rho, 0, (size_t)nn * sizeof(double), st));
  if (b.nrows == 0 || pr.npairs == 0) return cudaSuccess;
  LCP_CUDA_TRY(cudaMemsetAsync(w.cmax, 0, ((size_t)pr.natom * 32 + kF64CmaxTail) * sizeof(uint32_t), st));
  int32_t* nodd = reinterpret_cast<int32_t*>(w.cmax + (size_t)pr.natom * 32);
  uint32_t* smax = w.cmax + (size_t)pr.natom * 32 + kF64CmaxTail;
  unsigned long long* next = reinterpret_cast<unsigned long long*>(nodd + 2);
  int32_t* odd = w.btop + b.nbricks;
  const unsigned blocks = (unsigned)std::min<int64_t>(pr.npairs, 152 * 16);
  f64_dsym_kernel<<<blocks, 128, 0, st>>>(pr, dm, w.dsym, w.cmax, smax);
  LCP_CUDA_TRY(cudaGetLastError());
  f64_dfix_kernel<<<blocks, 128, 0, st>>>(pr, w.dsym, w.cmax, w.dfix);
  LCP_CUDA_TRY(cudaGetLastError());
  f64_btop_kernel<<<(unsigned)std::min<int64_t>((b.nbricks + 7) / 8, 152 * 8), 256, 0, st>>>(b, w.dsym, w.cmax, smax, w.btop, odd, nodd);
  LCP_CUDA_TRY(cudaGetLastError());
  F64DensArgs a{b, w.dfix, w.cmax, w.btop, rho, f, dm, odd, nodd, next, F64Force{}, status};
  LCP_CUDA_TRY(raise_smem(f64_points_kernel<false>, kDSmemBytes));
  f64_points_kernel<false><<<(unsigned)std::min<int64_t>(b.nbricks, device_sms()), kDThreads, kDSmemBytes, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_f64_force(const F64Bricks& b, const F64Pairs& pr, int nch, const double* const* vpot,
                             const double* const* dm, const double* coef, const F64Force& f, const F64DensWork& w,
                             double gridvol, double* force, int* status, cudaStream_t st) {
  if (b.nrows == 0 || pr.npairs == 0) return cudaMemsetAsync(force, 0, (size_t)pr.natom * 3 * sizeof(double), st);
  const unsigned blocks = (unsigned)std::min<int64_t>(pr.npairs, 152 * 16);
  LCP_CUDA_TRY(raise_smem(f64_points_kernel<true>, kDSmemBytes));
  for (int c = 0; c < nch; ++c) {
    LCP_CUDA_TRY(cudaMemsetAsync(w.cmax, 0, (size_t)pr.natom * 32 * sizeof(uint32_t), st));
    LCP_CUDA_TRY(cudaMemsetAsync(f.part, 0, (size_t)b.nimg * kF64ForceParts * sizeof(double), st));
    f64_drow_kernel<<<blocks, 128, 0, st>>>(pr, dm[c], w.cmax);
    LCP_CUDA_TRY(cudaGetLastError());
    f64_drowfix_kernel<<<blocks, 128, 0, st>>>(pr, dm[c], w.cmax, w.dfix);
    LCP_CUDA_TRY(cudaGetLastError());
    F64DensArgs a{b, w.dfix, w.cmax, nullptr, nullptr, F64Source{}, nullptr, nullptr, nullptr, nullptr, f, status};
    a.f.vpot = vpot[c];
    a.f.w = coef[c];
    f64_points_kernel<true><<<(unsigned)std::min<int64_t>(b.nbricks, device_sms()), kDThreads, kDSmemBytes, st>>>(a);
    LCP_CUDA_TRY(cudaGetLastError());
    double* slices = f.part + b.nimg * kF64ForceParts;
    f64_force_slices_kernel<<<dim3((unsigned)pr.natom, kF64ForceSlices), 256, 0, st>>>(b.nimg, f.img_atom, f.part, slices);
    LCP_CUDA_TRY(cudaGetLastError());
    f64_force_sum_kernel<<<(unsigned)(pr.natom * 3 + 127) / 128, 128, 0, st>>>(pr.natom * 3, slices, gridvol, c > 0, force);
    LCP_CUDA_TRY(cudaGetLastError());
  }
  return cudaSuccess;
}

cudaError_t launch_f64_hamiltonian(const F64Bricks& b, const F64Source& f, const DevPairs& folded, const double* vpot,
                                   const F64HamWork& w, double gridvol, double* hks, int64_t hsize, int* status,
                                   cudaStream_t st) {
  if (b.nrows == 0 || folded.nu == 0) return cudaMemsetAsync(hks, 0, (size_t)hsize * sizeof(double), st);
  int32_t* nodd = reinterpret_cast<int32_t*>(w.acc + hsize * kF64Copies);
  unsigned long long* next = reinterpret_cast<unsigned long long*>(w.acc + hsize * kF64Copies + 1);
  LCP_CUDA_TRY(cudaMemsetAsync(w.acc, 0, ((size_t)hsize * kF64Copies + 2) * sizeof(double), st));
  f64_vprep_kernel<<<(unsigned)std::min<int64_t>(b.nbricks, 152 * 32), kHP, 0, st>>>(b, vpot, w.vb, w.vexp, w.odd, nodd);
  LCP_CUDA_TRY(cudaGetLastError());
  F64HamArgs a{b, f, w, vpot, nodd, next, hsize, status};
  LCP_CUDA_TRY(raise_smem(f64_hamiltonian_kernel, kHSmemBytes));
  f64_hamiltonian_kernel<<<(unsigned)std::min<int64_t>(b.nbricks, device_sms()), kHThreads, kHSmemBytes, st>>>(a);
  LCP_CUDA_TRY(cudaGetLastError());
  f64_finish_kernel<<<(unsigned)std::min<int64_t>(folded.nu, 152 * 16), 128, 0, st>>>(folded, f.numorbs, w.acc, hsize,
                                                                                       gridvol, hks);
  return cudaGetLastError();
}

}  // namespace lcp
