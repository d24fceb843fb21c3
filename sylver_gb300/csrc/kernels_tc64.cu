// Tensor-core Schur-complement update for FP64 fronts: C -= A B^T with FP64
// accuracy on the BF16 tensor cores (tcgen05, kind::f16).
//
// GB300 runs two FP64 multiply-adds per clock and SM; its BF16 tensor cores
// run about 4000.  Every operand row (the K entries of one front row) is
// written as x = 2^(e - 71) F with a power of two 2^e of one to two times the row's
// 2-norm and F a 72-bit integer (rounded to nearest), and F is cut into eight signed
// digits of nine bits, d1 .. d8, |d| <= 256, exact in BF16 (an error-free
// splitting after Ozaki, Ogita, Oishi and Rump, "Error-free transformations
// of matrix multiplication by using fast routines of matrix multiplication
// and its applications", 2012).  The 36 digit products with index sum
// s = p + q <= 9 are formed on the tensor cores, one FP32 accumulator per s and
// 64 columns of k; its terms are integers, and only s = 8 and 9 can pass 2^24, when
// nearly all digits sit at +-256.  The epilogue converts each accumulator to an
// integer and adds it, shifted by 79 - (9 s - 2) bits, to a 96-bit sum in units of
// 2^(ei + ej - 79); the row norms bound that sum by 2^79 (Cauchy-Schwarz).  C itself is
// updated by one FP64 subtraction.
//
// What that leaves out, relative to 2^(ei + ej), which is one to four times the
// product of the two row norms: per term the seven products with s = 10 (at
// most 7 2^-72), the rounding of F (2^-72 of the row norms) and that of s = 8 and 9
// in the epilogue (2^-68 per 64 columns, and 2^-64 where their sums pass 2^24): below
// (K + 1) 2^-68 if all of it lines up, about sqrt(K) 2^-72 on random digits.  An FP64
// sum of the terms commits up to K 2^-53 sum |a b|.  So an entry d is taken from the
// digits where |d| >= 2^-15 2^(ei + ej), which keeps what is left out below
// (K + 1) 2^-53 |d|, or where |C| >= K 2^-12 2^(ei + ej), which keeps it below 2^-56 |C|; others
// (rows whose large entries do not meet: graded rows, nodes far from one another) are
// summed in FP64 by k_redo64.  Seven digits and no such test left entries of a 20^3
// box up to 2700 units of 2^-53 |L| |L^T| off (an FP64 sum: 22), and those of distant nodes
// of a 100 x 100 grid with a mass term without a correct bit.
//
// Bound by the MMAs.  The products with one digit of A take one or two MMAs, its
// digits of B side by side (12 MMAs per 16 k instead of 36: one costs about 90
// clocks for any N up to 128); the eight accumulators change hands in two halves,
// so that one is drained while the other fills; sixteen warps drain, and four of
// the groups are rounded by adding a constant, since conversions run at 16 per
// clock and SM.  The additions of a group have no branch between them and the next
// group's read: one wait per half, and warps without columns add too.  Steady rate
// of useful FP64 operations (4500 rows, K = 2048): 37 TFLOP/s, 27 on entries of random
// sign, of which 1 % go to k_redo64
// (k_update on the FP64 pipe: 1.0; seven digits and 28 products: 47).
//
// A row with an infinity or NaN gets a scale exponent that turns every entry
// it touches into NaN, as the FP64 products would.
#include "digits.cuh"
#include "tc.hpp"
#include "tc_ptx.cuh"

namespace sylver_gb300 {

namespace {

constexpr int OT = 128, ON = 64;                   // tile rows and columns
constexpr int OZ_STAGES = 2;
constexpr int OZ_A_TILE = OT * OZ_KC * 2;          // one digit plane of an operand tile: 8, 4 KiB
constexpr int OZ_B_TILE = ON * OZ_KC * 2;
constexpr int OZ_A_BYTES = OZ_DIGITS * OZ_A_TILE;
constexpr int OZ_B_BYTES = OZ_DIGITS * OZ_B_TILE;
constexpr int OZ_STAGE_BYTES = OZ_A_BYTES + OZ_B_BYTES;  // 96 KiB
constexpr int OZ_GROUPS = OZ_DIGITS;               // s = 2 .. 9
constexpr int OZ_HALF = 4;                         // groups 0 .. 3 and 4 .. 7 change hands
constexpr int OZ_DRAIN = 2;                        // k chunks summed in an accumulator
constexpr int OZ_EPI_WARP0 = 2;
constexpr int OZ_EPI_WARPS = 16;
constexpr int OZ_EC = ON / (OZ_EPI_WARPS / 4);       // columns per epilogue warp
constexpr int OZ_THREADS = 32 * (OZ_EPI_WARP0 + OZ_EPI_WARPS);
constexpr int OZ_TMEM_COLS = 512;                  // eight accumulators of 64 columns

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y,
                                            int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(su32(dst)),
      "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(su32(bar))
      : "memory");
}

// K-major, 64-byte swizzle descriptor: 512 B between 8-row groups, swizzle
// mode 4 (64 B); the other fields as in sw128_desc.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;
  return d;
}

// kind::f16, FP32 accumulator, BF16 operands, both K-major, 128 x n
__device__ __forceinline__ uint32_t oz_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(OT >> 4) << 24);
}

// A sum in units of 2^-79 of the row and column scales, modulo 2^96.
struct Fix96 {
  uint32_t w0, w1, w2;
};
// a += (hi, mid, lo) 2^(32 i)
__device__ __forceinline__ void add96(Fix96& a, uint32_t lo, uint32_t mid, uint32_t hi) {
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
      : "+r"(a.w0), "+r"(a.w1), "+r"(a.w2)
      : "r"(lo), "r"(mid), "r"(hi));
}
__device__ __forceinline__ void add64(Fix96& a, uint32_t mid, uint32_t hi) {
  asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, %3;"
      : "+r"(a.w1), "+r"(a.w2)
      : "r"(mid), "r"(hi));
}

// a 2^(e - 79), |e| <= OZ_EXP_SAFE, rounded to nearest in integer arithmetic
// (conversions and FP64 multiplies run at two per clock and SM); small: the
// magnitude is below 2^(e - 15)
constexpr int OZ_EXP_SAFE = 900;
__device__ __forceinline__ double fixed_to_double(Fix96 a, int e, bool& weak) {
  const uint32_t sgn = a.w2 & 0x80000000u;
  if (sgn) {
    const uint32_t l = a.w0, m = a.w1, h = a.w2;
    asm("sub.cc.u32 %0, 0, %3;\n\tsubc.cc.u32 %1, 0, %4;\n\tsubc.u32 %2, 0, %5;"
        : "=&r"(a.w0), "=&r"(a.w1), "=&r"(a.w2)
        : "r"(l), "r"(m), "r"(h));
  }
  const bool small = a.w2 == 0;
  weak = small;
  // leading 64 bits
  const uint32_t h = small ? a.w1 : a.w2, m = small ? a.w0 : a.w1, l = small ? 0u : a.w0;
  const int lz = __clzll((long long)(((unsigned long long)h << 32) | m));
  const uint32_t th = h ? __funnelshift_l(m, h, lz) : m << (lz & 31);
  const uint32_t tl = h ? __funnelshift_l(l, m, lz) : 0u;
  const unsigned long long u = ((unsigned long long)th << 32) | tl;
  const unsigned long long r = (u >> 11) + ((u >> 10) & 1);
  // biased exponent of the leading bit less one: r carries its low bit
  const unsigned long long b = ((unsigned long long)sgn << 32) |
                               (((unsigned long long)((small ? 1006 : 1038) + e - lz) << 52) + r);
  return __longlong_as_double(u ? (long long)b : 0ll);
}

// 2^(e - clamp(e)) for row and column exponents outside the safe range; NaN
// where a row or column had a non-finite entry
__device__ __noinline__ double extreme_scale(int e) {
  if (e > OZ_NONFINITE / 2) return __longlong_as_double(0x7ff8000000000000ll);
  const int r = e - max(-OZ_EXP_SAFE, min(OZ_EXP_SAFE, e));
  return __longlong_as_double((long long)(1023 + max(-1000, min(1000, r))) << 52);
}

// sum += round(v) * 2^(79 - (9 s - 2)) for group s = G + 2.  The hardware
// conversion runs at 16 per clock and SM; groups 0 and 1 (below 2^20 by the row
// norms, 64 columns) are rounded by adding 1.5 2^23, groups 6 and 7, whose unit is
// 2^-70 and less, by adding 1.5 2^26 (to a multiple of eight: 2^-68 of the scales
// at most).  What the added constants leave in the sum is group_bias() per call
// of each.
constexpr float OZ_MAGIC23 = 12582912.f, OZ_MAGIC26 = 100663296.f;
template <int G>
__device__ __forceinline__ void add_group(Fix96& a, float v) {
  constexpr int SH = 63 - 9 * G;  // 63, 54, 45, 36, 27, 18, 9, 0
  if constexpr (G < 2) {
    const uint32_t u = __float_as_uint(v + OZ_MAGIC23);
    add64(a, u << (SH - 32), u >> (64 - SH));
  } else if constexpr (G < 4) {
    const int u = __float2int_rn(v);
    add64(a, (uint32_t)u << (SH - 32), (uint32_t)(u >> (64 - SH)));
  } else if constexpr (G < 6) {
    const int u = __float2int_rn(v);
    add96(a, (uint32_t)u << SH, (uint32_t)(u >> (32 - SH)), (uint32_t)(u >> 31));
  } else {  // one is 8 units
    const uint32_t u = __float_as_uint(v + OZ_MAGIC26);
    add96(a, u << (SH + 3), u >> (29 - SH), 0u);
  }
}
// n times what one call of each group's constant adds, modulo 2^96
__device__ __forceinline__ Fix96 group_bias(uint32_t n) {
  constexpr unsigned long long B23 = 0x4b400000ull, B26 = 0x4cc00000ull;
  constexpr unsigned long long LO = (B26 << 12) + (B26 << 3);  // below 2^44
  constexpr unsigned long long HI = (B23 << 31) + (B23 << 22); // times 2^32, below 2^62
  Fix96 r{0, 0, 0};
  const unsigned long long lo = LO * n, hi = HI * n;  // (n < 2^20)
  add96(r, (uint32_t)lo, (uint32_t)(lo >> 32), 0u);
  add64(r, (uint32_t)hi, (uint32_t)(hi >> 32));
  return r;
}

// Persistent: CTA b processes tiles b, b + gridDim.x, ...
//   warp 0 lane 0 : TMA producer (one 3D load of all digit tiles per operand
//                   and 32-wide k chunk),
//   warp 1 lane 0 : MMA issuer; the eight groups have neighbouring accumulators of
//                   64 columns, and the digit tiles of B lie one after another
//                   in shared memory, so one MMA multiplies a digit of A by up
//                   to four of B (N = 256) into as many groups; an MMA takes
//                   about 90 clocks for any N up to 128, and one per digit pair
//                   would make 36 instead of 12 per 16 columns of k.  The
//                   accumulators sum two k chunks; groups 0 .. 3 and 4 .. 7
//                   change hands separately, so that the epilogue reads one half
//                   while the MMAs fill the other,
//   warps 2..17   : epilogue; each thread keeps the fixed-point sums of one
//                   row and 16 columns in registers and reads the next eight
//                   columns of an accumulator while it adds the current ones.
// Eight accumulators fill the tensor memory at 64 columns; with 128 columns
// and four accumulators in turn each k chunk had to be drained by itself, and the
// float-to-integer conversions (16 per clock and SM) alone took as long as the
// MMAs.
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_update_tc64(const __grid_constant__ CUtensorMap mapa,
                  const __grid_constant__ CUtensorMap mapb, double* __restrict__ arena,
                  const int* __restrict__ sexp, const OzTask* __restrict__ tasks, int ntask,
                  unsigned* __restrict__ redo, unsigned* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[OZ_STAGES], empty[OZ_STAGES], acc_full[2], acc_empty[2], done;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  volatile int* abortp = &abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(tasks + blockIdx.x) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&mapa) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&mapb) : "memory");
    for (int s = 0; s < OZ_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], OZ_EPI_WARPS);
    }
    mbar_init(&done, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     su32(&tmem_slot)),
                 "r"(OZ_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  int issued = 0;  // TMA chunks issued by the producer
  if (warp == 0) {
    if (lane == 0) {
      int g = 0;
      for (int ti = blockIdx.x; ti < ntask && !*abortp; ti += gridDim.x) {
        const OzTask t = tasks[ti];
        const int nk = (t.K + OZ_KC - 1) / OZ_KC;
        bool ok = true;
        for (int kc = 0; kc < nk; ++kc, ++g) {
          const int s = g % OZ_STAGES;
          if (g >= OZ_STAGES &&
              !mbar_wait_or_abort(&empty[s], ((g / OZ_STAGES) - 1) & 1, err, abortp)) {
            ok = false;
            break;
          }
          unsigned char* st = smem + s * OZ_STAGE_BYTES;
          mbar_expect_tx(&full[s], OZ_STAGE_BYTES);
          const int x = kc * OZ_KC;
          tma_load_3d(st, &mapa, x, t.a_row, 0, &full[s]);
          tma_load_3d(st + OZ_A_BYTES, &mapb, x, t.b_row, 0, &full[s]);
          issued = g + 1;
        }
        if (!ok) break;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int g = 0, it = 0;  // k chunks; uses of each accumulator
      bool ok = true;
      for (int ti = blockIdx.x; ti < ntask && ok; ti += gridDim.x) {
        const int nk = (tasks[ti].K + OZ_KC - 1) / OZ_KC;
        for (int kc = 0; kc < nk && ok; ++kc, ++g) {
          const int s = g % OZ_STAGES;
          const bool first = kc % OZ_DRAIN == 0;
          const bool last = kc % OZ_DRAIN == OZ_DRAIN - 1 || kc == nk - 1;
          if (!mbar_wait_or_abort(&full[s], (g / OZ_STAGES) & 1, err, abortp)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t ad = sw64_desc(su32(smem + s * OZ_STAGE_BYTES));
          const uint64_t bd = sw64_desc(su32(smem + s * OZ_STAGE_BYTES + OZ_A_BYTES));
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            // the epilogue has read this half's previous sums
            if (first && it > 0) {
              if (!mbar_wait_or_abort(&acc_empty[half], (it - 1) & 1, err, abortp)) {
                ok = false;
                break;
              }
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            // digit p of A times digits q0, q0 + 1, ... of B: groups g0 .. gl
            const int gl = half ? OZ_GROUPS - 1 : OZ_HALF - 1;
#pragma unroll
            for (int p = 0; p <= gl; ++p) {
              const int g0 = max(p, half ? OZ_HALF : 0), q0 = g0 - p;
              const uint64_t ap = ad + (uint64_t)(p * (OZ_A_TILE >> 4));
              const uint64_t bq = bd + (uint64_t)(q0 * (OZ_B_TILE >> 4));
#pragma unroll
              for (int kk = 0; kk < OZ_KC / 16; ++kk)
                mma_bf16(tmem + (uint32_t)(g0 * ON), ap + 2 * kk, bq + 2 * kk,
                         oz_idesc((gl - g0 + 1) * ON),
                         (p > 0 || kk > 0) ? 1u : (first ? 0u : 1u));
            }
            if (last) mma_commit(&acc_full[half]);
          }
          if (last) ++it;
          if (ok) mma_commit(&empty[s]);
        }
      }
      // every MMA issued so far has completed once `done` fires
      mma_commit(&done);
    }
  } else {
    // TMEM lanes [32q, 32q + 32) are this warp's, and columns [16h, 16h + 16)
    // of each tile (of a tile of at most 32 columns: [8h, 8h + 8))
    const int q = warp & 3, h = (warp - OZ_EPI_WARP0) >> 2;
    int it = 0;
    bool ok = true;
    uint32_t ta = 0;  // this warp's columns of accumulator 0
    // start the read of columns [8 b, 8 b + 8) of group gr's accumulator into v, after a
    // wait for its half at the half's first read (warp-uniform: tcgen05.ld is a
    // warp-collective instruction)
    auto fetch = [&](int gr, int b, uint32_t (&v)[8]) {
      if (b == 0 && (gr == 0 || gr == OZ_HALF)) {
        int ready = 0;
        if (lane == 0)
          ready = mbar_wait_or_abort(&acc_full[gr >= OZ_HALF], it & 1, err, abortp);
        ready = __shfl_sync(0xffffffffu, ready, 0);
        if (!ready) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      tmem_ld8_async(ta + (uint32_t)(gr * ON + 8 * b), v);
      return true;
    };
    // the read has landed: hand a half's accumulators back after its last one
    auto landed = [&](int gr, int b, uint32_t (&v)[8]) {
      tmem_ld_wait(v);
      if (b == 0 || (gr != OZ_HALF - 1 && gr != OZ_GROUPS - 1)) return;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[gr >= OZ_HALF]);
    };
    for (int ti = blockIdx.x; ti < ntask && ok; ti += gridDim.x) {
      const OzTask t = tasks[ti];
      const int rt = q * 32 + lane, row = t.row0 + rt;
      const int hw = t.colEnd - t.col0 <= ON / 2 ? OZ_EC / 2 : OZ_EC;
      ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * hw);
      const int c0 = t.col0 + h * hw, ce = min(t.colEnd, c0 + hw);
      const bool on = c0 < ce;  // warp-uniform
      const bool has = row < t.rowEnd;
      // row exponent; lane j holds column c0 + j's
      const int ei = has ? sexp[t.a_row + rt] : 0;
      const int ejl = c0 + lane < ce ? sexp[t.b_row + h * hw + lane] : 0;
      // (what the rounding constants will have added is taken out at the end)
      Fix96 acc[OZ_EC];
      const int nk = (t.K + OZ_KC - 1) / OZ_KC;
#pragma unroll
      for (int j = 0; j < OZ_EC; ++j) acc[j] = Fix96{0, 0, 0};
      for (int kc = 0; kc < nk; kc += OZ_DRAIN) {
        uint32_t va[8], vb[8];
        // (warps without columns add like the others: a branch around the
        // additions kept them from mixing with the reads, 35.5 -> 31.9 TFLOP/s)
        auto add = [&](auto gc, int b, uint32_t (&v)[8]) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            add_group<decltype(gc)::value>(acc[8 * b + j], __uint_as_float(v[j]));
        };
        auto group = [&](auto gc) {
          constexpr int G = decltype(gc)::value;
          if (!ok) return;
          landed(G, 0, va);
          fetch(G, 1, vb);
          add(gc, 0, va);
          landed(G, 1, vb);
          // (the other half's groups may have to be waited for: add first)
          if constexpr (G + 1 == OZ_HALF) add(gc, 1, vb);
          if constexpr (G + 1 < OZ_GROUPS) ok = fetch(G + 1, 0, va);
          if constexpr (G + 1 != OZ_HALF) add(gc, 1, vb);
        };
        ok = fetch(0, 0, va);
        group(std::integral_constant<int, 0>{});
        group(std::integral_constant<int, 1>{});
        group(std::integral_constant<int, 2>{});
        group(std::integral_constant<int, 3>{});
        group(std::integral_constant<int, 4>{});
        group(std::integral_constant<int, 5>{});
        group(std::integral_constant<int, 6>{});
        group(std::integral_constant<int, 7>{});
        if (!ok) break;
        ++it;
      }
      if (!ok) break;
      if (!on) {
        if (lane == 0) redo[ti * OZ_EPI_WARPS + 4 * h + q] = 0;
        continue;
      }
      // columns [c0, cend) of this row are updated (lower triangle, in range)
      const int cend = has ? min(ce, row + 1) : c0;
      const bool safe = __all_sync(0xffffffffu, abs(ei) <= OZ_EXP_SAFE / 2 &&
                                                    abs(ejl) <= OZ_EXP_SAFE / 2);
      double* cp = arena + t.off + row + (int64_t)c0 * t.ld;
      Fix96 bias = group_bias((nk + OZ_DRAIN - 1) / OZ_DRAIN);
      const int lk = 32 - __clz(t.K);  // K < 2^lk
      unsigned left = 0;               // columns left to k_redo64
#pragma unroll
      for (int b = 0; b < OZ_EC / 8; ++b) {
        if (c0 + 8 * b >= ce) break;  // warp-uniform
        double cv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          cv[j] = c0 + 8 * b + j < cend ? cp[(int64_t)(8 * b + j) * t.ld] : 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int jj = 8 * b + j;
          const int e = ei + __shfl_sync(0xffffffffu, ejl, jj);
          Fix96 a = acc[jj];
          asm("sub.cc.u32 %0, %0, %3;\n\tsubc.cc.u32 %1, %1, %4;\n\tsubc.u32 %2, %2, %5;"
              : "+r"(a.w0), "+r"(a.w1), "+r"(a.w2)
              : "r"(bias.w0), "r"(bias.w1), "r"(bias.w2));
          bool weak;
          double d;
          if (safe) {
            d = fixed_to_double(a, e, weak);
          } else {
            d = fixed_to_double(a, max(-OZ_EXP_SAFE, min(OZ_EXP_SAFE, e)), weak);
            d *= extreme_scale(e);
          }
          // exponent of C against K 2^(e - 12)
          const int xc = (int)((unsigned long long)__double_as_longlong(cv[j]) >> 52) & 0x7ff;
          weak = weak && e > OZ_EMPTY / 2 && e < OZ_NONFINITE / 2 && xc - 1023 < e - 12 + lk;
          if (c0 + jj < cend) {
            if (weak) left |= 1u << jj;
            else cp[(int64_t)jj * t.ld] = cv[j] - d;
          }
        }
      }
      const unsigned any = __reduce_or_sync(0xffffffffu, left);
      const int slot = ti * OZ_EPI_WARPS + 4 * h + q;
      if (lane == 0) redo[slot] = any;
      if (any) redo[ntask * OZ_EPI_WARPS + slot * 32 + lane] = left;
    }
  }
  __syncthreads();
  // all MMAs this CTA issued have drained once `done` fires; wait for it even
  // after a failure, before TMEM is freed
  mbar_wait(&done, 0, err);
  // copies still in flight after a failure: wait (bounded) for the last one
  // issued on each stage before the shared memory they target goes away
  if (*abortp && warp == 0 && lane == 0) {
    for (int g = issued - 1; g >= 0 && g >= issued - OZ_STAGES; --g)
      mbar_wait(&full[g % OZ_STAGES], (g / OZ_STAGES) & 1, err);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(OZ_TMEM_COLS)
                 : "memory");
}

// ---------------------------------------------------------------------------
// The entries that k_update_tc64 left, as FP64 sums (redo: a word of column bits
// per tile and epilogue warp, then one per lane of each).  There are few (56^3:
// 0.2 % of the words' columns, most of them of rows far from one another), so that
// what counts is how long one takes: where a column has few, each takes a warp whose
// lanes share its products; else the eight warps of a CTA split few columns' K
// products, at least 32 each, or take a column of 32 rows each.  One warp per column took 18 us for K = 256 (56^3: 5.3 ms of updates in
// all).  Where many are left it is bound by the FP64 pipe.

constexpr int REDO_WARPS = 8, REDO_K = 32, REDO_U = 16;

__global__ void __launch_bounds__(32 * REDO_WARPS) k_redo64(double* __restrict__ arena,
                                                            const OzTask* __restrict__ tasks,
                                                            int ntask,
                                                            const unsigned* __restrict__ redo) {
  __shared__ double part[REDO_WARPS][32];
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slots = ntask * OZ_EPI_WARPS, step = gridDim.x;
  for (int64_t s0 = blockIdx.x; s0 < slots; s0 += 32 * (int64_t)step) {
    const int64_t sl = s0 + (int64_t)lane * step;
    const unsigned word = sl < slots ? redo[sl] : 0u;  // the same in every warp
    for (unsigned any = __ballot_sync(0xffffffffu, word != 0); any; any &= any - 1) {
      const int src = __ffs(any) - 1, slot = (int)(s0 + (int64_t)src * step);
      const OzTask t = tasks[slot / OZ_EPI_WARPS];
      const int h = slot % OZ_EPI_WARPS >> 2, q = slot & 3;
      const int hw = t.colEnd - t.col0 <= ON / 2 ? OZ_EC / 2 : OZ_EC;
      const int c0 = t.col0 + h * hw, ce = min(t.colEnd, c0 + hw);
      const int row = t.row0 + q * 32 + lane;
      const int64_t ld = t.ld;
      const double* p = arena + t.off + (int64_t)t.k0 * ld;
      const double* ap = p + min(row, t.rowEnd - 1);
      const unsigned mine = redo[slots + (int64_t)slot * 32 + lane];
      unsigned m = 0;  // columns taken whole
      int cnt = 0;
      for (unsigned a = __shfl_sync(0xffffffffu, word, src); a; a &= a - 1) {
        const int jj = __ffs(a) - 1, col = c0 + jj;
        unsigned rows = __ballot_sync(0xffffffffu, (mine >> jj & 1) && row >= col && row < t.rowEnd);
        if (col >= ce) break;
        if (__popc(rows) * (t.K / 32 + 20) >= t.K) {  // (20: a load and five shuffles)
          m |= 1u << jj;
          continue;
        }
        // few rows: one warp each, a lane per 32nd product
        for (; rows; rows &= rows - 1) {
          if (cnt++ % REDO_WARPS != warp) continue;
          const int r = t.row0 + q * 32 + __ffs(rows) - 1;
          double* c = arena + t.off + (int64_t)col * ld + r;
          const double cv = *c;
          double s = 0.0;
#pragma unroll 4
          for (int k = lane; k < t.K; k += 32) s = fma(p[k * ld + r], p[k * ld + col], s);
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == 0) *c = cv - s;
        }
      }
      // nsl slices of K by 8 / nsl columns at a time
      int nsl = 1;
      while (t.K > nsl * REDO_K && 2 * nsl * __popc(m) <= REDO_WARPS) nsl *= 2;
      const int kw = (t.K + nsl - 1) / nsl, ka = warp % nsl * kw, kb = min(ka + kw, t.K);
      while (m) {  // block-uniform
        int jj = -1;
        for (int c = 0; c < REDO_WARPS / nsl && m; ++c, m &= m - 1)
          if (c == warp / nsl) jj = __ffs(m) - 1;
        const int col = c0 + jj;
        const bool live = jj >= 0 && col < ce;  // warp-uniform
        const bool store =
            live && warp % nsl == 0 && (mine >> jj & 1) && row >= col && row < t.rowEnd;
        double* c = arena + t.off + (int64_t)col * ld + row;
        const double cv = store ? *c : 0.0;
        double s = 0.0;
        if (live) {
          for (int k = ka; k < kb; k += REDO_U) {
            double x[REDO_U], y[REDO_U];
#pragma unroll
            for (int u = 0; u < REDO_U; ++u) {
              x[u] = k + u < kb ? ap[(k + u) * ld] : 0.0;
              y[u] = k + u < kb ? p[(k + u) * ld + col] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < REDO_U; ++u) {
              if (k + u >= kb) break;
              s = fma(x[u], y[u], s);
            }
          }
        }
        if (nsl > 1) {
          part[warp][lane] = s;
          __syncthreads();
          if (warp % nsl == 0)
            for (int u = 1; u < nsl; ++u) s += part[warp + u][lane];
          __syncthreads();
        }
        if (store) *c = cv - s;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Scale exponent and digits of 32 front rows (one CTA): a first pass over
// the K columns for the row norms (exponents and a 24-bit sum of squares,
// integer and FP32 arithmetic only), a second one, from L2, for the digits.

constexpr int SPLIT_ROWS = 32, SPLIT_K = 64;

__global__ void __launch_bounds__(256) k_oz_split(const double* __restrict__ arena,
                                                  const OzSplit* __restrict__ sp,
                                                  uint16_t* __restrict__ planes,
                                                  int64_t pstride, int pitch,
                                                  int* __restrict__ sexp) {
  __shared__ long long F[SPLIT_ROWS][SPLIT_K + 1];
  __shared__ int re[8][SPLIT_ROWS], rbad[8][SPLIT_ROWS];
  __shared__ float rs[8][SPLIT_ROWS];
  __shared__ int es[SPLIT_ROWS];
  const OzSplit t = sp[blockIdx.x];
  const int i0 = blockIdx.y * SPLIT_ROWS;
  if (i0 >= t.rows) return;  // uniform over the CTA
  const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const bool has = i0 + lane < t.rows;
  const long long* src = reinterpret_cast<const long long*>(arena) + t.off +
                         (int64_t)t.c0 * t.ld + t.r0 + i0 + lane;
  int e = OZ_EMPTY;
  float s = 0.f;
  bool bad = false;
  for (int k0 = ty; k0 < t.K; k0 += 64) {
    long long x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + 8 * u;
      x[u] = (has && k < t.K) ? src[(int64_t)k * t.ld] : 0ll;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) norm_add(e, s, x[u], bad);
  }
  re[ty][lane] = e;
  rs[ty][lane] = s;
  rbad[ty][lane] = bad;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) e = max(e, re[w][lane]);
  s = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    const int d = e - re[w][lane];
    if (d <= 60) s += rs[w][lane] * __uint_as_float((unsigned)(127 - 2 * d) << 23);
    bad = bad || rbad[w][lane];
  }
  e = bad ? OZ_NONFINITE : norm_exponent(e, s);
  if (ty == 0) es[lane] = e;
  if (ty == 0 && has) sexp[t.base + i0 + lane] = e;
  const int kpad = (t.K + OZ_KC - 1) / OZ_KC * OZ_KC;
  for (int k0 = 0; k0 < kpad; k0 += SPLIT_K) {
    long long x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + ty + 8 * u;
      x[u] = (has && k < t.K) ? src[(int64_t)k * t.ld] : 0ll;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) F[lane][ty + 8 * u] = x[u];
    __syncthreads();
    if (k0 + 2 * lane < kpad) {
      for (int r = ty; r < SPLIT_ROWS && i0 + r < t.rows; r += 8) {
        store_digits(F[r][2 * lane], F[r][2 * lane + 1], es[r],
                     planes + (int64_t)(t.base + i0 + r) * pitch + k0 + 2 * lane, pstride);
      }
    }
    __syncthreads();
  }
}

}  // namespace

static size_t tc64_smem_bytes() { return (size_t)OZ_STAGES * OZ_STAGE_BYTES + 1024; }

static int g_num_sms64 = 0;

void prepare_tc64_kernels() {
  SG_CUDA(cudaFuncSetAttribute(k_update_tc64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)tc64_smem_bytes()));
  int dev = 0;
  SG_CUDA(cudaGetDevice(&dev));
  SG_CUDA(cudaDeviceGetAttribute(&g_num_sms64, cudaDevAttrMultiProcessorCount, dev));
}

void make_digit_maps(CUtensorMap* maps, const uint16_t* planes, int64_t pstride, int64_t rows,
                     int pitch) {
  cuuint64_t dims[3] = {(cuuint64_t)pitch, (cuuint64_t)std::max<int64_t>(rows, 1), OZ_DIGITS};
  cuuint64_t strides[2] = {(cuuint64_t)pitch * sizeof(uint16_t),
                           (cuuint64_t)pstride * sizeof(uint16_t)};
  cuuint32_t estr[3] = {1, 1, 1};
  for (int q = 0; q < 2; ++q) {
    cuuint32_t box[3] = {OZ_KC, (cuuint32_t)(q ? ON : OT), OZ_DIGITS};
    CUresult r = encode_fn()(&maps[q], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)planes, dims,
                             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw CudaError("cuTensorMapEncodeTiled failed");
  }
}

void launch_oz_split(const double* arena, const OzSplit* sp, int nsplit, int64_t max_rows,
                     uint16_t* planes, int64_t pstride, int pitch, int* sexp, cudaStream_t s) {
  if (nsplit <= 0 || max_rows <= 0) return;
  dim3 grid((unsigned)nsplit, (unsigned)((max_rows + SPLIT_ROWS - 1) / SPLIT_ROWS));
  k_oz_split<<<grid, 256, 0, s>>>(arena, sp, planes, pstride, pitch, sexp);
}

void launch_update_tc64(const CUtensorMap* maps, double* arena, const int* sexp, const OzTask* t,
                        int ntask, unsigned* redo, unsigned* err, cudaStream_t s) {
  if (ntask <= 0) return;
  const int sms = g_num_sms64 > 0 ? g_num_sms64 : NUM_SMS;
  k_update_tc64<<<std::min(ntask, sms), OZ_THREADS, tc64_smem_bytes(), s>>>(
      maps[0], maps[1], arena, sexp, t, ntask, redo, err);
  launch_pdl(k_redo64, dim3(std::min(ntask * OZ_EPI_WARPS, 8 * sms)), dim3(32 * REDO_WARPS), 0, s,
             arena, t, ntask, (const unsigned*)redo);
}

size_t update_tc64_redo_words(int64_t ntask) { return (size_t)ntask * OZ_EPI_WARPS * 33; }

}  // namespace sylver_gb300
