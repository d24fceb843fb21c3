// Tensor-core Schur-complement update for FP64 fronts: C -= A B^T with FP64
// accuracy on the BF16 tensor cores (tcgen05, kind::f16).
//
// GB300 runs two FP64 multiply-adds per clock and SM; its BF16 tensor cores
// run about 4000.  Every operand row (the K entries of one front row) is
// written as x = 2^(e - 62) F with a power of two 2^e >= the row's 2-norm and
// F a 63-bit integer (rounded to nearest), and F is cut into seven signed
// digits of nine bits, d1 .. d7, |d| <= 256, exact in BF16 (an error-free
// splitting after Ozaki, Ogita, Oishi and Rump, "Error-free transformations
// of matrix multiplication by using fast routines of matrix multiplication
// and its applications", 2012).  The 28 digit products with index sum
// s = p + q <= 8 are formed on the tensor cores, one FP32 accumulator per s and
// 64 columns of k: its terms are integers and their sums stay below 2^24, so
// nothing is rounded there (s = 7 and 8 can pass 2^24 when nearly all digits
// sit at +-256; what is lost then is below 2^-60 of the norms).  The epilogue converts each accumulator to an
// integer and adds it, shifted by 62 - (9 s - 2) bits, to a 64-bit fixed-point
// sum in units of 2^(e_i + e_j - 62); the row norms bound that sum by 2^62
// (Cauchy-Schwarz).  The dropped products, the rounding of F and of the sum
// are each below 2^-62 of the product of the two row norms, against
// 2^-53 per term of an FP64 sum; C itself is updated by one FP64 subtraction.
//
// Bound by the MMAs, and next by the epilogue's additions (with those left out 55
// TFLOP/s, with a third of the MMAs 56).  The
// products with one digit of A take one or two MMAs, its digits of B side by side
// (11 MMAs per 16 k instead of 28: one costs about 90 clocks for any N up to
// 128); the seven accumulators change hands in two halves, so that one is
// drained while the other fills; sixteen warps drain, and four of the seven
// groups are rounded by adding a constant, since conversions run at 16 per clock
// and SM.  The additions of a group have no branch between them and the next
// group's read: one wait per half, and warps without columns add too.  Steady rate
// of useful FP64 operations (4500 rows, K = 2048): 26 TFLOP/s with an MMA per
// digit pair and eight warps, 32 with a wait and a branch per group, 47 now
// (k_update on the FP64 pipe: 1.0).  Loads do not bound it: handing a stage back
// digit by digit instead of whole changed nothing.
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
constexpr int OZ_STAGE_BYTES = OZ_A_BYTES + OZ_B_BYTES;  // 84 KiB
constexpr int OZ_GROUPS = OZ_DIGITS;               // s = 2 .. 8
constexpr int OZ_HALF = 4;                         // groups 0 .. 3 and 4 .. 6 change hands
constexpr int OZ_DRAIN = 2;                        // k chunks summed in an accumulator
constexpr int OZ_EPI_WARP0 = 2;
constexpr int OZ_EPI_WARPS = 16;
constexpr int OZ_EC = ON / (OZ_EPI_WARPS / 4);       // columns per epilogue warp
constexpr int OZ_THREADS = 32 * (OZ_EPI_WARP0 + OZ_EPI_WARPS);
constexpr int OZ_TMEM_COLS = 512;                  // seven accumulators of 64 columns

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

// acc 2^(e - 62), |e| <= OZ_EXP_SAFE, rounded to nearest in integer arithmetic
// (conversions and FP64 multiplies run at two per clock and SM)
constexpr int OZ_EXP_SAFE = 900;
__device__ __forceinline__ double fixed_to_double(long long acc, int e) {
  const unsigned long long sgn = (unsigned long long)acc & 0x8000000000000000ull;
  unsigned long long u = acc < 0 ? 0ull - (unsigned long long)acc : (unsigned long long)acc;
  const int lz = __clzll((long long)u);
  u <<= lz & 63;
  const unsigned long long m = (u >> 11) + ((u >> 10) & 1);
  // biased exponent of the leading bit: 1024 + e - lz; m carries its low bit
  const unsigned long long b = sgn | (((unsigned long long)(1023 + e - lz) << 52) + m);
  return __longlong_as_double(u ? (long long)b : 0ll);
}

// 2^(e - clamp(e)) for row and column exponents outside the safe range; NaN
// where a row or column had a non-finite entry
__device__ __noinline__ double extreme_scale(int e) {
  if (e > OZ_NONFINITE / 2) return __longlong_as_double(0x7ff8000000000000ll);
  const int r = e - max(-OZ_EXP_SAFE, min(OZ_EXP_SAFE, e));
  return __longlong_as_double((long long)(1023 + max(-1000, min(1000, r))) << 52);
}

// fixed-point sum += round(v) * 2^(62 - (9 s - 2)) for group s = G + 2.  The
// hardware conversion runs at 16 per clock and SM; groups 0 and 1 (below 2^20 by
// the row norms, 64 columns) are rounded by adding 1.5 2^23, groups 5 and 6, whose
// unit is 2^-61 and less, by adding 1.5 2^26 (to a multiple of eight: 2^-59 of the
// norms at most).  What the added constants leave in the sum is
// group_bias() per call of each.
constexpr float OZ_MAGIC23 = 12582912.f, OZ_MAGIC26 = 100663296.f;
template <int G>
__device__ __forceinline__ void add_group(unsigned long long& acc, float v) {
  constexpr int SH = 46 - 9 * G;  // 46, 37, 28, 19, 10, 1, -8
  if constexpr (G < 2) {
    const unsigned u = __float_as_uint(v + OZ_MAGIC23);
    const unsigned hi = (unsigned)(acc >> 32) + (u << (SH - 32));
    acc = ((unsigned long long)hi << 32) | (unsigned)acc;
  } else if constexpr (G < 5) {
    acc += (unsigned long long)((long long)__float2int_rn(v) * (long long)(1 << SH));
  } else if constexpr (G == 5) {
    acc += (unsigned long long)__float_as_uint(v + OZ_MAGIC26) * (8u << SH);
  } else {  // one is 8 units: >> 5 in all
    acc += (__float_as_uint(v + OZ_MAGIC26) + 16) >> 5;
  }
}
// (modulo 2^64, as the sum is until its constants are out)
__device__ __forceinline__ unsigned long long group_bias() {
  constexpr unsigned B23 = 0x4b400000u, B26 = 0x4cc00000u;
  return ((unsigned long long)((B23 << 14) + (B23 << 5)) << 32) + (unsigned long long)B26 * 16 +
         (B26 >> 5);
}

// Persistent: CTA b processes tiles b, b + gridDim.x, ...
//   warp 0 lane 0 : TMA producer (one 3D load of all seven digit tiles per
//                   operand and 32-wide k chunk),
//   warp 1 lane 0 : MMA issuer; the seven groups have neighbouring accumulators of
//                   64 columns, and the digit tiles of B lie one after another
//                   in shared memory, so one MMA multiplies a digit of A by up
//                   to four of B (N = 256) into as many groups; an MMA takes
//                   about 90 clocks for any N up to 128, and one per digit pair
//                   made 28 instead of 11 per 16 columns of k.  The
//                   accumulators sum two k chunks; groups 0 .. 3 and 4 .. 6
//                   change hands separately, so that the epilogue reads one half
//                   while the MMAs fill the other,
//   warps 2..17   : epilogue; each thread keeps the fixed-point sums of one
//                   row and 16 columns in registers and reads the next group's
//                   accumulator while it adds the current one.
// Seven accumulators fill the tensor memory at 64 columns; with 128 columns
// and four accumulators in turn each k chunk had to be drained by itself, and the
// float-to-integer conversions (16 per clock and SM) alone took as long as the
// MMAs.
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_update_tc64(const __grid_constant__ CUtensorMap mapa,
                  const __grid_constant__ CUtensorMap mapb, double* __restrict__ arena,
                  const int* __restrict__ sexp, const TcTask* __restrict__ tasks, int ntask,
                  unsigned* __restrict__ err) {
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
        const TcTask t = tasks[ti];
        bool ok = true;
        for (int kc = 0; kc < t.nk; ++kc, ++g) {
          const int s = g % OZ_STAGES;
          if (g >= OZ_STAGES &&
              !mbar_wait_or_abort(&empty[s], ((g / OZ_STAGES) - 1) & 1, err, abortp)) {
            ok = false;
            break;
          }
          unsigned char* st = smem + s * OZ_STAGE_BYTES;
          mbar_expect_tx(&full[s], OZ_STAGE_BYTES);
          const int x = (t.kc0 + kc) * OZ_KC;
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
        const int nk = tasks[ti].nk;
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
    // start the read of group gr's accumulator into v, after a wait for its half
    // at the half's first group (warp-uniform: tcgen05.ld is a warp-collective
    // instruction)
    auto fetch = [&](int gr, uint32_t (&v)[OZ_EC]) {
      if (gr == 0 || gr == OZ_HALF) {
        int ready = 0;
        if (lane == 0)
          ready = mbar_wait_or_abort(&acc_full[gr >= OZ_HALF], it & 1, err, abortp);
        ready = __shfl_sync(0xffffffffu, ready, 0);
        if (!ready) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      tmem_ld16_async(ta + (uint32_t)(gr * ON), v);
      return true;
    };
    // the read of group gr has landed: hand a half's accumulators back after
    // its last group
    auto landed = [&](int gr, uint32_t (&v)[OZ_EC]) {
      tmem_ld_wait(v);
      if (gr != OZ_HALF - 1 && gr != OZ_GROUPS - 1) return;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[gr >= OZ_HALF]);
    };
    for (int ti = blockIdx.x; ti < ntask && ok; ti += gridDim.x) {
      const TcTask t = tasks[ti];
      const int rt = q * 32 + lane, row = t.row0 + rt;
      const int hw = t.colEnd - t.col0 <= ON / 2 ? OZ_EC / 2 : OZ_EC;
      ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * hw);
      const int c0 = t.col0 + h * hw, ce = min(t.colEnd, c0 + hw);
      const bool on = c0 < ce;  // warp-uniform
      const bool has = row < t.rowEnd;
      // row exponent; lane j holds column c0 + j's
      const int ei = has ? sexp[t.a_row + rt] : 0;
      const int ejl = c0 + lane < ce ? sexp[t.b_row + h * hw + lane] : 0;
      // (what the rounding constants will have added is taken out beforehand)
      unsigned long long acc[OZ_EC];
      const unsigned long long bias = ((t.nk + OZ_DRAIN - 1) / OZ_DRAIN) * group_bias();
#pragma unroll
      for (int j = 0; j < OZ_EC; ++j) acc[j] = 0ull - bias;
      for (int kc = 0; kc < t.nk; kc += OZ_DRAIN) {
        uint32_t va[OZ_EC], vb[OZ_EC];
        // (warps without columns add like the others: a branch around the
        // additions kept them from mixing with the reads, 35.5 -> 31.9 TFLOP/s)
        auto add = [&](auto gc, uint32_t (&v)[OZ_EC]) {
#pragma unroll
          for (int j = 0; j < OZ_EC; ++j)
            add_group<decltype(gc)::value>(acc[j], __uint_as_float(v[j]));
        };
        auto step = [&](auto gc, uint32_t (&cur)[OZ_EC], uint32_t (&nxt)[OZ_EC]) {
          constexpr int G = decltype(gc)::value;
          if (!ok) return;
          landed(G, cur);
          // (the other half's groups may have to be waited for: add first)
          if constexpr (G + 1 == OZ_HALF) add(gc, cur);
          if constexpr (G + 1 < OZ_GROUPS) ok = fetch(G + 1, nxt);
          if constexpr (G + 1 != OZ_HALF) add(gc, cur);
        };
        ok = fetch(0, va);
        step(std::integral_constant<int, 0>{}, va, vb);
        step(std::integral_constant<int, 1>{}, vb, va);
        step(std::integral_constant<int, 2>{}, va, vb);
        step(std::integral_constant<int, 3>{}, vb, va);
        step(std::integral_constant<int, 4>{}, va, vb);
        step(std::integral_constant<int, 5>{}, vb, va);
        step(std::integral_constant<int, 6>{}, va, vb);
        if (!ok) break;
        ++it;
      }
      if (!ok) break;
      if (!on) continue;
      // columns [c0, cend) of this row are updated (lower triangle, in range)
      const int cend = has ? min(ce, row + 1) : c0;
      const bool safe = __all_sync(0xffffffffu, abs(ei) <= OZ_EXP_SAFE / 2 &&
                                                    abs(ejl) <= OZ_EXP_SAFE / 2);
      double* cp = arena + t.c_off + row + (int64_t)c0 * t.ldc;
#pragma unroll
      for (int b = 0; b < OZ_EC / 8; ++b) {
        if (c0 + 8 * b >= ce) break;  // warp-uniform
        double cv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          cv[j] = c0 + 8 * b + j < cend ? cp[(int64_t)(8 * b + j) * t.ldc] : 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int jj = 8 * b + j;
          const int e = ei + __shfl_sync(0xffffffffu, ejl, jj);
          double d;
          if (safe) {
            d = fixed_to_double((long long)acc[jj], e);
          } else {
            d = fixed_to_double((long long)acc[jj], max(-OZ_EXP_SAFE, min(OZ_EXP_SAFE, e)));
            d *= extreme_scale(e);
          }
          if (c0 + jj < cend) cp[(int64_t)jj * t.ldc] = cv[j] - d;
        }
      }
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
  e = norm_exponent(e, s);
  if (ty == 0 && has) sexp[t.base + i0 + lane] = bad ? OZ_NONFINITE : e;
  const bool zero = bad || !(s > 0.f);
  const int kpad = (t.K + OZ_KC - 1) / OZ_KC * OZ_KC;
  for (int k0 = 0; k0 < kpad; k0 += SPLIT_K) {
    long long x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + ty + 8 * u;
      x[u] = (has && k < t.K) ? src[(int64_t)k * t.ld] : 0ll;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) F[lane][ty + 8 * u] = zero ? 0ll : to_fixed(x[u], e);
    __syncthreads();
    if (k0 + 2 * lane < kpad) {
      for (int r = ty; r < SPLIT_ROWS && i0 + r < t.rows; r += 8) {
        store_digits(F[r][2 * lane], F[r][2 * lane + 1],
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

void launch_update_tc64(const CUtensorMap* maps, double* arena, const int* sexp, const TcTask* t,
                        int ntask, unsigned* err, cudaStream_t s) {
  if (ntask <= 0) return;
  const int grid = std::min(ntask, g_num_sms64 > 0 ? g_num_sms64 : 148);
  k_update_tc64<<<grid, OZ_THREADS, tc64_smem_bytes(), s>>>(maps[0], maps[1], arena, sexp, t, ntask,
                                                               err);
}

}  // namespace sylver_gb300
