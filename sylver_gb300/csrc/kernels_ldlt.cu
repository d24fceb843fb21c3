// Threshold-pivoted LDL^T kernels: a-posteriori pivoting (APP) by block
// columns of 32, threshold partial pivoting (TPP) for what fails.  Pivot
// decisions, 2x2 inversions and the acceptance test run in FP64 whatever the
// storage type.
//
// Reference algorithm (math and control flow, not code), with the block
// size equal to the inner block size 32 (one level of blocking):
//   APP block-column loop          src/factor_indef.hxx:1338-1474 (notask),
//                                  :885-1183
//   Block::factor: block_ldlt<T,32> on a full 32x32 diagonal block,
//     ldlt_tpp_factor on a partial one (nrow() x ncol(), so the first CB
//     rows of the block row take part)  src/kernels/ldlt_app.hxx:458-560
//   apply_pivot<OP_N/OP_T> + check_threshold
//                                  src/kernels/ldlt_app.hxx:145-255, :579-601
//   Column::adjust (split 2x2)     include/sylver/kernels/Column.hxx:87-101
//   restore_if_required            src/kernels/ldlt_app.hxx:405-431
//   Block::update / calcLD         src/kernels/ldlt_app.hxx:619-718
//   permute_failed                 src/factor_indef.hxx:1190-1288
//   factor_front_indef_failed      src/factor_failed.hxx:29-157
// SPRAL's block_ldlt and ldlt_tpp_factor are not vendored; the pivot
// searches below restate the published algorithms (Duff, Hogg & Lopez,
// SISC 2020): complete pivoting with a 1x1 / 2x2 choice on a full block,
// threshold partial pivoting elsewhere.
//
// Layout difference, same elimination: the reference leaves failed columns
// in their block and applies later pivots to them through the blocks to
// their left (ApplyT / UpdateT), then permutes them to the back at the end.
// Here the commit of a block moves its failed columns behind all columns not
// yet processed, so the next block is the same set of columns as the
// reference's next block, later pivots reach the failed columns as ordinary
// rows below (same multipliers, same threshold test), and at the end they
// are already at the back, in the order the reference puts them.
//
// D^-1 uses the reference storage (src/kernels/ldlt_app.hxx:166-171):
// 1x1 [d^-1, 0], 2x2 [a, b, Inf, c] with (a b; b c) = D^-1, zero pivot [0, 0].
//
// Arithmetic order: every multiply-add of the FP64 path is an explicit
// __fma_rn / __dmul_rn and the file is compiled without FMA contraction, so
// that a CPU restatement with std::fma in the same order reproduces the
// factors bit for bit.
#include <cfloat>

#include "ldlt_dev.hpp"
#include "pivot.cuh"
#include "tile_update.cuh"

namespace sylver_gb300 {

namespace {

constexpr int BW = LDLT_BW;
constexpr int LDB = BW + 1;

__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double dinf() { return __longlong_as_double(0x7ff0000000000000LL); }

__device__ __forceinline__ int block_width(const LdltFront& F, int k) {
  return min(BW, F.n - BW * k);
}
// CB rows that join a partial diagonal block (the reference's block row of
// 32 rows reaches past n)
__device__ __forceinline__ int extra_rows(const LdltFront& F, int w) {
  return w == BW ? 0 : min(BW - w, F.m - F.n);
}

// Warp-wide argmax of v over lanes (first maximum: lowest index on ties);
// lanes with nothing to offer pass v = -1, idx = -1.
template <typename C>
__device__ __forceinline__ void warp_argmax(C& v, int& idx) {
  for (int o = 16; o > 0; o >>= 1) {
    C ov = __shfl_xor_sync(0xffffffffu, v, o);
    int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov > v || (ov == v && oi >= 0 && (idx < 0 || oi < idx))) {
      v = ov;
      idx = oi;
    }
  }
}

// ---------------------------------------------------------------------------
// Magnitude keys for pivot searches: |v| as an unsigned integer, which orders
// like the value, plus one; 0 for NaN (never chosen, as by `>` comparisons).
__device__ __forceinline__ unsigned mag_key(float v) {
  const unsigned b = __float_as_uint(v) & 0x7fffffffu;
  return b > 0x7f800000u ? 0u : b + 1;
}
__device__ __forceinline__ unsigned long long mag_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
  return b > 0x7ff0000000000000ull ? 0ull : b + 1;
}
__device__ __forceinline__ double key_mag(unsigned k) {
  return k ? (double)__uint_as_float(k - 1) : -1.0;
}
__device__ __forceinline__ double key_mag(unsigned long long k) {
  return k ? __longlong_as_double((long long)(k - 1)) : -1.0;
}
__device__ __forceinline__ unsigned warp_max(unsigned k) { return __reduce_max_sync(~0u, k); }
__device__ __forceinline__ unsigned long long warp_max(unsigned long long k) {
  const unsigned hi = (unsigned)(k >> 32), mh = __reduce_max_sync(~0u, hi);
  const unsigned ml = __reduce_max_sync(~0u, hi == mh ? (unsigned)k : 0u);
  return ((unsigned long long)mh << 32) | ml;
}

// ---------------------------------------------------------------------------
// Diagonal block of step k (one CTA of eight warps per front).
//   full block (32 columns): complete pivoting over the block, 1x1 or 2x2;
//   partial block (w < 32 columns, the front's last): threshold partial
//   pivoting over the w columns with rows = the w block rows followed by the
//   first e = min(32 - w, m - n) contribution rows.
// Output: the factored block (unit L, lower) in blk, D^-1, the local
// permutation, the number of pivots taken (ndiag, also the initial
// npass_raw), the L rows of the e extra rows into the apply panel; the block
// permutation is applied to the variable list (the commit applies it to the
// rows of the eliminated columns).
//
// Bound by the serial chain of pivots.  The triangle stays in registers, three
// entries per thread, and nothing is swapped: an entry keeps its two labels
// (original panel rows) and lane x of every warp holds the current position of
// label x.  A pivot takes two block barriers -- every warp reduces its entries'
// magnitudes with redux, ties by position; the owners publish the pivot column
// through shared memory; every thread updates its entries -- where one warp
// with the triangle in shared memory took up to 32 shared-memory round trips
// for the search and as many for the update.  Per launch on the shifted
// 7-point 48^3 (FP32), on 27 x 24 x 21 and on a 14^3 saddle point (FP64): 93,
// 119 and 104 us before, 30, 39 and 37 us now (of which the permutation of the
// eliminated columns' rows moved to the commit).
constexpr int DG_T = 256, DG_W = DG_T / 32, DG_E = 3;
template <typename T>
__global__ void __launch_bounds__(DG_T) k_app_diag(T* __restrict__ arena, T* __restrict__ scratch,
                                                   const LdltFront* __restrict__ fr,
                                                   const CtaMap* __restrict__ cm, LdltStep st) {
  using C = T;  // block arithmetic; FP64 for the pivot tests and 2x2 inverses
  using K = decltype(mag_key(C(0)));
  constexpr unsigned ALL = 0xffffffffu;
  __shared__ C Ls[BW][LDB];  // Ls[s][x]: pivot s's column of L at label x
  __shared__ C col1[BW], col2[BW], dg[BW];
  __shared__ K pkey[DG_W];
  __shared__ unsigned ptie[DG_W];
  __shared__ double dv[2 * BW];
  __shared__ int perm[BW];
  const LdltFront F = fr[cm[blockIdx.x].f];
  const int q = F.fidx, w = block_width(F, st.k), e = extra_rows(F, w), R = w + e;
  const int p = st.p_cur[q];
  const T* A = arena + F.off;
  const int ld = F.ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto prow = [&](int i) { return i < w ? p + i : F.n + (i - w); };  // panel row -> front row
  // entries (er >= ec) of the 32 x 32 lower triangle: columns g and 31 - g
  // together hold 33 of them
  C v[DG_E];
  int er[DG_E], ec[DG_E];
#pragma unroll
  for (int u = 0; u < DG_E; ++u) {
    const int id = tid + DG_T * u, g = id / 33, o = id % 33;
    const bool first = o < BW - g;
    ec[u] = first ? g : BW - 1 - g;
    er[u] = first ? g + o : o - 1;
    if (g >= BW / 2 || er[u] >= R || ec[u] >= w) ec[u] = -1;
    v[u] = ec[u] >= 0 ? (C)A[(int64_t)(p + ec[u]) * ld + prow(er[u])] : C(0);
  }
#pragma unroll
  for (int u = 0; u < DG_E; ++u)
    if (ec[u] >= 0 && er[u] == ec[u]) dg[ec[u]] = v[u];
  for (int idx = tid; idx < BW * LDB; idx += DG_T) (&Ls[0][0])[idx] = C(0);
  if (tid < 2 * BW) dv[tid] = 0.0;
  __syncthreads();
  int mp = lane;  // position of label `lane`
  auto at = [&](int pos) { return __ffs(__ballot_sync(ALL, mp == pos)) - 1; };  // its label
  auto swap_pos = [&](int x, int y) {
    if (mp == x) mp = y;
    else if (mp == y) mp = x;
  };
  // column of label l (every other label's entry with it) into dst
  auto publish = [&](int l, C* dst) {
#pragma unroll
    for (int u = 0; u < DG_E; ++u)
      if (ec[u] >= 0 && er[u] != ec[u]) {
        if (ec[u] == l) dst[er[u]] = v[u];
        else if (er[u] == l) dst[ec[u]] = v[u];
      }
  };
  // update of the entries past position `last` with f(entry, later label,
  // earlier label); the diagonal ones are published
  auto update = [&](int last, auto f) {
#pragma unroll
    for (int u = 0; u < DG_E; ++u) {
      const int pr = __shfl_sync(ALL, mp, er[u] & 31), pc = __shfl_sync(ALL, mp, ec[u] & 31);
      if (ec[u] >= 0 && pr > last && pc > last) {
        const bool rl = pr >= pc;
        v[u] = f(v[u], rl ? er[u] : ec[u], rl ? ec[u] : er[u]);
        if (er[u] == ec[u]) dg[ec[u]] = v[u];
      }
    }
  };
  // 1x1 pivot at position s (label l, its column in col1)
  auto elim1 = [&](int s, int l) {
    const C di = quot(C(1), dg[l]);
    update(s, [&](C x, int i, int j) { return fma_(-col1[i], mul_(col1[j], di), x); });
    if (warp == DG_W - 1) {
      if (lane < R && mp > s) Ls[s][lane] = mul_(col1[lane], di);
      if (lane == l) {
        Ls[s][l] = C(1);
        dv[2 * s] = (double)di;
        dv[2 * s + 1] = 0.0;
      }
    }
  };
  // 2x2 pivot at positions s, s + 1 (labels l1, l2; columns in col1, col2)
  auto elim2 = [&](int s, int l1, int l2) {
    const double a11 = dg[l1], a21 = col1[l2], a22 = dg[l2];
    const double det = __dsub_rn(mul_(a11, a22), mul_(a21, a21));
    const double i11 = quot(a22, det), i12 = quot(-a21, det), i22 = quot(a11, det);
    update(s + 1, [&](C x, int i, int j) {
      const double w1 = col1[j], w2 = col2[j];
      const C x1 = (C)fma_(i11, w1, mul_(i12, w2)), x2 = (C)fma_(i12, w1, mul_(i22, w2));
      return fma_(-col2[i], x2, fma_(-col1[i], x1, x));
    });
    if (warp == DG_W - 1) {
      if (lane < R && mp > s + 1) {
        const double w1 = col1[lane], w2 = col2[lane];
        Ls[s][lane] = (C)fma_(i11, w1, mul_(i12, w2));
        Ls[s + 1][lane] = (C)fma_(i12, w1, mul_(i22, w2));
      }
      if (lane == l1) {
        Ls[s][l1] = C(1);
        dv[2 * s] = i11;
        dv[2 * s + 1] = i12;
        dv[2 * s + 2] = dinf();
        dv[2 * s + 3] = i22;
      }
      if (lane == l2) Ls[s + 1][l2] = C(1);
    }
  };
  int s = 0;
  if (w == BW) {
    // ---- complete pivoting (block_ldlt)
    while (s < w) {
      K key = 0;
      unsigned tie = ~0u;
#pragma unroll
      for (int u = 0; u < DG_E; ++u) {
        const int pr = __shfl_sync(ALL, mp, er[u] & 31), pc = __shfl_sync(ALL, mp, ec[u] & 31);
        if (ec[u] >= 0 && pr >= s && pc >= s) {
          const K ku = mag_key(v[u]);
          const unsigned tu = min(pr, pc) * BW + max(pr, pc);  // column first, then row
          if (ku > key || (ku == key && tu < tie)) { key = ku; tie = tu; }
        }
      }
      {
        const K m = warp_max(key);
        const unsigned tm = __reduce_min_sync(ALL, key == m ? tie : ~0u);
        if (lane == 0) { pkey[warp] = m; ptie[warp] = tm; }
      }
      __syncthreads();
      key = pkey[lane & (DG_W - 1)];
      tie = ptie[lane & (DG_W - 1)];
      {
        const K m = warp_max(key);
        tie = __reduce_min_sync(ALL, key == m ? tie : ~0u);
        key = m;
      }
      const double amax = key_mag(key);
      if (!(amax >= st.small)) {
        // the rest of the block is (numerically) zero: zero pivots, whose
        // columns of L and D are zero
        if (warp == 0 && mp >= s) Ls[mp][lane] = C(1);
        if (tid == 0) atomicOr(st.status, st.action ? ST_ZERO_PIVOT : ST_SINGULAR);
        s = w;
        break;
      }
      const int t = tie % BW, qq = tie / BW;  // t >= qq
      bool two = false;
      int piv = t;
      if (t != qq) {
        const double dt = fabs((double)dg[at(t)]), dq = fabs((double)dg[at(qq)]);
        if (fmax(dt, dq) >= mul_(st.u, amax)) piv = (dt >= dq) ? t : qq;
        else two = true;
      }
      if (!two) {
        const int l = at(piv);
        swap_pos(s, piv);
        publish(l, col1);
        __syncthreads();
        elim1(s, l);
        s += 1;
      } else {
        const int l1 = at(qq), l2 = at(t);
        swap_pos(s, qq);
        swap_pos(s + 1, (t == s) ? qq : t);
        publish(l1, col1);
        publish(l2, col2);
        __syncthreads();
        elim2(s, l1, l2);
        s += 2;
      }
    }
  } else {
    // ---- threshold partial pivoting over the w candidates (ldlt_tpp_factor)
    const double lim = quot(1.0, st.u);
    while (s < w) {
      int decided = 0, piv = -1, tpiv = -1, lc = -1, lt = -1;
      for (int c = s; c < w && !decided; ++c) {
        lc = at(c);
        publish(lc, col1);
        __syncthreads();
        const bool in = lane < R && mp >= s && lane != lc;
        K key = in ? mag_key(col1[lane]) : K(0);
        K m = warp_max(key);
        const unsigned tm = __reduce_min_sync(ALL, in && key == m && m ? (unsigned)mp : ~0u);
        const double amax = fmax(key_mag(m), 0.0), acc = fabs((double)dg[lc]);
        if (amax < st.small && acc < st.small) { decided = 3; piv = c; break; }
        if (acc >= mul_(st.u, amax)) { decided = 1; piv = c; break; }
        if (tm < (unsigned)w) {
          lt = at(tm);
          publish(lt, col2);
          __syncthreads();
          const bool in2 = in && lane != lt;
          const double ap2 = fmax(key_mag(warp_max(in2 ? key : K(0))), 0.0);
          const double at2 = fmax(key_mag(warp_max(in2 ? mag_key(col2[lane]) : K(0))), 0.0);
          const double a11 = dg[lc], a22 = dg[lt], a21 = col1[lt];
          const double det = __dsub_rn(mul_(a11, a22), mul_(a21, a21));
          if (fabs(det) > st.small && isfinite(det)) {
            const double i11 = quot(a22, det), i12 = quot(-a21, det), i22 = quot(a11, det);
            if (fma_(fabs(i11), ap2, mul_(fabs(i12), at2)) <= lim &&
                fma_(fabs(i12), ap2, mul_(fabs(i22), at2)) <= lim) {
              decided = 2; piv = c; tpiv = tm;
              break;
            }
          }
        }
        __syncthreads();  // the columns are read before the next candidate's
      }
      if (!decided) break;
      if (decided == 3) {
        if (!st.action) {
          if (tid == 0) atomicOr(st.status, ST_SINGULAR);
          break;
        }
        swap_pos(s, piv);
        if (warp == 0 && lane == lc) {
          Ls[s][lc] = C(1);
          atomicOr(st.status, ST_ZERO_PIVOT);
        }
        s += 1;
      } else if (decided == 1) {
        swap_pos(s, piv);
        elim1(s, lc);
        s += 1;
      } else {
        swap_pos(s, piv);
        swap_pos(s + 1, (tpiv == s) ? piv : tpiv);
        elim2(s, lc, lt);
        s += 2;
      }
      __syncthreads();  // the columns are read before the next pivot's
    }
  }
  const int nd = s;
  if (warp == 0) perm[mp] = lane;
  __syncthreads();
  C* blk = reinterpret_cast<C*>(st.blk) + (int64_t)q * BW * LDB;
  for (int idx = tid; idx < BW * LDB; idx += DG_T) {
    const int i = idx % LDB, j = idx / LDB;
    blk[idx] = i < BW ? Ls[j][perm[i]] : C(0);
  }
  if (tid < 2 * BW) st.bdinv[q * 2 * BW + tid] = dv[tid];
  if (tid < BW) st.lperm[q * BW + tid] = perm[tid];
  if (tid == 0) {
    st.ndiag[q] = nd;
    st.npass_raw[q] = nd;
  }
  // L of the extra rows (partial block) goes where apply puts rows below
  if (e > 0) {
    T* pan = scratch + F.pan_off;
    for (int idx = tid; idx < e * nd; idx += DG_T) {
      int i = w + idx % e, kk = idx / e;
      pan[(int64_t)kk * F.m + prow(i)] = (T)Ls[kk][i];
    }
  }
  // the block permutation on the variable list
  if (warp == 0) {
    int* var = st.var + F.var_off + p;
    int vv = (lane < w) ? var[perm[lane]] : 0;
    __syncwarp();
    if (lane < w) var[lane] = vv;
  }
}

// rows below block step k in a compressed index: [p + w, n), then (a partial
// block's extra rows excluded) [n + e, m)
struct BelowRows {
  int lo, n, e, m;
  __device__ int count() const { return (n - lo) + (m - n - e); }
  __device__ int row(int ci) const { return ci < n - lo ? lo + ci : n + e + (ci - (n - lo)); }
};

// Pivot kinds of a diagonal block's first `cnt` columns (D^-1 in dv)
enum { PV_ONE, PV_FIRST, PV_SECOND, PV_ZERO };
__device__ __forceinline__ int pivot_kind(const double* dv, int k, int cnt) {
  if (k > 0 && isinf(dv[2 * k])) return PV_SECOND;
  if (k + 1 < cnt && isinf(dv[2 * k + 2])) return PV_FIRST;
  return dv[2 * k] == 0.0 ? PV_ZERO : PV_ONE;
}
// |x| > lim in integer or FP32 arithmetic (false for NaN): same outcome as the
// FP64 comparison, off the FP64 pipe.  lim > 0.
__device__ __forceinline__ bool above(float x, double lim) {
  return fabsf(x) > __double2float_rd(lim);
}
__device__ __forceinline__ bool above(double x, double lim) {
  const long long b = __double_as_longlong(x) & 0x7fffffffffffffffll;
  return b > __double_as_longlong(lim) && b <= 0x7ff0000000000000ll;
}

// ---------------------------------------------------------------------------
// Rows below the diagonal block: x = a P L_kk^-T D^-1 over the ndiag pivots,
// into the apply panel; the least pivot with |x| > 1/u lowers npass_raw.
// One row per thread with its 32 values in registers, every load in flight at
// once, L read from shared memory in 16-byte broadcasts (with the row in shared
// memory a multiply-add took two shared loads and a store).  FP64 goes
// through k_app_apply64.  Per launch on the shifted 48^3: 42 us before,
// 14 us now.
__global__ void __launch_bounds__(AppRows<float>::v)
    k_app_apply32(const float* __restrict__ arena, float* __restrict__ scratch,
                  const LdltFront* __restrict__ fr, const CtaMap* __restrict__ cm, LdltStep st) {
  constexpr int RT = AppRows<float>::v;
  __shared__ __align__(16) float L[BW][BW + 4];  // zero past the ndiag pivots
  __shared__ double dv[2 * BW];
  __shared__ int perm[BW], kind[BW];
  __shared__ int fail;
  const CtaMap c = cm[blockIdx.x];
  const LdltFront F = fr[c.f];
  const int q = F.fidx, w = block_width(F, st.k), e = extra_rows(F, w);
  const int p = st.p_cur[q], nd = st.ndiag[q];
  if (nd == 0) return;
  const float* A = arena + F.off;
  const int64_t ld = F.ld, pm = F.m;
  const int tid = threadIdx.x;
  const float* blk = reinterpret_cast<const float*>(st.blk) + (int64_t)q * BW * LDB;
  for (int idx = tid; idx < BW * BW; idx += RT) {
    const int j = idx / BW, k = idx % BW;
    L[j][k] = (j < nd && k < nd) ? blk[j * LDB + k] : 0.f;
  }
  for (int k = tid; k < 2 * BW; k += RT) dv[k] = st.bdinv[q * 2 * BW + k];
  if (tid < BW) perm[tid] = st.lperm[q * BW + tid];
  if (tid == 0) fail = nd;
  __syncthreads();
  if (tid < BW) kind[tid] = pivot_kind(dv, tid, nd);
  __syncthreads();
  const BelowRows br{p + w, F.n, e, F.m};
  const int nrow = br.count();
  const double lim = quot(1.0, st.u);
  float* pan = scratch + F.pan_off;
  for (int t0 = c.local * RT; t0 < nrow; t0 += c.count * RT) {
    const int ci = t0 + tid;
    if (ci < nrow) {
      const int r = br.row(ci);
      float x[BW];
#pragma unroll
      for (int k = 0; k < BW; ++k) x[k] = k < nd ? A[(p + perm[k]) * ld + r] : 0.f;
      // x L^T = a  (unit lower L)
#pragma unroll
      for (int j = 0; j < BW - 1; ++j) {
        if (j >= nd) break;
        const float xj = -x[j];
#pragma unroll
        for (int kv = (j + 1) / 4 * 4; kv < BW; kv += 4) {
          const float4 lv = *reinterpret_cast<const float4*>(&L[j][kv]);
          if (kv > j) x[kv] = fma_(xj, lv.x, x[kv]);
          if (kv + 1 > j) x[kv + 1] = fma_(xj, lv.y, x[kv + 1]);
          if (kv + 2 > j) x[kv + 2] = fma_(xj, lv.z, x[kv + 2]);
          x[kv + 3] = fma_(xj, lv.w, x[kv + 3]);
        }
      }
      // times D^-1 (apply_pivot OP_N)
#pragma unroll
      for (int k = 0; k < BW; ++k) {
        if (k >= nd) break;
        const int kd = kind[k];
        if (kd == PV_ONE) {
          x[k] = mul_(x[k], (float)dv[2 * k]);
        } else if (kd == PV_FIRST) {
          if (k + 1 < BW) {
            const double x1 = x[k], x2 = x[k + 1];
            x[k] = (float)fma_(dv[2 * k], x1, mul_(dv[2 * k + 1], x2));
            x[k + 1] = (float)fma_(dv[2 * k + 1], x1, mul_(dv[2 * k + 3], x2));
          }
        } else if (kd == PV_ZERO) {
          const double v = x[k];
          x[k] = (float)((fabs(v) < st.small) ? 0.0 : dinf() * v);
        }
      }
      int first = nd;
#pragma unroll
      for (int k = BW - 1; k >= 0; --k)
        if (k < nd && above(x[k], lim)) first = k;
      if (first < nd) atomicMin(&fail, first);
#pragma unroll
      for (int k = 0; k < BW; ++k)
        if (k < nd) pan[k * pm + r] = x[k];
    }
  }
  __syncthreads();
  if (tid == 0 && fail < nd) atomicMin(&st.npass_raw[q], fail);
}

// The same for FP64, four lanes per row (128 threads for 32 rows), lane group c
// holding columns c, c + 4, ...: an FP64 instruction keeps a scheduler's pipe for
// 65 clocks however many lanes it has, so a row per lane left 3/4 of the SM's
// pipes idle wherever a launch has fewer rows than the chip has warps.  Every
// entry keeps its operations and their order.  14^3 saddle point: 30 -> 16 us per
// launch.
constexpr int R4 = AppRows<double>::v, T4 = 4 * R4;  // rows, threads
constexpr int NC4 = BW / 4, RW4 = 8;                 // columns a lane, rows a warp
// the row's values in columns k - 1 and k + 1, k = 4 u + c
__device__ __forceinline__ void neighbours4(const double (&x)[NC4], int u, int rl, int c,
                                            double& prev, double& next) {
  constexpr unsigned FULL = 0xffffffffu;
  const double n0 = __shfl_sync(FULL, x[u], rl + ((c + 1) & 3) * RW4);
  const double n1 = u + 1 < NC4 ? __shfl_sync(FULL, x[u + 1 < NC4 ? u + 1 : u], rl) : 0.0;
  const double p0 = __shfl_sync(FULL, x[u], rl + ((c + 3) & 3) * RW4);
  const double p1 = u > 0 ? __shfl_sync(FULL, x[u > 0 ? u - 1 : 0], rl + 3 * RW4) : 0.0;
  next = c < 3 ? n0 : n1;
  prev = c > 0 ? p0 : p1;
}

__global__ void __launch_bounds__(T4) k_app_apply64(const double* __restrict__ arena,
                                                    double* __restrict__ scratch,
                                                    const LdltFront* __restrict__ fr,
                                                    const CtaMap* __restrict__ cm, LdltStep st) {
  __shared__ double L[BW][BW + 2];  // zero past the ndiag pivots
  __shared__ double dv[2 * BW];
  __shared__ int perm[BW], kind[BW];
  __shared__ int fail, has2;
  const CtaMap c = cm[blockIdx.x];
  const LdltFront F = fr[c.f];
  const int q = F.fidx, w = block_width(F, st.k), e = extra_rows(F, w);
  const int p = st.p_cur[q], nd = st.ndiag[q];
  if (nd == 0) return;
  const double* A = arena + F.off;
  const int64_t ld = F.ld, pm = F.m;
  const int tid = threadIdx.x, lane = tid & 31, rl = lane % RW4, cg = lane / RW4;
  const double* blk = st.blk + (int64_t)q * BW * LDB;
  for (int idx = tid; idx < BW * BW; idx += T4) {
    const int j = idx / BW, k = idx % BW;
    L[j][k] = (j < nd && k < nd) ? blk[j * LDB + k] : 0.0;
  }
  if (tid < 2 * BW) dv[tid] = st.bdinv[q * 2 * BW + tid];
  if (tid < BW) perm[tid] = st.lperm[q * BW + tid];
  if (tid == 0) fail = nd;
  __syncthreads();
  if (tid < BW) {
    kind[tid] = pivot_kind(dv, tid, nd);
    const unsigned two = __ballot_sync(0xffffffffu, kind[tid] == PV_FIRST && tid < nd);
    if (tid == 0) has2 = two != 0;
  }
  __syncthreads();
  const BelowRows br{p + w, F.n, e, F.m};
  const int nrow = br.count();
  const double lim = quot(1.0, st.u);
  double* pan = scratch + F.pan_off;
  for (int t0 = c.local * R4; t0 < nrow; t0 += c.count * R4) {
    const int ci = t0 + (tid >> 5) * RW4 + rl;
    const bool has = ci < nrow;
    const int r = has ? br.row(ci) : 0;
    double x[NC4];
#pragma unroll
    for (int u = 0; u < NC4; ++u) {
      const int k = 4 * u + cg;
      x[u] = has && k < nd ? A[(p + perm[k]) * ld + r] : 0.0;
    }
    // x L^T = a  (unit lower L)
#pragma unroll
    for (int u0 = 0; u0 < NC4; ++u0) {
      for (int jj = 0; jj < 4 && 4 * u0 + jj < nd; ++jj) {
        const double xj = -__shfl_sync(0xffffffffu, x[u0], rl + jj * RW4);
        const double* lj = &L[4 * u0 + jj][cg];
        if (cg > jj) x[u0] = fma_(xj, lj[4 * u0], x[u0]);
#pragma unroll
        for (int u = u0 + 1; u < NC4; ++u) x[u] = fma_(xj, lj[4 * u], x[u]);
      }
    }
    // times D^-1 (apply_pivot OP_N)
    double y[NC4];
#pragma unroll
    for (int u = 0; u < NC4; ++u) {
      const int k = 4 * u + cg;
      double xp = 0.0, xn = 0.0;
      if (has2) neighbours4(x, u, rl, cg, xp, xn);
      double v = x[u];
      if (k < nd) {
        const int kd = kind[k];
        if (kd == PV_ONE) {
          v = mul_(x[u], dv[2 * k]);
        } else if (kd == PV_FIRST && k + 1 < BW) {
          v = fma_(dv[2 * k], x[u], mul_(dv[2 * k + 1], xn));
        } else if (kd == PV_SECOND && k > 0 && kind[k - 1] == PV_FIRST) {
          v = fma_(dv[2 * k - 1], xp, mul_(dv[2 * k + 1], x[u]));
        } else if (kd == PV_ZERO) {
          v = (fabs(x[u]) < st.small) ? 0.0 : dinf() * x[u];
        }
      }
      y[u] = v;
    }
    if (has) {
      int first = nd;
#pragma unroll
      for (int u = NC4 - 1; u >= 0; --u) {
        const int k = 4 * u + cg;
        if (k < nd && above(y[u], lim)) first = k;
      }
      if (first < nd) atomicMin(&fail, first);
#pragma unroll
      for (int u = 0; u < NC4; ++u) {
        const int k = 4 * u + cg;
        if (k < nd) pan[k * pm + r] = y[u];
      }
    }
  }
  __syncthreads();
  if (tid == 0 && fail < nd) atomicMin(&st.npass_raw[q], fail);
}

// ---------------------------------------------------------------------------
// Commit over rows [p, m): passed columns get L (and L*D of the rows from
// p + npass on, for the trailing update), failed columns get back their
// values from before the step in the block's symmetric order (the front
// itself is the backup: nothing before the commit writes it in the block's
// columns).  The block's permutation is applied to its rows of the eliminated
// columns.  The CTA with local index 0 stores D and the state.  One row per
// thread, its 32 values in registers: 35 -> 16 us per launch on the shifted
// 48^3.  FP64 goes through k_app_commit64.
__global__ void __launch_bounds__(AppRows<float>::v)
    k_app_commit32(float* __restrict__ arena, float* __restrict__ scratch,
                   const LdltFront* __restrict__ fr, const CtaMap* __restrict__ cm, LdltStep st) {
  constexpr int RT = AppRows<float>::v;
  __shared__ float L[BW][LDB];
  __shared__ double dv[2 * BW];
  __shared__ double dca[BW], dcb[BW];  // D of a 2x2 pair's two columns
  __shared__ int perm[BW], kind[BW];
  const CtaMap c = cm[blockIdx.x];
  const LdltFront F = fr[c.f];
  const int q = F.fidx, w = block_width(F, st.k);
  const int p = st.p_cur[q], nd = st.ndiag[q];
  float* A = arena + F.off;
  const int64_t ld = F.ld, pm = F.m;
  const int tid = threadIdx.x;
  const float* blk = reinterpret_cast<const float*>(st.blk) + (int64_t)q * BW * LDB;
  // only the tile of the block's own rows reads L (the rest come from apply)
  if (c.local == 0)
    for (int idx = tid; idx < BW * LDB; idx += RT) (&L[0][0])[idx] = blk[idx];
  for (int k = tid; k < 2 * BW; k += RT) dv[k] = st.bdinv[q * 2 * BW + k];
  if (tid < BW) perm[tid] = st.lperm[q * BW + tid];
  __syncthreads();
  // the block's permutation on its rows of the eliminated columns [0, p),
  // shared by the front's CTAs, PU columns in flight per warp (one CTA with
  // one column in flight took most of the diagonal kernel at the top fronts)
  {
    constexpr int PU = 4;
    const int lane = tid & 31, pl = perm[lane];
    if (__any_sync(0xffffffffu, lane < w && pl != lane))
      for (int c0 = (c.local * (RT / 32) + (tid >> 5)) * PU; c0 < p;
           c0 += c.count * (RT / 32) * PU) {
        float v[PU];
#pragma unroll
        for (int u = 0; u < PU; ++u)
          v[u] = (lane < w && c0 + u < p) ? A[(c0 + u) * ld + p + pl] : 0.f;
        __syncwarp();
#pragma unroll
        for (int u = 0; u < PU; ++u)
          if (lane < w && c0 + u < p) A[(c0 + u) * ld + p + lane] = v[u];
      }
  }
  // Column::adjust: drop the first half of a 2x2 pivot split by the test
  int np = min(st.npass_raw[q], nd);
  if (np > 0 && isfinite(dv[2 * (np - 1)]) && dv[2 * (np - 1) + 1] != 0.0) np--;
  if (tid < BW) {
    const int kd = pivot_kind(dv, tid, np);
    kind[tid] = kd;
    if (kd == PV_FIRST || (kd == PV_SECOND && tid < np)) {
      const int k = kd == PV_FIRST ? tid : tid - 1;
      const double a = dv[2 * k], b = dv[2 * k + 1], cc = dv[2 * k + 3];
      const double det = __dsub_rn(mul_(a, cc), mul_(b, b));
      dca[tid] = quot(kd == PV_FIRST ? cc : -b, det);
      dcb[tid] = quot(kd == PV_FIRST ? -b : a, det);
    }
  }
  __syncthreads();
  const float* pan = scratch + F.pan_off;
  float* ldp = scratch + F.ldp_off;
  for (int t0 = p + c.local * RT; t0 < F.m; t0 += c.count * RT) {
    const int r = t0 + tid;
    const bool in_blk = r < p + w;
    const int i = r - p;
    // phase 1: L of the passed columns, the values failed columns keep
    // (in-block rows all belong to the tile that starts at p, so no other
    // CTA writes what this one reads)
    float l[BW];
    if (r < F.m && !in_blk) {
#pragma unroll
      for (int k = 0; k < BW; ++k)
        l[k] = k < np ? pan[k * pm + r] : k < w ? A[(p + perm[k]) * ld + r] : 0.f;
    } else if (r < F.m) {
#pragma unroll
      for (int k = 0; k < BW; ++k) {
        float v = 0.f;
        if (k < np) {
          v = (i > k) ? L[k][i] : (i == k ? 1.f : 0.f);
        } else if (k < w && i >= k) {
          const int ai = perm[i], ak = perm[k];
          v = A[(p + min(ai, ak)) * ld + p + max(ai, ak)];
        }
        l[k] = v;
      }
    }
    __syncthreads();
    if (r < F.m) {
#pragma unroll
      for (int k = 0; k < BW; ++k)
        if (k < w && !(in_blk && i < k)) A[(p + k) * ld + r] = l[k];
      if (r >= p + np) {
#pragma unroll
        for (int k = 0; k < BW; ++k) {
          if (k >= np) break;
          const int kd = kind[k];
          float v = 0.f;
          if (kd == PV_ONE) {
            v = l[k] / (float)dv[2 * k];
          } else if (kd == PV_FIRST) {
            if (k + 1 < BW) v = (float)fma_((double)l[k], dca[k], mul_((double)l[k + 1], dcb[k]));
          } else if (kd == PV_SECOND) {
            if (k > 0) v = (float)fma_((double)l[k - 1], dca[k], mul_((double)l[k], dcb[k]));
          }
          ldp[k * pm + r] = v;
        }
      }
    }
    __syncthreads();
  }
  if (c.local == 0) {
    for (int k = tid; k < 2 * np; k += RT) st.dall[F.d_off + 2 * p + k] = dv[k];
    if (tid == 0) {
      const int nf = st.nf_cur[q];
      st.npass[q] = np;
      st.p_next[q] = p + np;
      st.nf_next[q] = nf + (w - np);
      if (st.k == F.nblk - 1) st.p_final[q] = p + np;
    }
  }
}

// The same for FP64, four lanes per row as in k_app_apply64 (a row's 32 FP64
// divisions were half of the launch): 22 -> 13 us per launch on the 14^3 saddle
// point.
__global__ void __launch_bounds__(T4) k_app_commit64(double* __restrict__ arena,
                                                     double* __restrict__ scratch,
                                                     const LdltFront* __restrict__ fr,
                                                     const CtaMap* __restrict__ cm, LdltStep st) {
  __shared__ double L[BW][LDB];
  __shared__ double dv[2 * BW];
  __shared__ double dca[BW], dcb[BW];  // D of a 2x2 pair's two columns
  __shared__ int perm[BW], kind[BW];
  __shared__ int has2;
  const CtaMap c = cm[blockIdx.x];
  const LdltFront F = fr[c.f];
  const int q = F.fidx, w = block_width(F, st.k);
  const int p = st.p_cur[q], nd = st.ndiag[q];
  double* A = arena + F.off;
  const int64_t ld = F.ld, pm = F.m;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rl = lane % RW4, cg = lane / RW4;
  const double* blk = st.blk + (int64_t)q * BW * LDB;
  // only the tile of the block's own rows reads L (the rest come from apply)
  if (c.local == 0)
    for (int idx = tid; idx < BW * LDB; idx += T4) (&L[0][0])[idx] = blk[idx];
  if (tid < 2 * BW) dv[tid] = st.bdinv[q * 2 * BW + tid];
  if (tid < BW) perm[tid] = st.lperm[q * BW + tid];
  __syncthreads();
  // the block's permutation on its rows of the eliminated columns [0, p)
  {
    constexpr int PU = 4;
    const int pl = perm[lane];
    if (__any_sync(0xffffffffu, lane < w && pl != lane))
      for (int c0 = (c.local * (T4 / 32) + warp) * PU; c0 < p; c0 += c.count * (T4 / 32) * PU) {
        double v[PU];
#pragma unroll
        for (int u = 0; u < PU; ++u)
          v[u] = (lane < w && c0 + u < p) ? A[(c0 + u) * ld + p + pl] : 0.0;
        __syncwarp();
#pragma unroll
        for (int u = 0; u < PU; ++u)
          if (lane < w && c0 + u < p) A[(c0 + u) * ld + p + lane] = v[u];
      }
  }
  // Column::adjust: drop the first half of a 2x2 pivot split by the test
  int np = min(st.npass_raw[q], nd);
  if (np > 0 && isfinite(dv[2 * (np - 1)]) && dv[2 * (np - 1) + 1] != 0.0) np--;
  if (tid < BW) {
    const int kd = pivot_kind(dv, tid, np);
    kind[tid] = kd;
    if (kd == PV_FIRST || (kd == PV_SECOND && tid < np)) {
      const int k = kd == PV_FIRST ? tid : tid - 1;
      const double a = dv[2 * k], b = dv[2 * k + 1], cc = dv[2 * k + 3];
      const double det = __dsub_rn(mul_(a, cc), mul_(b, b));
      dca[tid] = quot(kd == PV_FIRST ? cc : -b, det);
      dcb[tid] = quot(kd == PV_FIRST ? -b : a, det);
    }
    const unsigned two = __ballot_sync(0xffffffffu, kd == PV_FIRST || kd == PV_SECOND);
    if (tid == 0) has2 = two != 0;
  }
  __syncthreads();
  const double* pan = scratch + F.pan_off;
  double* ldp = scratch + F.ldp_off;
  for (int t0 = p + c.local * R4; t0 < F.m; t0 += c.count * R4) {
    const int r = t0 + warp * RW4 + rl;
    const bool has = r < F.m, in_blk = r < p + w;
    const int i = r - p;
    // phase 1: L of the passed columns, the values failed columns keep
    // (in-block rows all belong to the tile that starts at p, so no other
    // CTA writes what this one reads)
    double l[NC4];
#pragma unroll
    for (int u = 0; u < NC4; ++u) {
      const int k = 4 * u + cg;
      double v = 0.0;
      if (has && !in_blk) {
        v = k < np ? pan[k * pm + r] : k < w ? A[(p + perm[k]) * ld + r] : 0.0;
      } else if (has) {
        if (k < np) {
          v = (i > k) ? L[k][i] : (i == k ? 1.0 : 0.0);
        } else if (k < w && i >= k) {
          const int ai = perm[i], ak = perm[k];
          v = A[(p + min(ai, ak)) * ld + p + max(ai, ak)];
        }
      }
      l[u] = v;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < NC4; ++u) {
      const int k = 4 * u + cg;
      double lp = 0.0, ln = 0.0;
      if (has2) neighbours4(l, u, rl, cg, lp, ln);
      if (!has) continue;
      if (k < w && !(in_blk && i < k)) A[(p + k) * ld + r] = l[u];
      if (r >= p + np && k < np) {
        const int kd = kind[k];
        double v = 0.0;
        if (kd == PV_ONE) {
          v = l[u] / dv[2 * k];
        } else if (kd == PV_FIRST) {
          if (k + 1 < BW) v = fma_(l[u], dca[k], mul_(ln, dcb[k]));
        } else if (kd == PV_SECOND) {
          if (k > 0) v = fma_(lp, dca[k], mul_(l[u], dcb[k]));
        }
        ldp[k * pm + r] = v;
      }
    }
    __syncthreads();
  }
  if (c.local == 0) {
    for (int k = tid; k < 2 * np; k += T4) st.dall[F.d_off + 2 * p + k] = dv[k];
    if (tid == 0) {
      const int nf = st.nf_cur[q];
      st.npass[q] = np;
      st.p_next[q] = p + np;
      st.nf_next[q] = nf + (w - np);
      if (st.k == F.nblk - 1) st.p_final[q] = p + np;
    }
  }
}

// ---------------------------------------------------------------------------
// Move the f = w - npass failed columns of step k (now at [a, a + f),
// a = p + npass) behind the others: positions [a, n) take the variables in
// the order [a + f, n) then [a, a + f).  Copy rows [a, m) of columns [0, n)
// (lower part) and the variable list out, then write them back permuted.
__device__ __forceinline__ int moved_from(int i, int a, int n, int f) {
  return i < n - f ? i + f : a + (i - (n - f));
}

template <typename T>
__global__ void __launch_bounds__(256) k_app_move_copy(const T* __restrict__ arena,
                                                       T* __restrict__ scratch,
                                                       const LdltFront* __restrict__ fr,
                                                       const CtaMap* __restrict__ cm,
                                                       LdltStep st) {
  const CtaMap c = cm[blockIdx.x];
  const LdltFront F = fr[c.f];
  const int q = F.fidx, w = block_width(F, st.k), np = st.npass[q], f = w - np;
  if (f == 0) return;
  const int a = st.p_cur[q] + np, n = F.n, m = F.m, mm = m - a;
  const T* A = arena + F.off;
  T* mv = scratch + F.mv_off;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int col = c.local * 8 + warp; col < n; col += c.count * 8)
    for (int r = max(a, col) + lane; r < m; r += 32)
      mv[(int64_t)col * mm + (r - a)] = A[(int64_t)col * F.ld + r];
  if (c.local == 0)
    for (int i = a + threadIdx.x; i < n; i += blockDim.x)
      st.mvvar[F.mvvar_off + i] = st.var[F.var_off + i];
}

template <typename T>
__global__ void __launch_bounds__(256) k_app_move_write(T* __restrict__ arena,
                                                        const T* __restrict__ scratch,
                                                        const LdltFront* __restrict__ fr,
                                                        const CtaMap* __restrict__ cm,
                                                        LdltStep st) {
  const CtaMap c = cm[blockIdx.x];
  const LdltFront F = fr[c.f];
  const int q = F.fidx, w = block_width(F, st.k), np = st.npass[q], f = w - np;
  if (f == 0) return;
  const int a = st.p_cur[q] + np, n = F.n, m = F.m, mm = m - a;
  T* A = arena + F.off;
  const T* mv = scratch + F.mv_off;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int col = c.local * 8 + warp; col < n; col += c.count * 8) {
    if (col < a) {
      // eliminated column: permute its rows [a, n)
      for (int r = a + lane; r < n; r += 32)
        A[(int64_t)col * F.ld + r] = mv[(int64_t)col * mm + (moved_from(r, a, n, f) - a)];
    } else {
      const int oc = moved_from(col, a, n, f);
      for (int r = col + lane; r < m; r += 32) {
        T v;
        if (r < n) {
          const int orr = moved_from(r, a, n, f);
          const int hi = max(orr, oc), lo = min(orr, oc);
          v = mv[(int64_t)lo * mm + (hi - a)];
        } else {
          v = mv[(int64_t)oc * mm + (r - a)];
        }
        A[(int64_t)col * F.ld + r] = v;
      }
    }
  }
  if (c.local == 0)
    for (int i = a + threadIdx.x; i < n; i += blockDim.x)
      st.var[F.var_off + i] = st.mvvar[F.mvvar_off + moved_from(i, a, n, f)];
}

// ---------------------------------------------------------------------------
// Trailing update of step k: rows [o, m) x columns [o, n), o = p + npass,
// lower part, C -= (L D) L^T over the npass passed columns.  Lower-triangular
// tile space enumerated column by column; CTAs stride over it.
template <typename T, int TM, int KT>
__global__ void __launch_bounds__(256) k_app_update(T* __restrict__ arena,
                                                    const T* __restrict__ scratch,
                                                    const LdltFront* __restrict__ fr,
                                                    const CtaMap* __restrict__ cm,
                                                    LdltStep st) {
  __shared__ __align__(16) T As[2][KT][TM];
  __shared__ __align__(16) T Bs[2][KT][TM];
  const CtaMap c = cm[blockIdx.x];
  const LdltFront F = fr[c.f];
  const int q = F.fidx, p = st.p_cur[q], np = st.npass[q];
  if (np == 0) return;
  const int o = p + np;
  if (o >= F.n) return;
  const int R = (F.m - o + TM - 1) / TM, C = (F.n - o + TM - 1) / TM;
  const int total = C * R - C * (C - 1) / 2;
  T* front = arena + F.off;
  for (int t = c.local; t < total; t += c.count) {
    int cj = 0, rem = t;
    while (rem >= R - cj) { rem -= R - cj; ++cj; }
    const int ri = cj + rem;
    tile_update_body<T, TM, TM, KT>(front, F.ld, scratch + F.ldp_off, F.m,
                                    front + (int64_t)p * F.ld, F.ld, o + ri * TM, o + cj * TM,
                                    F.m, F.n, 0, np, As, Bs);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Threshold partial pivoting over columns [pstart, n), one CTA per front,
// right-looking updates restricted to the candidate columns (all rows).
template <typename T>
__global__ void __launch_bounds__(256) k_ldlt_tpp(T* __restrict__ arena,
                                                  const LdltFront* __restrict__ fr,
                                                  LdltStep st, double u,
                                                  const int* __restrict__ pstart,
                                                  int* __restrict__ out_nelim) {
  const LdltFront F = fr[blockIdx.x];
  T* A = arena + F.off;
  const int ld = F.ld, m = F.m, n = F.n;
  int* var = st.var + F.var_off;
  double* D = st.dall + F.d_off;
  const int tid = threadIdx.x, nt = blockDim.x;
  __shared__ double rv[8];
  __shared__ int ri[8];
  auto at = [&](int r, int c) -> T& { return A[(int64_t)c * ld + r]; };
  auto sym = [&](int r, int c) -> double { return r >= c ? (double)at(r, c) : (double)at(c, r); };
  auto swap_xy = [&](int x, int y) {
    if (x == y) return;
    if (x > y) { int t = x; x = y; y = t; }
    for (int k = tid; k < m; k += nt) {
      if (k < x) { T t = at(x, k); at(x, k) = at(y, k); at(y, k) = t; }
      else if (k == x) { T t = at(x, x); at(x, x) = at(y, y); at(y, y) = t; }
      else if (k < y) { T t = at(k, x); at(k, x) = at(y, k); at(y, k) = t; }
      else if (k > y) { T t = at(k, x); at(k, x) = at(k, y); at(k, y) = t; }
    }
    if (tid == 0) { int t = var[x]; var[x] = var[y]; var[y] = t; }
    __syncthreads();
  };
  // block max of |col c| over rows [lo, m) excluding ex1, ex2 (first maximum)
  auto colmax = [&](int c, int lo, int ex1, int ex2, int& arg) -> double {
    double b = -1.0;
    int bi = -1;
    for (int r = lo + tid; r < m; r += nt) {
      if (r == ex1 || r == ex2) continue;
      double v = fabs(sym(r, c));
      if (v > b) { b = v; bi = r; }
    }
    warp_argmax(b, bi);
    if ((tid & 31) == 0) { rv[tid >> 5] = b; ri[tid >> 5] = bi; }
    __syncthreads();
    if (tid == 0) {
      for (int qq = 1; qq < nt / 32; ++qq)
        if (rv[qq] > rv[0] || (rv[qq] == rv[0] && ri[qq] >= 0 && (ri[0] < 0 || ri[qq] < ri[0]))) {
          rv[0] = rv[qq]; ri[0] = ri[qq];
        }
    }
    __syncthreads();
    double res = rv[0];
    arg = ri[0];
    __syncthreads();
    return fmax(res, 0.0);
  };
  const double lim = quot(1.0, u);
  int ne = pstart[F.fidx];
  while (ne < n) {
    int decided = 0, piv = -1, tpiv = -1;
    for (int c = ne; c < n && !decided; ++c) {
      int t;
      double amax = colmax(c, ne, c, -1, t);
      double acc = fabs(sym(c, c));
      if (amax < st.small && acc < st.small) { decided = 3; piv = c; break; }
      if (acc >= mul_(u, amax)) { decided = 1; piv = c; break; }
      if (t >= 0 && t < n) {
        int dummy;
        double ap2 = colmax(c, ne, c, t, dummy);
        double at2 = colmax(t, ne, c, t, dummy);
        double a11 = sym(c, c), a22 = sym(t, t), a21 = sym(t, c);
        double det = __dsub_rn(mul_(a11, a22), mul_(a21, a21));
        if (fabs(det) > st.small && isfinite(det)) {
          double i11 = quot(a22, det), i12 = quot(-a21, det), i22 = quot(a11, det);
          if (fma_(fabs(i11), ap2, mul_(fabs(i12), at2)) <= lim &&
              fma_(fabs(i12), ap2, mul_(fabs(i22), at2)) <= lim) {
            decided = 2; piv = c; tpiv = t;
          }
        }
      }
    }
    if (!decided) break;
    if (decided == 3) {
      if (!st.action) {
        if (tid == 0) atomicOr(st.status, ST_SINGULAR);
        break;
      }
      swap_xy(ne, piv);
      for (int r = ne + tid; r < m; r += nt) at(r, ne) = T(r == ne ? 1 : 0);
      if (tid == 0) {
        D[2 * ne] = 0.0;
        D[2 * ne + 1] = 0.0;
        atomicOr(st.status, ST_ZERO_PIVOT);
      }
      __syncthreads();
      ne += 1;
    } else if (decided == 1) {
      swap_xy(ne, piv);
      const int k = ne;
      const double di = quot(1.0, (double)at(k, k));
      const int wdt = n - k - 1;
      for (int e = tid; e < wdt * (m - k - 1); e += nt) {
        int j = k + 1 + e % wdt, rr = k + 1 + e / wdt;
        if (rr >= j)
          at(rr, j) = (T)fma_(-(double)at(rr, k), mul_((double)at(j, k), di), (double)at(rr, j));
      }
      __syncthreads();
      for (int rr = k + 1 + tid; rr < m; rr += nt) at(rr, k) = (T)mul_((double)at(rr, k), di);
      if (tid == 0) {
        at(k, k) = T(1);
        D[2 * k] = di;
        D[2 * k + 1] = 0.0;
      }
      __syncthreads();
      ne += 1;
    } else {
      const int k = ne;
      swap_xy(k, piv);
      swap_xy(k + 1, (tpiv == k) ? piv : tpiv);
      const double a11 = at(k, k), a21 = at(k + 1, k), a22 = at(k + 1, k + 1);
      const double det = __dsub_rn(mul_(a11, a22), mul_(a21, a21));
      const double i11 = quot(a22, det), i12 = quot(-a21, det), i22 = quot(a11, det);
      const int wdt = n - k - 2;
      for (int e = tid; wdt > 0 && e < wdt * (m - k - 2); e += nt) {
        int j = k + 2 + e % wdt, rr = k + 2 + e / wdt;
        if (rr >= j) {
          const double w1 = at(j, k), w2 = at(j, k + 1);
          const double l1 = fma_(i11, w1, mul_(i12, w2)), l2 = fma_(i12, w1, mul_(i22, w2));
          at(rr, j) = (T)fma_(-(double)at(rr, k + 1), l2,
                              fma_(-(double)at(rr, k), l1, (double)at(rr, j)));
        }
      }
      __syncthreads();
      for (int rr = k + 2 + tid; rr < m; rr += nt) {
        const double w1 = at(rr, k), w2 = at(rr, k + 1);
        at(rr, k) = (T)fma_(i11, w1, mul_(i12, w2));
        at(rr, k + 1) = (T)fma_(i12, w1, mul_(i22, w2));
      }
      if (tid == 0) {
        at(k, k) = T(1);
        at(k + 1, k) = T(0);
        at(k + 1, k + 1) = T(1);
        D[2 * k] = i11;
        D[2 * k + 1] = i12;
        D[2 * k + 2] = dinf();
        D[2 * k + 3] = i22;
      }
      __syncthreads();
      ne += 2;
    }
  }
  if (tid == 0) out_nelim[F.fidx] = ne;
}

// ---------------------------------------------------------------------------
// L*D of contribution rows [n, m) over columns [0, nelim) (F.p = nelim).
// A slice's CTAs stride over tiles of LDLT_RT rows x CLD columns, one row per
// thread, a tile's loads all in flight.  Bound by the latency of a tile's batches,
// one after another: on the 14^3 saddle point (FP64) 51 us per launch with all
// nelim columns on the thread of a row, 28 us in tiles of 32 columns, 11 us in
// tiles of 8.
constexpr int CLD = LDLT_CLD, CLD_U = 8;
template <typename T>
__global__ void __launch_bounds__(LDLT_RT) k_ldlt_calc_ld(const T* __restrict__ arena,
                                                         T* __restrict__ scratch,
                                                         const LdltFront* __restrict__ fr,
                                                         const CtaMap* __restrict__ cm,
                                                         LdltStep st) {
  // column k: 0 divide by ca, 1 first of a 2x2 pair (l_k ca + l_k+1 cb),
  // 2 second of a pair (l_k-1 ca + l_k cb), 3 zero pivot
  __shared__ int kind[CLD];
  __shared__ double ca[CLD], cb[CLD];
  const CtaMap c = cm[blockIdx.x];
  const LdltFront F = fr[c.f];
  const T* A = arena + F.off;
  const double* D = st.dall + F.d_off;
  T* out = scratch + F.ldp_off;
  const int ne = F.p, tid = threadIdx.x;
  const int64_t ldo = F.m, ld = F.ld;
  const int nr = (F.m - F.n + LDLT_RT - 1) / LDLT_RT, nc = (ne + CLD - 1) / CLD;
  for (int t = c.local; t < nr * nc; t += c.count) {
    const int k0 = t / nr * CLD, kw = min(CLD, ne - k0);
    const int r = F.n + t % nr * LDLT_RT + tid;
    __syncthreads();
    if (tid < kw) {
      const int k = k0 + tid;
      const bool second = k > 0 && isinf(D[2 * k]);
      if (second || (k + 1 < ne && isinf(D[2 * k + 2]))) {
        const int p = second ? k - 1 : k;
        const double a = D[2 * p], b = D[2 * p + 1], cc = D[2 * p + 3];
        const double det = __dsub_rn(mul_(a, cc), mul_(b, b));
        kind[tid] = second ? 2 : 1;
        ca[tid] = quot(second ? -b : cc, det);
        cb[tid] = quot(second ? a : -b, det);
      } else {
        kind[tid] = D[2 * k] == 0.0 ? 3 : 0;
        ca[tid] = D[2 * k];
      }
    }
    __syncthreads();
    if (r >= F.m) continue;
    for (int j0 = 0; j0 < kw; j0 += CLD_U) {
      // l[u] = L(r, k0 + j0 + u - 1): one column more on either side, for pairs
      T l[CLD_U + 2];
#pragma unroll
      for (int u = 0; u < CLD_U + 2; ++u) {
        const int k = k0 + j0 + u - 1;
        l[u] = (k >= 0 && k < ne) ? A[k * ld + r] : T(0);
      }
#pragma unroll
      for (int u = 0; u < CLD_U; ++u) {
        const int j = j0 + u;
        if (j >= kw) break;
        const int kd = kind[j];
        T v = T(0);
        if (kd == 0) v = l[u + 1] / (T)ca[j];
        else if (kd == 1) v = (T)fma_((double)l[u + 1], ca[j], mul_((double)l[u + 2], cb[j]));
        else if (kd == 2) v = (T)fma_((double)l[u], ca[j], mul_((double)l[u + 1], cb[j]));
        out[(k0 + j) * ldo + r] = v;
      }
    }
  }
}

template <typename ACC>
__global__ void k_solve_diag(const FrontDesc* __restrict__ fr, const int* __restrict__ var,
                             const double* __restrict__ dall, const int64_t* __restrict__ d_off,
                             ACC* __restrict__ x, int n, int nrhs) {
  const FrontDesc f = fr[blockIdx.x];
  const double* D = dall + d_off[blockIdx.x];
  const int* v = var + f.rl;
  const int ne = f.n;
  for (int e = threadIdx.x; e < ne * nrhs; e += blockDim.x) {
    int k = e % ne, r = e / ne;
    ACC* xr = x + (int64_t)r * n;
    bool second = k > 0 && isinf(D[2 * k]);  // (k-1, k) is a 2x2 pair
    if (second) continue;
    if (k + 1 < ne && isinf(D[2 * k + 2])) {
      double a = xr[v[k]], b = xr[v[k + 1]];
      xr[v[k]] = (ACC)fma_(D[2 * k], a, mul_(D[2 * k + 1], b));
      xr[v[k + 1]] = (ACC)fma_(D[2 * k + 1], a, mul_(D[2 * k + 3], b));
    } else {
      xr[v[k]] = (ACC)mul_(D[2 * k], (double)xr[v[k]]);
    }
  }
}

}  // namespace

template <typename T>
void launch_app_diag(T* arena, T* scratch, const LdltFront* fr, const CtaMap* cm, int ncta,
                     LdltStep st, cudaStream_t s) {
  if (ncta > 0) k_app_diag<T><<<ncta, DG_T, 0, s>>>(arena, scratch, fr, cm, st);
}
template <typename T>
void launch_app_apply(const T* arena, T* scratch, const LdltFront* fr, const CtaMap* cm, int ncta,
                      LdltStep st, cudaStream_t s) {
  if (ncta <= 0) return;
  if constexpr (sizeof(T) == 8) k_app_apply64<<<ncta, T4, 0, s>>>(arena, scratch, fr, cm, st);
  else k_app_apply32<<<ncta, AppRows<T>::v, 0, s>>>(arena, scratch, fr, cm, st);
}
template <typename T>
void launch_app_commit(T* arena, T* scratch, const LdltFront* fr, const CtaMap* cm, int ncta,
                       LdltStep st, cudaStream_t s) {
  if (ncta <= 0) return;
  if constexpr (sizeof(T) == 8) k_app_commit64<<<ncta, T4, 0, s>>>(arena, scratch, fr, cm, st);
  else k_app_commit32<<<ncta, AppRows<T>::v, 0, s>>>(arena, scratch, fr, cm, st);
}
template <typename T>
void launch_app_move(T* arena, T* scratch, const LdltFront* fr, const CtaMap* cm, int ncta,
                     LdltStep st, cudaStream_t s) {
  if (ncta <= 0) return;
  k_app_move_copy<T><<<ncta, 256, 0, s>>>(arena, scratch, fr, cm, st);
  k_app_move_write<T><<<ncta, 256, 0, s>>>(arena, scratch, fr, cm, st);
}
template <typename T>
void launch_app_update(T* arena, const T* scratch, const LdltFront* fr, const CtaMap* cm,
                       int ncta, LdltStep st, cudaStream_t s) {
  if (ncta > 0)
    k_app_update<T, AppTile<T>::v, 16><<<ncta, 256, 0, s>>>(arena, scratch, fr, cm, st);
}
template <typename T>
void launch_ldlt_tpp(T* arena, const LdltFront* fr, int nf, LdltStep st, double u_eff,
                     const int* pstart, int* out_nelim, cudaStream_t s) {
  if (nf > 0) k_ldlt_tpp<T><<<nf, 256, 0, s>>>(arena, fr, st, u_eff, pstart, out_nelim);
}
template <typename T>
void launch_ldlt_calc_ld(const T* arena, T* scratch, const LdltFront* fr, const CtaMap* cm,
                         int ncta, LdltStep st, cudaStream_t s) {
  if (ncta > 0) k_ldlt_calc_ld<T><<<ncta, LDLT_RT, 0, s>>>(arena, scratch, fr, cm, st);
}
template <typename ACC>
void launch_solve_diag(const FrontDesc* fr, int nf, const int* var, const double* dall,
                       const int64_t* d_off, ACC* x, int n, int nrhs, cudaStream_t s) {
  if (nf > 0) k_solve_diag<ACC><<<nf, 256, 0, s>>>(fr, var, dall, d_off, x, n, nrhs);
}

#define SG_INST(T)                                                                            \
  template void launch_app_diag<T>(T*, T*, const LdltFront*, const CtaMap*, int, LdltStep,     \
                                   cudaStream_t);                                             \
  template void launch_app_apply<T>(const T*, T*, const LdltFront*, const CtaMap*, int,        \
                                    LdltStep, cudaStream_t);                                  \
  template void launch_app_commit<T>(T*, T*, const LdltFront*, const CtaMap*, int, LdltStep,   \
                                     cudaStream_t);                                           \
  template void launch_app_move<T>(T*, T*, const LdltFront*, const CtaMap*, int, LdltStep,     \
                                   cudaStream_t);                                             \
  template void launch_app_update<T>(T*, const T*, const LdltFront*, const CtaMap*, int,       \
                                     LdltStep, cudaStream_t);                                 \
  template void launch_ldlt_tpp<T>(T*, const LdltFront*, int, LdltStep, double, const int*,    \
                                   int*, cudaStream_t);                                       \
  template void launch_ldlt_calc_ld<T>(const T*, T*, const LdltFront*, const CtaMap*, int,     \
                                       LdltStep, cudaStream_t);                               \
  template void launch_solve_diag<T>(const FrontDesc*, int, const int*, const double*,         \
                                     const int64_t*, T*, int, int, cudaStream_t);
SG_INST(float)
SG_INST(double)
#undef SG_INST

}  // namespace sylver_gb300
