// Panel step of FP64 fronts in one launch: Cholesky of the panel's diagonal
// block (at most 32 x 32), the triangular solve of the rows below it, and the
// digits of those rows for the tensor-core update of the group's other columns.
//
// Bound by the FP64 pipe (two multiply-adds per clock and SM) and by the chain
// of 32 pivots.  Every CTA factorises the diagonal block for itself, which
// costs no more than half of its own rows' solve and saves a launch and a
// round trip through memory per step; pivots take 1/sqrt from an FP32
// estimate and one cubic step instead of an IEEE square root and division, which
// ran on every thread of the block before.  A panel takes at least 18 us with 16 rows
// a CTA and 24 us with 32: 29,000 clocks for the block (32 pivots of about 600 with
// their updates of the block of four, eight updates of 1,200 behind it) and 9,400 or
// 15,700 for the rows' substitution; a launch of 1500 panels' blocks on 33x29x31
// was 69 us with a kernel each for block and rows.  33x29x31: 6.8 ms of
// block and row kernels -> 2.3 ms; 56^3: 24 ms -> 11.1 ms.
//
// Reference behaviour replaced: factorize_diag_block, solve_block
// (src/kernels/factor.hxx:56-160).
#include "digits.cuh"
#include "pivot.cuh"

namespace sylver_gb300 {

namespace {

constexpr int PB = 32;         // panel width
constexpr int PLD = PB + 1;
constexpr int P64_THREADS = 128;

// One CTA of four warps: rows [r0, r1) of a panel.
//   diagonal block: in blocks of four columns; one warp, a row per lane,
//     factorises the block's columns in registers (its pivots reach the other
//     lanes by shuffles, no barrier), then all threads apply it to the triangle
//     behind it, an entry per thread;
//   rows: NG lanes per row, lane group c holding columns c, c + NG, ...; the
//     substitution runs on unscaled values z_j = x_j L(j, j) with
//     L(i, j) / L(j, j) prepared in shared memory, so each of its steps is one
//     shuffle and one multiply-add deep.
// Loops are unrolled only where registers must be indexed: a panel runs each
// instruction a few times, and fetching 30 KB of code took longer than that.
template <int NG>
__global__ void __launch_bounds__(P64_THREADS)
    k_panel64(double* __restrict__ arena, const P64Task* __restrict__ tasks,
              double* __restrict__ dstore, uint16_t* __restrict__ planes, int64_t pstride,
              int pitch, int* __restrict__ sexp, unsigned* __restrict__ status) {
  constexpr int CB = 4;               // columns of a diagonal sub-block
  constexpr int RW = 32 / NG;         // rows per warp
  constexpr int RC = 4 * RW;          // rows per tile of the CTA
  constexpr int NC = PB / NG;         // columns per lane
  __shared__ double Ls[PB * PLD];     // Ls[k * PLD + i] = L(i, k), then L(i, k) / L(k, k)
  __shared__ double ds[PB], rinv[PB];
  __shared__ long long F[RC][PB + 1];  // rows to cut into digits
  __shared__ int es[RC];               // and their scale exponents
  const P64Task t = tasks[blockIdx.x];
  double* a = arena + t.off;
  const int64_t ld = t.ld;
  const int k0 = t.k0, w = t.w, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // this CTA's first rows, in flight during the diagonal block
  const int rl = lane % RW, cg = lane / RW;
  const int tr = warp * RW + rl;
  double v[NC];
  auto load_rows = [&](int r0) {
#pragma unroll
    for (int u = 0; u < NC; ++u) {
      const int j = NG * u + cg;
      v[u] = (r0 + tr < t.r1 && j < w) ? a[(int64_t)(k0 + j) * ld + r0 + tr] : 0.0;
    }
  };
  // rows and columns beyond the panel's width: identity
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int j = 4 * u + warp;
    Ls[j * PLD + lane] = (lane < w && j <= lane) ? a[(int64_t)(k0 + j) * ld + k0 + lane]
                                                 : (j == lane ? 1.0 : 0.0);
  }
  load_rows(t.r0);
  __syncthreads();
  bool bad = false;
#pragma unroll 1
  for (int b = 0; b < PB; b += CB) {
    // (another scheduler's FP64 pipe in each of the CTAs that share an SM)
    if (warp == ((b / CB + blockIdx.x / NUM_SMS) & 3)) {
      double c[CB];
#pragma unroll
      for (int u = 0; u < CB; ++u) c[u] = Ls[(b + u) * PLD + lane];
#pragma unroll
      for (int k = 0; k < CB; ++k) {
        double d = __shfl_sync(0xffffffffu, c[k], b + k);
        if (!(d > 0.0)) {
          bad = true;
          d = 1.0;
        }
        const double r = rsqrt64(d);
        const double l = lane > b + k ? c[k] * r : 0.0;
        c[k] = l;
        if (lane == 0) {
          ds[b + k] = d;
          rinv[b + k] = r;
        }
#pragma unroll
        for (int u = k + 1; u < CB; ++u)
          c[u] = fma(-l, __shfl_sync(0xffffffffu, l, b + u), c[u]);
      }
#pragma unroll
      for (int u = 0; u < CB; ++u) Ls[(b + u) * PLD + lane] = c[u];
    }
    __syncthreads();
    const int o = b + CB, T = PB - o;
#pragma unroll 1
    for (int x = tid; x < T * (T + 1) / 2; x += P64_THREADS) {
      // x-th entry (i, j), i >= j, of the triangle by rows
      int i = (int)((sqrtf(8.f * (float)x + 1.f) - 1.f) * 0.5f);
      if (i * (i + 1) / 2 > x) --i;
      else if ((i + 1) * (i + 2) / 2 <= x) ++i;
      const int j = x - i * (i + 1) / 2;
      double s = Ls[(o + j) * PLD + o + i];
#pragma unroll
      for (int k = 0; k < CB; ++k)
        s = fma(-Ls[(b + k) * PLD + o + i], Ls[(b + k) * PLD + o + j], s);
      Ls[(o + j) * PLD + o + i] = s;
    }
    __syncthreads();
  }
  if (t.didx >= 0) {
    if (bad && lane == 0) atomicOr(status, ST_NOT_POSDEF);
    double* o = dstore + (int64_t)t.didx * (PB * PB);
#pragma unroll 1
    for (int j = warp; j < PB; j += 4)
      if (lane > j) o[j * PB + lane] = Ls[j * PLD + lane];
    if (warp == 0) o[lane * PB + lane] = sqrt(ds[lane]);
    __syncthreads();
  }
  if (t.r0 >= t.r1) return;
  // Ls(i, k) <- L(i, k) / L(k, k)
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int j = 4 * u + warp;
    Ls[j * PLD + lane] *= rinv[j];
  }
  __syncthreads();
#pragma unroll 1
  for (int r0 = t.r0; r0 < t.r1; r0 += RC) {
    const int row = r0 + tr;
    const bool has = row < t.r1;
    if (r0 > t.r0) load_rows(r0);
#pragma unroll
    for (int u0 = 0; u0 < NC; ++u0) {
#pragma unroll 1
      for (int jj = 0; jj < NG; ++jj) {
        const double z = __shfl_sync(0xffffffffu, v[u0], rl + jj * RW);
        const double* lj = Ls + (NG * u0 + jj) * PLD + cg;
        if (cg > jj) v[u0] = fma(-z, lj[NG * u0], v[u0]);
#pragma unroll
        for (int u = u0 + 1; u < NC; ++u) v[u] = fma(-z, lj[NG * u], v[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < NC; ++u) {
      const int j = NG * u + cg;
      v[u] *= rinv[j];
      if (has && j < w) a[(int64_t)(k0 + j) * ld + row] = v[u];
    }
    if (t.base < 0) continue;
    // digits of the rows just solved, for the update by this panel
    int e = OZ_EMPTY;
    float s = 0.f;
    bool nf = false;
#pragma unroll
    for (int u = 0; u < NC; ++u) norm_add(e, s, __double_as_longlong(v[u]), nf);
#pragma unroll
    for (int o = RW; o < 32; o += o) {
      norm_merge(e, s, __shfl_xor_sync(0xffffffffu, e, o), __shfl_xor_sync(0xffffffffu, s, o));
      nf = __shfl_xor_sync(0xffffffffu, (int)nf, o) || nf;
    }
    e = nf ? OZ_NONFINITE : norm_exponent(e, s);
    const int64_t srow = (int64_t)t.base + (r0 - t.r0);
    if (cg == 0) es[tr] = e;
    if (cg == 0 && has) sexp[srow + tr] = e;
#pragma unroll
    for (int u = 0; u < NC; ++u) F[tr][NG * u + cg] = __double_as_longlong(v[u]);
    __syncthreads();
#pragma unroll 1
    for (int rr = tid >> 4; rr < RC; rr += 8) {
      const int k = 2 * (tid & 15);
      if (r0 + rr < t.r1)
        store_digits(F[rr][k], F[rr][k + 1], es[rr], planes + (srow + rr) * pitch + k, pstride);
    }
    __syncthreads();
  }
}

// The level's diagonal blocks into the fronts (the panel kernel's CTAs all
// read the assembled block, so none may overwrite it).
__global__ void __launch_bounds__(256) k_diag_store64(double* __restrict__ arena,
                                                      const P64Task* __restrict__ tasks,
                                                      const double* __restrict__ dstore) {
  const P64Task t = tasks[blockIdx.x];
  const double* o = dstore + (int64_t)t.didx * (PB * PB);
  const int lane = threadIdx.x & 31;
  for (int j = threadIdx.x >> 5; j < t.w; j += 8)
    if (lane >= j && lane < t.w)
      arena[t.off + (int64_t)(t.k0 + j) * t.ld + t.k0 + lane] = o[j * PB + lane];
}

}  // namespace

void launch_panel64(double* arena, const P64Task* t, int ntask, int rows, double* dstore,
                    uint16_t* planes, int64_t pstride, int pitch, int* sexp, unsigned* status,
                    cudaStream_t s) {
  if (ntask <= 0) return;
  auto kern = rows <= 16 ? k_panel64<8> : k_panel64<4>;
  kern<<<ntask, P64_THREADS, 0, s>>>(arena, t, dstore, planes, pstride, pitch, sexp, status);
}

void launch_diag_store64(double* arena, const P64Task* t, int ntask, const double* dstore,
                         cudaStream_t s) {
  if (ntask <= 0) return;
  k_diag_store64<<<ntask, 256, 0, s>>>(arena, t, dstore);
}

}  // namespace sylver_gb300
