// Self-check of the tensor-core contribution-block update: a synthetic front
// (m = k + rows, ld = m) with random L21 and a zero contribution block goes
// through the same split + TMA + tcgen05 path the factorization uses; the
// result is compared with -L21 L21^T formed in FP64 on the host.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "../../include/sylver_gb300.h"
#include "numeric.hpp"
#include "tc.hpp"

using namespace sylver_gb300;

extern "C" int sylver_gb300_tc_selfcheck(int rows, int k, double* max_rel_err) {
  if (rows < 1 || k < 1 || !max_rel_err) return SYLVER_ERROR_UNKNOWN;
  Runtime& rt = Runtime::get();
  if (!rt.init()) return SYLVER_ERROR_CUDA_UNKNOWN;
  try {
    const int m = k + rows, ld = (m + 3) / 4 * 4,
              pitch = (k + TC_KCHUNK - 1) / TC_KCHUNK * TC_KCHUNK;
    std::vector<float> h((size_t)ld * m, 0.f);
    std::mt19937 gen(7);
    std::uniform_real_distribution<float> U(-1.f, 1.f);
    for (int c = 0; c < k; ++c)
      for (int r = k; r < m; ++r) h[(size_t)c * ld + r] = U(gen);
    DevMem arena, planes, sp, tk, err;
    arena.ensure(h.size() * sizeof(float));
    SG_CUDA(cudaMemcpy(arena.p, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice));
    const int64_t pstride = ((int64_t)rows * pitch + 63) / 64 * 64;
    planes.ensure((size_t)3 * pstride * sizeof(uint16_t));
    std::vector<TcSplit> hs{{0, ld, m, k, k, 0, 0}};
    std::vector<TcTask> ht;
    for (int cj = 0; cj * 128 < rows; ++cj)
      for (int ri = cj; ri * 128 < rows; ++ri)
        ht.push_back({0, ld, k + ri * 128, k + cj * 128, m, m, ri * 128, cj * 128,
                      (k + TC_KCHUNK - 1) / TC_KCHUNK});
    sp.upload(hs, rt.stream);
    tk.upload(ht, rt.stream);
    err.ensure(sizeof(unsigned));
    SG_CUDA(cudaMemsetAsync(err.p, 0, sizeof(unsigned), rt.stream));
    CUtensorMap maps[3];
    for (int q = 0; q < 3; ++q)
      make_panel_map(&maps[q], planes.as<uint16_t>() + q * pstride, rows, pitch);
    launch_split_t(arena.as<float>(), sp.as<TcSplit>(), 1, (int64_t)rows,
                   planes.as<uint16_t>(), pstride, pitch, rt.stream);
    launch_update_tc(maps, arena.as<float>(), tk.as<TcTask>(), (int)ht.size(),
                     err.as<unsigned>(), rt.stream);
    unsigned herr = 0;
    SG_CUDA(cudaMemcpyAsync(&herr, err.p, sizeof(unsigned), cudaMemcpyDeviceToHost, rt.stream));
    std::vector<float> out(h.size());
    SG_CUDA(cudaMemcpyAsync(out.data(), arena.p, h.size() * sizeof(float),
                            cudaMemcpyDeviceToHost, rt.stream));
    SG_CUDA(cudaStreamSynchronize(rt.stream));
    if (herr) return SYLVER_ERROR_CUDA_UNKNOWN;
    double worst = 0.0, scale = 0.0;
    for (int j = 0; j < rows; ++j)
      for (int i = j; i < rows; ++i) {
        double ref = 0.0;
        for (int c = 0; c < k; ++c)
          ref -= (double)h[(size_t)c * ld + k + i] * (double)h[(size_t)c * ld + k + j];
        double got = out[(size_t)(k + j) * ld + k + i];
        worst = std::max(worst, std::fabs(got - ref));
        scale = std::max(scale, std::fabs(ref));
      }
    *max_rel_err = scale > 0 ? worst / scale : worst;
    return SYLVER_SUCCESS;
  } catch (const std::exception&) {
    return SYLVER_ERROR_CUDA_UNKNOWN;
  }
}

namespace {

struct Tc64Result {
  double norm_err = 0.0;   // over the product of the two row norms, in 2^-53
  double entry_err = 0.0;  // over (k + 3) |L| |L^T| + 9/8 |C|, in 2^-53
  long changed = 0;        // words outside the updated triangle that changed
};

// One FP64 update of a synthetic front: L21 entries of magnitude 2^-spread .. 1,
// each row scaled by a power of two up to 2^+-rowexp, C - L21 L21^T formed in
// long double.  fill: C, of 2^-60 .. 2^4 times the row norms, and every other
// word of the front (the upper triangle, the rows that pad a column) hold known
// values; else zeros.  Row `special` (>= 0) gets an infinity: entries outside its
// row and column must not see it, and every entry in them must be NaN.
int tc64_check(int rows, int k, int spread, int rowexp, int tile_cols, int special, bool fill,
               Tc64Result* res) {
  Runtime& rt = Runtime::get();
  if (!rt.init()) return SYLVER_ERROR_CUDA_UNKNOWN;
  try {
    const int m = k + rows, ld = (m + 3) / 4 * 4 + (fill ? 4 : 0), pitch = (k + 63) / 64 * 64;
    std::vector<double> h((size_t)ld * m, 0.0);
    std::mt19937_64 gen(7);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    std::uniform_int_distribution<int> S(-spread, 0), R(-rowexp, rowexp), F(-60, 4);
    std::vector<double> norm(rows);
    std::vector<int> rexp(rows);
    if (fill)
      for (auto& v : h) v = U(gen);
    for (int r = 0; r < rows; ++r) {
      const int e = rexp[r] = rowexp > 0 ? R(gen) : 0;
      long double q = 0;
      for (int c = 0; c < k; ++c) {
        const double v = std::ldexp(U(gen), e + S(gen));
        h[(size_t)c * ld + k + r] = v;
        const long double w = std::ldexp(v, -e);
        q += w * w;
      }
      norm[r] = (double)std::sqrt(q);  // of the row times 2^-e
    }
    if (fill)
      for (int j = 0; j < rows; ++j)
        for (int i = j; i < rows; ++i)
          h[(size_t)(k + j) * ld + k + i] = std::ldexp(U(gen), rexp[i] + rexp[j] + F(gen));
    if (special >= 0) h[(size_t)(k / 2) * ld + k + special] = INFINITY;
    DevMem arena, planes, sexp, sp, tk, redo, err;
    arena.ensure(h.size() * sizeof(double));
    SG_CUDA(cudaMemcpy(arena.p, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
    const int64_t pstride = ((int64_t)rows * pitch + 63) / 64 * 64;
    planes.ensure((size_t)OZ_DIGITS * pstride * sizeof(uint16_t));
    sexp.ensure((size_t)rows * sizeof(int));
    std::vector<OzSplit> hs{{0, ld, k, rows, 0, k, 0}};
    std::vector<OzTask> ht;
    for (int c = 0; c < rows; c += tile_cols)
      for (int r = c; r < rows; r += 128)
        ht.push_back({0, ld, k + r, k + c, m, std::min(m, k + c + tile_cols), r, c, 0, k, 0});
    sp.upload(hs, rt.stream);
    tk.upload(ht, rt.stream);
    err.ensure(sizeof(unsigned));
    SG_CUDA(cudaMemsetAsync(err.p, 0, sizeof(unsigned), rt.stream));
    redo.ensure(update_tc64_redo_words((int64_t)ht.size()) * sizeof(unsigned));
    CUtensorMap maps[2];
    make_digit_maps(maps, planes.as<uint16_t>(), pstride, rows, pitch);
    launch_oz_split(arena.as<double>(), sp.as<OzSplit>(), 1, rows, planes.as<uint16_t>(), pstride,
                    pitch, sexp.as<int>(), rt.stream);
    launch_update_tc64(maps, arena.as<double>(), sexp.as<int>(), tk.as<OzTask>(), (int)ht.size(),
                       redo.as<unsigned>(), err.as<unsigned>(), rt.stream);
    unsigned herr = 0;
    SG_CUDA(cudaMemcpyAsync(&herr, err.p, sizeof(unsigned), cudaMemcpyDeviceToHost, rt.stream));
    std::vector<double> out(h.size());
    SG_CUDA(cudaMemcpyAsync(out.data(), arena.p, h.size() * sizeof(double),
                            cudaMemcpyDeviceToHost, rt.stream));
    SG_CUDA(cudaStreamSynchronize(rt.stream));
    if (herr) return SYLVER_ERROR_CUDA_UNKNOWN;
    auto worse = [](double& w, double e) { w = std::isnan(e) ? INFINITY : std::max(w, e); };
    for (int c = 0; c < m; ++c)
      for (int r = 0; r < ld; ++r)
        if ((c < k || r < c || r >= m) &&
            std::memcmp(&h[(size_t)c * ld + r], &out[(size_t)c * ld + r], sizeof(double)))
          ++res->changed;
    for (int j = 0; j < rows; ++j)
      for (int i = j; i < rows; ++i) {
        const size_t at = (size_t)(k + j) * ld + k + i;
        if (i == special || j == special) {
          if (!std::isnan(out[at])) res->norm_err = res->entry_err = INFINITY;
          continue;
        }
        const int e = rexp[i] + rexp[j];  // in units of 2^e: no overflow
        const long double c0 = std::ldexp((long double)h[at], -e);
        long double ref = c0, mag = 0.0;
        for (int c = 0; c < k; ++c) {
          const long double x = std::ldexp(h[(size_t)c * ld + k + i], -rexp[i]);
          const long double y = std::ldexp(h[(size_t)c * ld + k + j], -rexp[j]);
          ref -= x * y;
          mag += std::fabs(x * y);
        }
        const long double d = std::fabs(std::ldexp((long double)out[at], -e) - ref);
        worse(res->norm_err, (double)std::ldexp(d / norm[i] / norm[j], 53));
        // (2^-1074: results that underflow)
        const long double tol = (k + 3) * mag + 1.125L * std::fabs(c0) +
                                std::ldexp(1.0L, -1074 + 53 - e);
        worse(res->entry_err, (double)std::ldexp(d / tol, 53));
      }
    return SYLVER_SUCCESS;
  } catch (const std::exception&) {
    return SYLVER_ERROR_CUDA_UNKNOWN;
  }
}

}  // namespace

extern "C" int sylver_gb300_tc64_selfcheck(int rows, int k, int spread, int special,
                                           double* max_err) {
  if (rows < 1 || k < 1 || spread < 0 || special >= rows || !max_err) return SYLVER_ERROR_UNKNOWN;
  Tc64Result r;
  const int rc = tc64_check(rows, k, spread, spread > 0 ? 200 : 0, OZ_TILE_COLS, special, false, &r);
  if (rc == SYLVER_SUCCESS) *max_err = r.norm_err;
  return rc;
}

extern "C" int sylver_gb300_tc64_entrycheck(int rows, int k, int spread, int rowexp, int narrow,
                                            int special, double* max_err, long* changed) {
  if (rows < 1 || k < 1 || spread < 0 || spread > 900 || rowexp < 0 || rowexp > 500 ||
      special >= rows || !max_err || !changed)
    return SYLVER_ERROR_UNKNOWN;
  Tc64Result r;
  const int rc = tc64_check(rows, k, spread, rowexp, narrow ? OZ_TILE_COLS / 2 : OZ_TILE_COLS,
                            special, true, &r);
  *max_err = r.entry_err;
  *changed = r.changed;
  return rc;
}
