// lbm_sweeps.cuh - the nearest-image history of the in-place sweeps of
// beads_links (B/partlib.f90:959-985), shared by the particle kernels and the
// host check of its two forms.
#pragma once
#include <cmath>
#include <cstring>

#include "lbm_collide.cuh"

namespace lbm {
namespace {

// The reference's beads_links keeps shifting the particle centre toward the
// current point and never resets it inside its loop nest
// (B/partlib.f90:961-982): at point p_j = j - 0.5 of a sweep j = 1..n it
// applies "if (c - p > n/2) c -= n; if (c - p < -n/2) c += n" to the value
// left by the previous point.  fl(c - p) is monotone in p, so both shift
// predicates are monotone along a sweep and the points where a shift fires
// are found by bisection instead of visiting every point.
// The points of one sweep where the shifted coordinate changes, with the
// value after each change: a sweep starting from c changes at most a few
// times (a shift down at the first point, a shift up once c - p drops
// below -n/2), so any point's value is a lookup in this short list.
constexpr int MAXEV = 6;
struct SweepEv {
  int nev;
  int ok;
  int j[MAXEV];
  double v[MAXEV];
  double v0;
};
static_assert(7 * sizeof(SweepEv) <= kSweepBytes, "sweep slab too small");
__host__ __device__ __noinline__ SweepEv sweep_events(double c, int n, int nh) {
  SweepEv s;
  s.nev = 0;
  s.ok = 1;
  s.v0 = c;
  const double dn = (double)n, dnh = (double)nh;
  int j = 1;
  for (int guard = 0; guard < 16; ++guard) {
    const double p = (double)j - 0.5;
    const double before = c;
    if ((c - p) > dnh) c = c - dn;
    if ((c - p) < -dnh) c = c + dn;
    long long bits, bits_before;
    memcpy(&bits, &c, sizeof c);
    memcpy(&bits_before, &before, sizeof c);
    if (bits != bits_before) {
      if (s.nev < MAXEV) { s.j[s.nev] = j; s.v[s.nev] = c; ++s.nev; } else s.ok = 0;
    }
    if (j >= n) return s;
    int jn = n + 1;
    const double p1 = (double)(j + 1) - 0.5;
    if ((c - p1) > dnh) {
      jn = j + 1;
    } else if ((c - ((double)n - 0.5)) < -dnh) {
      // the first point m in [j + 1, n] where the shift up fires.  In exact
      // arithmetic that is the first m > c + n/2 + 1/2, and fl(c - p) is
      // within an ulp of c - p, so the FP64 first point lies within two of
      // floor(c + n/2 + 1/2) + 1: scan from two below it with the
      // reference's expression (monotone in m) after checking that the start
      // is not past it; bisect where either check fails (not expected).
      auto up = [&](int m) { return (c - ((double)m - 0.5)) < -dnh; };
      int lo = j + 1, hi = n;
      int m = (int)floor(c + dnh + 0.5) - 1;
      m = m < lo ? lo : (m > hi ? hi : m);
      bool found = false;
      if (m == lo || !up(m - 1)) {
        for (int t = 0; t < 6 && m <= hi; ++t, ++m)
          if (up(m)) { found = true; break; }
        if (!found) lo = m;
      } else {
        hi = m - 1;
      }
      if (!found) {
        while (lo < hi) {
          int mid = (lo + hi) >> 1;
          if (up(mid)) hi = mid; else lo = mid + 1;
        }
        m = lo;
      }
      jn = m;
    }
    if (jn > n) return s;
    j = jn;
  }
  s.ok = 0;
  return s;
}
// sweep_events for a centre whose shifts are not in doubt: the same list, with
// the decisions taken on the centre in 64-bit fixed point at 2^-kSweepFx
// (integer operations) wherever it is farther than kSweepNear from a tie, and
// only the shifts themselves in FP64, whose latency bounds this serial chain
// (a sweep of sweep_events takes some thirty dependent FP64 operations, this
// one two at most).  Then either nothing happens at the first point or one
// shift down, and at most one shift up later on.  ev gets the list, c the
// value at the end of the sweep; false, with neither changed, when a decision
// is in doubt or the shifts are of another kind (an odd n whose shift down is
// taken back at the same point, a centre beyond the box).
constexpr int kSweepFx = 40;
constexpr long long kSweepNear = 1LL << 6;
__host__ __device__ __forceinline__ bool sweep_fast(double& c, int n, int nh, SweepEv* ev) {
  if (!(fabs(c) < 4194304.0)) return false;  // 2^22: the fixed point holds it
  const long long one = 1LL << kSweepFx, half = one >> 1;
  const long long N = (long long)n << kSweepFx, H = (long long)nh << kSweepFx;
  long long C = fx_from_k(c, kSweepFx);
  auto doubt = [](long long d) { return (d < 0 ? -d : d) <= kSweepNear; };
  // the first point, p = 1/2
  const long long d1 = C - half - H;
  if (doubt(d1)) return false;
  const bool down = d1 > 0;
  if (down) C -= N;
  // after it: neither shift may apply to the value at p = 1/2 (up) or, for the
  // points beyond, be left over (down)
  const long long u1 = C - half + H, d2 = C - half - one - H;
  if (u1 <= kSweepNear || d2 >= -kSweepNear) return false;
  // the first point m > c + n/2 + 1/2 shifts up
  const long long t = C + H + half;
  const long long frac = t & (one - 1);
  if (frac <= kSweepNear || frac >= one - kSweepNear) return false;
  const int m = (int)(t >> kSweepFx) + 1;
  const bool up = m <= n;
  // beyond it nothing is left to shift down
  if (up && C + N - (((long long)m << kSweepFx) + half) - H >= -kSweepNear) return false;
  if (m < 2) return false;
  const double v0 = c, dn = (double)n;
  const double v1 = down ? c - dn : c;
  const double v2 = up ? v1 + dn : v1;
  ev->nev = (down ? 1 : 0) + (up ? 1 : 0);
  ev->ok = 1;
  ev->v0 = v0;
  if (down) { ev->j[0] = 1; ev->v[0] = v1; }
  if (up) {
    ev->j[down ? 1 : 0] = m;
    ev->v[down ? 1 : 0] = v2;
  }
  c = v2;
  return true;
}
__host__ __device__ __forceinline__ double sweep_value(const SweepEv& s, int jq) {
  double v = s.v0;
  for (int e = 0; e < s.nev; ++e)
    if (s.j[e] <= jq) v = s.v[e];
  return v;
}

}  // namespace
}  // namespace lbm
