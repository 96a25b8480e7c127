// Shared device code of the bond kernels: real spherical harmonics with the gradient of their polynomial extension,
// and the cubic Hermite evaluation of the radial functions.
#pragma once

#include "kernels.h"

namespace gb {

// recurrence coefficients of the real spherical harmonics for l <= 4, set once per process by
// bond_tables_init(): a, b indexed l (l + 1) / 2 + m, c and d indexed l (libgrace/include/grace/fused_cpu.h:686-702)
struct SHTable {
  float a[15], b[15], c[5], d[5];
};
const SHTable &sh_table_host();

// Y[lm] (and G[lm] = dY/d(x, y, z) of the polynomial extension) of the unit vector (rx, ry, rz); Y00 = 1,
// lm = l (l + 1) + m (libgrace/include/grace/fused_cpu.h:711-798).  Out: a functor out(lm, y, gx, gy, gz).
template<int LMAX, bool GRAD, class Out>
__device__ __forceinline__ void sph_harm(const SHTable &t, float rx, float ry, float rz, Out out)
{
  constexpr int NP = (LMAX + 1) * (LMAX + 2) / 2;
  float plm[NP], dplm[NP];
  plm[0] = 1.0f;
  dplm[0] = 0.0f;
  if (LMAX > 0) {
    plm[1] = 1.7320508075688772f * rz;
    dplm[1] = 1.7320508075688772f;
    plm[2] = -1.224744871391589f;
    dplm[2] = 0.0f;
  }
#pragma unroll
  for (int l = 2; l <= LMAX; l++) {
#pragma unroll
    for (int mm = 0; mm < l - 1; mm++) {
      const int id = l * (l + 1) / 2 + mm, i1 = (l - 1) * l / 2 + mm, i2 = (l - 2) * (l - 1) / 2 + mm;
      plm[id] = t.a[id] * (rz * plm[i1] + t.b[id] * plm[i2]);
      dplm[id] = t.a[id] * (plm[i1] + rz * dplm[i1] + t.b[id] * dplm[i2]);
    }
    const int prev = (l - 1) * l / 2 + l - 1, i0 = l * (l + 1) / 2 + l - 1, i1 = l * (l + 1) / 2 + l;
    plm[i0] = t.d[l] * plm[prev] * rz;
    plm[i1] = t.c[l] * plm[prev];
    dplm[i0] = t.d[l] * (dplm[prev] * rz + plm[prev]);
    dplm[i1] = t.c[l] * dplm[prev];
  }
  const float sq2 = 1.4142135623730951f;
#pragma unroll
  for (int l = 0; l <= LMAX; l++) {
    const int c = l * (l + 1), p0 = l * (l + 1) / 2;
    out(c, plm[p0], 0.0f, 0.0f, dplm[p0]);
    float pr = rx, pi = ry, prx = 1.0f, pry = 0.0f, pix = 0.0f, piy = 1.0f;
#pragma unroll
    for (int mm = 1; mm <= l; mm++) {
      const float sg = (mm % 2 == 0) ? sq2 : -sq2;
      const float pv = plm[p0 + mm], dpv = dplm[p0 + mm];
      out(c + mm, sg * pr * pv, sg * prx * pv, sg * pry * pv, sg * pr * dpv);
      out(c - mm, sg * pi * pv, sg * pix * pv, sg * piy * pv, sg * pi * dpv);
      if (GRAD) {
        const float nrx = prx * rx + pr - pix * ry, nry = pry * rx - piy * ry - pi;
        const float nix = prx * ry + pix * rx + pi, niy = pry * ry + pr + piy * rx;
        prx = nrx; pry = nry; pix = nix; piy = niy;
      }
      const float nr = pr * rx - pi * ry, ni = pr * ry + pi * rx;
      pr = nr; pi = ni;
    }
  }
}

// Sums of four per-lane values over the groups of G consecutive lanes of a warp (G = 8, 16 or 32) with 1 + log2(G)
// shuffles instead of 4 log2(G): the halves of a group first trade two of the values, the quarters one, and from then
// on every lane carries a single value.  Afterwards lane q G / 4 of a group (q = 0 .. 3) holds the sum of value q in
// `out`; the additions pair the same lanes as a butterfly per value, so the sums are bit-identical to it.
template<int G>
__device__ __forceinline__ float group_sum4(float v0, float v1, float v2, float v3, int lane_in_group)
{
  const bool up = lane_in_group & (G / 2), odd = lane_in_group & (G / 4);
  const float r0 = __shfl_xor_sync(0xffffffffu, up ? v0 : v2, G / 2), r1 = __shfl_xor_sync(0xffffffffu, up ? v1 : v3, G / 2);
  const float k0 = (up ? v2 : v0) + r0, k1 = (up ? v3 : v1) + r1;
  float v = (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, G / 4);
#pragma unroll
  for (int s = G / 8; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
  return v;
}

// ---- two channels per lane -------------------------------------------------------------------------------------
// The kernels of layers with an even number of channels keep two neighbouring channels in a lane: every sum is a packed
// two-wide FMA, a bond takes half the lanes and a warp works on several bonds at once.  Factors that are the same for both
// channels (harmonics) are staged in shared memory twice side by side, so that no instruction goes into pairing them.
__device__ __forceinline__ float2 pair_of(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

// radial functions of a channel pair from the table of pairs (rows of x x y y, then of z z w w: a load instruction of a bond covers a contiguous
// row; with the two quadruples of a pair side by side the lanes are 32 bytes apart and the kernels a fifth slower)
__device__ __forceinline__ float2 pair_value(float4 xy, float4 zw, float2 t)
{
  return __ffma2_rn(t, __ffma2_rn(t, __ffma2_rn(t, hi2(zw), lo2(zw)), hi2(xy)), lo2(xy));
}
// their derivative by the interval's offset: y + 2 t (z + 1.5 t w)
__device__ __forceinline__ float2 pair_slope(float4 xy, float4 zw, float2 t_2, float2 t_15)
{
  return __ffma2_rn(t_2, __ffma2_rn(t_15, hi2(zw), lo2(zw)), hi2(xy));
}

// Layers with four message functions split the harmonics of a bond between two groups of lanes, by whole degrees so that a
// group needs the radial functions of its own degrees only: lmax 3: {3, 0} and {2, 1}, eight harmonics each.  Position k of
// group h holds lm(h, k) of the degree in slot(h, k); where the groups hold another slot at a position, the lane selects.
template<int LMAX> struct LmSplit {
  static constexpr int NL = LMAX + 1, NLM = NL * NL;
  static constexpr int NS = LMAX == 1 ? 1 : LMAX == 4 ? 3 : 2;       // degrees of a group, at most
  static constexpr int NK = LMAX == 1 ? 3 : LMAX == 2 ? 5 : LMAX == 3 ? 8 : 13;
  // degree of slot s of group h, -1: none
  static constexpr __host__ __device__ int degree(int h, int s)
  {
    if (LMAX == 1) return s == 0 ? (h ? 0 : 1) : -1;
    if (LMAX == 2) return h ? (s < 2 ? 1 - s : -1) : s == 0 ? 2 : -1;
    if (LMAX == 3) return s > 1 ? -1 : h ? 2 - s : s == 0 ? 3 : 0;
    return h ? (s == 0 ? 3 : s == 1 ? 2 : 0) : s == 0 ? 4 : s == 1 ? 1 : -1;
  }
  static constexpr __host__ __device__ int slot(int h, int k)    // NS: no harmonic at the position
  {
    int at = 0;
    for (int s = 0; s < NS; s++) {
      const int l = degree(h, s);
      if (l < 0) break;
      at += 2 * l + 1;
      if (k < at) return s;
    }
    return NS;
  }
  static constexpr __host__ __device__ int lm(int h, int k)      // -1: none
  {
    int at = 0;
    for (int s = 0; s < NS; s++) {
      const int l = degree(h, s);
      if (l < 0) break;
      if (k < at + 2 * l + 1) return l * l + k - at;
      at += 2 * l + 1;
    }
    return -1;
  }
  static constexpr __host__ __device__ int place(int q)          // h NK + k of harmonic q
  {
    for (int h = 0; h < 2; h++)
      for (int k = 0; k < NK; k++)
        if (lm(h, k) == q) return h * NK + k;
    return -1;
  }
};
// place() at compile time, for the loops over harmonics whose index is a constant only after unrolling
template<int LMAX> struct LmPlaces {
  int v[25];
  constexpr LmPlaces() : v{}
  {
    for (int q = 0; q < 25; q++) v[q] = q < LmSplit<LMAX>::NLM ? LmSplit<LMAX>::place(q) : -1;
  }
};

// interval k and offset t of x = r / rcut in a table of N intervals (libgrace/include/grace/fused_cpu.h:1052-1058)
__device__ __forceinline__ void spline_locate(float x, int N, int &k, float &t)
{
  const float s = x * (float) N;
  k = (int) s;
  if (k > N - 1) k = N - 1;
  if (k < 0) k = 0;
  t = s - (float) k;
}

}    // namespace gb
