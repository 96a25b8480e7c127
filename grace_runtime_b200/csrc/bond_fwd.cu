// Forward bond kernel: the neighbour sums of a layer,
//   Q[(I, lm)][a][n] = sum_j Y_lm(rhat_ij) R[n, l](r_ij / rcut) msg_I(j)[n]
// with msg_I the message functions of the neighbour (layer 2: I < n_msg) and, as the last I, its chemical weight
// z[mu_j][n] (layer 1: A; layer 2: B0).  This is atom_scatter + atom_yi of the reference CPU driver
// (libgrace/include/grace/fused_cpu.h:947-1025) in the dense (I, lm) form of its GPU kernels
// (libgrace/include/grace/kk/grace_2l_fused_kk_impl.h:858-1070).
//
// One block of 4 warps per atom.  A lane owns channel n (NCH channels for C > 32); the 4 warps (and with C <= 16 the
// two half-warps) take the atom's bonds in turn, every thread keeping all NIT x NLM partial sums of its channel in
// registers; the partial sums of the warps are added in shared memory in a fixed order and written once, coalesced
// over n: no global atomics, bit-reproducible.
#include "bond_common.cuh"

namespace gb {

namespace {

constexpr int EB = 96;    // bonds staged per round: most atoms in one round

template<int LMAX, int NIT, int NCH, int LPE, bool EXACT>
__global__ void __launch_bounds__(128) bond_fwd_kernel(BondsDev b, LayerDev L, SHTable sht, float *__restrict__ Q,
                                                       int NA, int a0)
{
  // rows of the staged harmonics: a multiple of 4 floats (the lanes of a bond read them as broadcast 16-byte loads, a
  // quarter of the shared-memory transactions of scalar reads) plus 4, which spreads the rows over the banks
  constexpr int NL = LMAX + 1, NLM = NL * NL, NLM4 = (NLM + 3) / 4, NLMP = 4 * NLM4 + ((4 * NLM4 + 4) % 32 ? 4 : 8), NQ = NIT * NLM, CP = LPE * NCH, EPW = 32 / LPE;
  __shared__ __align__(16) float Ys[EB][NLMP];
  __shared__ float st[EB];
  __shared__ int sk[EB], smu[EB], sj[EB];
  __shared__ float red[NQ][CP];

  const int a = blockIdx.x, i = b.ilist ? b.ilist[a0 + a] : a0 + a, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int ln = lane % LPE, esub = lane / LPE;
  const int Ibase = blockIdx.y * NIT;
  const long long base = b.off[i];
  const int nb = b.cnt[i];
  const int mui = b.mu[i];
  const int C = L.C, nel = L.n_elements;

  float acc[NIT][NLM][NCH];
#pragma unroll
  for (int I = 0; I < NIT; I++)
#pragma unroll
    for (int q = 0; q < NLM; q++)
#pragma unroll
      for (int ch = 0; ch < NCH; ch++) acc[I][q][ch] = 0.0f;

  for (int b0 = 0; b0 < nb; b0 += EB) {
    const int nbat = min(EB, nb - b0);
    for (int e = tid; e < nbat; e += 128) {
      const float4 rec = b.rec[base + b0 + e];
      const float r = sqrtf(rec.x * rec.x + rec.y * rec.y + rec.z * rec.z), ir = 1.0f / r;
      const int j = __float_as_int(rec.w);
      const int muj = b.mu[j];
      int k;
      float t;
      spline_locate(r / L.rc[mui * nel + muj], L.N, k, t);
      sk[e] = k; st[e] = t; smu[e] = muj; sj[e] = j;
      float *y = Ys[e];
      sph_harm<LMAX, false>(sht, rec.x * ir, rec.y * ir, rec.z * ir,
                            [&](int lm, float v, float, float, float) { y[lm] = v; });
    }
    __syncthreads();
    for (int e0 = w * EPW; e0 < nbat; e0 += 4 * EPW) {
      const int e = e0 + esub;
      if (e < nbat) {
        const int k = sk[e], muj = smu[e], j = sj[e];
        const float t = st[e];
        float y[4 * NLM4];
#pragma unroll
        for (int q4 = 0; q4 < NLM4; q4++) {
          const float4 v = reinterpret_cast<const float4 *>(Ys[e])[q4];
          y[4 * q4] = v.x; y[4 * q4 + 1] = v.y; y[4 * q4 + 2] = v.z; y[4 * q4 + 3] = v.w;
        }
#pragma unroll
        for (int ch = 0; ch < NCH; ch++) {
          const int n = ln + ch * LPE;
          if (n < C) {
            float R[NL];
            if (EXACT) {    // exact radial MLP, evaluated per slot beforehand
              const float *rr = L.Rex + (size_t) (base + b0 + e) * (NL * C) + n;
#pragma unroll
              for (int l = 0; l < NL; l++) R[l] = __ldg(rr + l * C);
            } else {
              const float4 *cf = reinterpret_cast<const float4 *>(L.tab) + (size_t) k * NL * C + n;
#pragma unroll
              for (int l = 0; l < NL; l++) {
                const float4 c = __ldg(cf + l * C);
                R[l] = c.x + t * (c.y + t * (c.z + t * c.w));
              }
            }
#pragma unroll
            for (int I = 0; I < NIT; I++) {
              const int Ig = Ibase + I;
              float m = 0.0f;
              if (Ig < L.n_msg) m = __ldg(L.msg + ((size_t) j * L.n_msg + Ig) * C + n);
              else if (Ig == L.n_msg) m = __ldg(L.z + (size_t) muj * C + n);
#pragma unroll
              for (int l = 0; l < NL; l++) {
                const float rm = R[l] * m;
#pragma unroll
                for (int q = l * l; q < (l + 1) * (l + 1); q++) acc[I][q][ch] = fmaf(y[q], rm, acc[I][q][ch]);
              }
            }
          }
        }
      }
    }
    __syncthreads();
  }

  if (EPW == 2) {    // the two half-warps worked on different bonds: add them
#pragma unroll
    for (int I = 0; I < NIT; I++)
#pragma unroll
      for (int q = 0; q < NLM; q++) acc[I][q][0] += __shfl_xor_sync(0xffffffffu, acc[I][q][0], 16);
  }
  for (int ww = 0; ww < 4; ww++) {
    if (w == ww && esub == 0) {
#pragma unroll
      for (int I = 0; I < NIT; I++)
#pragma unroll
        for (int q = 0; q < NLM; q++)
#pragma unroll
          for (int ch = 0; ch < NCH; ch++) {
            float *r = &red[I * NLM + q][ln + ch * LPE];
            *r = (ww == 0) ? acc[I][q][ch] : *r + acc[I][q][ch];
          }
    }
    __syncthreads();
  }
  for (int idx = tid; idx < NQ * C; idx += 128) {
    const int q = idx / C, n = idx - q * C;
    if (Ibase + q / NLM <= L.n_msg) Q[((size_t) (Ibase * NLM + q) * NA + a) * C + n] = red[q][n];
  }
}

// Layers without message functions and with an even number of channels: LPB = 8, 16 or 32 lanes per bond, two channels per
// lane, 32 / LPB bonds per warp at a time.  Bound by the radial table: a bond reads NL C coefficient quadruples (2 KB at
// lmax 3, 32 channels) out of 2 MB, and the kernel moves them at the rate of the L1 and L2 caches (12 - 14 TB/s).  Against one
// channel per lane: GRACE-1L, 128,000 atoms, lmax 4: 1.80 -> 1.64 ms; GRACE-2L, 1,024,000 atoms, lmax 3: 11.7 ms both.
template<int LMAX, int LPB>
__global__ void __launch_bounds__(128, LMAX <= 3 ? 8 : 5) bond_fwd_pair_kernel(BondsDev b, LayerDev L, SHTable sht, float *__restrict__ Q, int NA, int a0)
{
  constexpr int NL = LMAX + 1, NLM = NL * NL, NP = (NLM + 1) / 2, ROW = NP | 1, BPW = 32 / LPB;    // odd rows: no bank conflicts
  constexpr int Y_F4 = EB * ROW, RED_F4 = 4 * NLM * LPB / 2, BUF = Y_F4 > RED_F4 ? Y_F4 : RED_F4;
  __shared__ float4 buf[BUF];    // harmonics of the bonds at hand (y0 y0 y1 y1); afterwards the sums of the warps
  __shared__ int4 meta[EB];      // interval, element, offset

  const int a = blockIdx.x, i = b.ilist ? b.ilist[a0 + a] : a0 + a, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int c = lane % LPB, sub = lane / LPB;
  const long long base = b.off[i];
  const int nb = b.cnt[i], mui = b.mu[i], C = L.C, C2 = C >> 1, nel = L.n_elements;
  const int rounds = max(1, (nb + EB - 1) / EB), per = (nb + rounds - 1) / rounds;
  float2 acc[NLM];
#pragma unroll
  for (int q = 0; q < NLM; q++) acc[q] = make_float2(0.f, 0.f);

  for (int b0 = 0; b0 < nb; b0 += per) {
    const int nbat = min(per, nb - b0);
    for (int e = tid; e < nbat; e += 128) {
      const float4 rec = b.rec[base + b0 + e];
      const float r = sqrtf(rec.x * rec.x + rec.y * rec.y + rec.z * rec.z), ir = 1.0f / r;
      const int muj = b.mu[__float_as_int(rec.w)];
      int k;
      float t;
      spline_locate(r / L.rc[mui * nel + muj], L.N, k, t);
      meta[e] = make_int4(k, muj, __float_as_int(t), 0);
      float2 *y = reinterpret_cast<float2 *>(buf + e * ROW);
      sph_harm<LMAX, false>(sht, rec.x * ir, rec.y * ir, rec.z * ir, [&](int lm, float v, float, float, float) { y[lm] = pair_of(v); });
    }
    __syncthreads();
    for (int e = w * BPW + sub; e < nbat; e += 4 * BPW) {
      if (c < C2) {
        const int4 m = meta[e];
        const float2 t = pair_of(__int_as_float(m.z));
        const float4 *cf = reinterpret_cast<const float4 *>(L.tab) + (size_t) m.x * NL * C + c;
        const float2 z = __ldg(reinterpret_cast<const float2 *>(L.z + (size_t) m.y * C) + c);
        float2 R[NL];
#pragma unroll
        for (int l = 0; l < NL; l++) R[l] = __fmul2_rn(pair_value(__ldg(cf + l * C), __ldg(cf + l * C + C2), t), z);
        const float4 *y = buf + e * ROW;
#pragma unroll
        for (int p = 0; p < NP; p++) {
          constexpr auto deg = [](int q) { int l = 0; while ((l + 1) * (l + 1) <= q) l++; return l; };
          const float4 v = y[p];
          acc[2 * p] = __ffma2_rn(lo2(v), R[deg(2 * p)], acc[2 * p]);
          if (2 * p + 1 < NLM) acc[2 * p + 1] = __ffma2_rn(hi2(v), R[deg(2 * p + 1)], acc[2 * p + 1]);
        }
      }
    }
    __syncthreads();
  }
  // the bonds of a warp by shuffles, the warps in order through shared memory
#pragma unroll
  for (int s = LPB; s < 32; s *= 2)
#pragma unroll
    for (int q = 0; q < NLM; q++) {
      acc[q].x += __shfl_xor_sync(0xffffffffu, acc[q].x, s);
      acc[q].y += __shfl_xor_sync(0xffffffffu, acc[q].y, s);
    }
  float2 *red = reinterpret_cast<float2 *>(buf);
  if (sub == 0) {
#pragma unroll
    for (int q = 0; q < NLM; q++) red[(w * NLM + q) * LPB + c] = acc[q];
  }
  __syncthreads();
  for (int x = tid; x < NLM * LPB; x += 128) {
    const int q = x / LPB, cc = x % LPB;
    if (cc >= C2) continue;
    float2 v = red[x];
#pragma unroll
    for (int ww = 1; ww < 4; ww++) {
      const float2 u = red[ww * NLM * LPB + x];
      v.x += u.x;
      v.y += u.y;
    }
    *(reinterpret_cast<float2 *>(Q + ((size_t) q * NA + a) * C) + cc) = v;
  }
}

// Layers with four message functions and at most 16 channels (an even number): 16 lanes per bond, lane = (group h of
// harmonics, channel pair c), two bonds per warp at a time; a lane keeps 5 x NK sums of two channels,
//   Q[(I, lm)][n] += (Y_lm R_l) msg_I.
// One channel per lane with the harmonics interleaved took 203 issued instructions per bond and was bound by them; this takes
// 103.  GRACE-2L, 1,024,000 atoms: 24.2 -> 15.9 ms.
template<int LMAX>
__global__ void __launch_bounds__(128) bond_fwd_msg_kernel(BondsDev b, LayerDev L, SHTable sht, float *__restrict__ Q, int NA, int a0)
{
  using SP = LmSplit<LMAX>;
  constexpr int NL = LMAX + 1, NLM = NL * NL, NI = 5, NK = SP::NK, NKP = (NK + 1) / 2, ROW = (2 * NKP) | 1;
  constexpr int Y_F4 = EB * ROW, RED_F4 = 4 * NI * 2 * NK * 8 / 2, BUF = Y_F4 > RED_F4 ? Y_F4 : RED_F4;
  __shared__ float4 buf[BUF];    // harmonics of the bonds at hand, per group (y0 y0 y1 y1); afterwards the sums of the warps
  __shared__ int4 meta[EB];      // interval, element, offset, neighbour

  const int a = blockIdx.x, i = b.ilist ? b.ilist[a0 + a] : a0 + a, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int c = lane & 7, h = (lane >> 3) & 1, sub = lane >> 4;
  const long long base = b.off[i];
  const int nb = b.cnt[i], mui = b.mu[i], C = L.C, C2 = C >> 1, nel = L.n_elements;
  const int rounds = max(1, (nb + EB - 1) / EB), per = (nb + rounds - 1) / rounds;
  float2 acc[NI][NK];
#pragma unroll
  for (int I = 0; I < NI; I++)
#pragma unroll
    for (int k = 0; k < NK; k++) acc[I][k] = make_float2(0.f, 0.f);

  for (int b0 = 0; b0 < nb; b0 += per) {
    const int nbat = min(per, nb - b0);
    for (int e = tid; e < nbat; e += 128) {
      const float4 rec = b.rec[base + b0 + e];
      const float r = sqrtf(rec.x * rec.x + rec.y * rec.y + rec.z * rec.z), ir = 1.0f / r;
      const int j = __float_as_int(rec.w), muj = b.mu[j];
      int k;
      float t;
      spline_locate(r / L.rc[mui * nel + muj], L.N, k, t);
      meta[e] = make_int4(k, muj, __float_as_int(t), j);
      float2 *y = reinterpret_cast<float2 *>(buf + e * ROW);
      constexpr LmPlaces<LMAX> places;
      sph_harm<LMAX, false>(sht, rec.x * ir, rec.y * ir, rec.z * ir, [&](int lm, float v, float, float, float) {
        const int at = places.v[lm];
        y[at < NK ? at : 2 * NKP + at - NK] = pair_of(v);
      });
#pragma unroll
      for (int hk = 0; hk < 4 * NKP; hk++) {    // positions without a harmonic
        const int hh = hk / (2 * NKP), k2 = hk % (2 * NKP);
        if (k2 >= NK || SP::lm(hh, k2) < 0) y[hk] = make_float2(0.f, 0.f);
      }
    }
    __syncthreads();
    for (int e = 2 * w + sub; e < nbat; e += 8) {
      if (c < C2) {
        const int4 m = meta[e];
        const float2 t = pair_of(__int_as_float(m.z));
        const float4 *cf = reinterpret_cast<const float4 *>(L.tab) + (size_t) m.x * NL * C + c;
        float2 R[SP::NS], mm[NI];
#pragma unroll
        for (int s = 0; s < SP::NS; s++) {
          constexpr auto some = [](int l) { return l < 0 ? 0 : l; };
          const int l = h ? some(SP::degree(1, s)) : some(SP::degree(0, s));
          R[s] = pair_value(__ldg(cf + l * C), __ldg(cf + l * C + C2), t);
        }
        const float2 *msg = reinterpret_cast<const float2 *>(L.msg + (size_t) m.w * 4 * C) + c;
#pragma unroll
        for (int I = 0; I < 4; I++) mm[I] = __ldg(msg + I * C2);
        mm[4] = __ldg(reinterpret_cast<const float2 *>(L.z + (size_t) m.y * C) + c);
        const float4 *y = buf + e * ROW + h * NKP;
        float4 v;
#pragma unroll
        for (int k = 0; k < NK; k++) {
          if (k % 2 == 0) v = y[k / 2];
          constexpr auto bound = [](int s) { return s < SP::NS ? s : SP::NS - 1; };
          const int s0 = bound(SP::slot(0, k)), s1 = bound(SP::slot(1, k));
          const float2 Rk = s0 == s1 ? R[s0] : h ? R[s1] : R[s0];
          const float2 yr = __fmul2_rn(k % 2 ? hi2(v) : lo2(v), Rk);
#pragma unroll
          for (int I = 0; I < NI; I++) acc[I][k] = __ffma2_rn(yr, mm[I], acc[I][k]);
        }
      }
    }
    __syncthreads();
  }
  float2 *red = reinterpret_cast<float2 *>(buf);    // [warp][I][h][k][c]
#pragma unroll
  for (int I = 0; I < NI; I++)
#pragma unroll
    for (int k = 0; k < NK; k++) {    // the two bonds of a warp
      acc[I][k].x += __shfl_xor_sync(0xffffffffu, acc[I][k].x, 16);
      acc[I][k].y += __shfl_xor_sync(0xffffffffu, acc[I][k].y, 16);
      if (sub == 0) red[(((w * NI + I) * 2 + h) * NK + k) * 8 + c] = acc[I][k];
    }
  __syncthreads();
  constexpr int ALL = NI * 2 * NK * 8;
  for (int x = tid; x < ALL; x += 128) {
    const int cc = x & 7, k = (x >> 3) % NK, hh = (x >> 3) / NK % 2, I = (x >> 3) / (2 * NK), q = SP::lm(hh, k);
    if (cc >= C2 || q < 0) continue;
    float2 v = red[x];
#pragma unroll
    for (int ww = 1; ww < 4; ww++) {
      const float2 u = red[ww * ALL + x];
      v.x += u.x;
      v.y += u.y;
    }
    *(reinterpret_cast<float2 *>(Q + ((size_t) (I * NLM + q) * NA + a) * C) + cc) = v;
  }
}

template<int LMAX, int NIT, int NCH, int LPE>
void launch_t(const BondsDev &b, const LayerDev &L, float *Q, int NA, int a0, int na)
{
  const int tiles = (L.n_msg + 1 + NIT - 1) / NIT;
  if (L.Rex) GB_LAUNCH((bond_fwd_kernel<LMAX, NIT, NCH, LPE, true>), dim3(na, tiles), 128, 0, b, L, sh_table_host(), Q, NA, a0);
  else GB_LAUNCH((bond_fwd_kernel<LMAX, NIT, NCH, LPE, false>), dim3(na, tiles), 128, 0, b, L, sh_table_host(), Q, NA, a0);
}

template<int LMAX> void launch_l(const BondsDev &b, const LayerDev &L, float *Q, int NA, int a0, int na)
{
  const int C = L.C, nI = L.n_msg + 1;
  if (C > 64) throw Unsupported("bond sums with more than 64 channels are not supported");
  if (L.pairs) {
    const SHTable &sh = sh_table_host();
    if (L.n_msg) GB_LAUNCH(bond_fwd_msg_kernel<LMAX>, na, 128, 0, b, L, sh, Q, NA, a0);
    else if (C > 32) GB_LAUNCH((bond_fwd_pair_kernel<LMAX, 32>), na, 128, 0, b, L, sh, Q, NA, a0);
    else if (C > 16) GB_LAUNCH((bond_fwd_pair_kernel<LMAX, 16>), na, 128, 0, b, L, sh, Q, NA, a0);
    else GB_LAUNCH((bond_fwd_pair_kernel<LMAX, 8>), na, 128, 0, b, L, sh, Q, NA, a0);
    return;
  }
  if (C > 32) launch_t<LMAX, 1, 2, 32>(b, L, Q, NA, a0, na);
  else if (C > 16) { if (nI == 5) launch_t<LMAX, 5, 1, 32>(b, L, Q, NA, a0, na); else launch_t<LMAX, 1, 1, 32>(b, L, Q, NA, a0, na); }
  else { if (nI == 5) launch_t<LMAX, 5, 1, 16>(b, L, Q, NA, a0, na); else launch_t<LMAX, 1, 1, 16>(b, L, Q, NA, a0, na); }
}

}    // namespace

__global__ void __launch_bounds__(128) bond_x_kernel(BondsDev b, const float *__restrict__ rc, int nel, float *x)
{
  const int i = blockIdx.x;
  const long long base = b.off[i];
  const int ns = (int) (b.off[i + 1] - base), nb = b.cnt[i], mui = b.mu[i];
  for (int s = threadIdx.x; s < ns; s += 128) {
    float v = 0.5f;
    if (s < nb) {
      const float4 rec = b.rec[base + s];
      const int j = __float_as_int(rec.w);
      v = sqrtf(rec.x * rec.x + rec.y * rec.y + rec.z * rec.z) / rc[mui * nel + b.mu[j]];
    }
    x[base + s] = v;
  }
}

void launch_bond_x(const BondsDev &b, const float *rc, int n_elements, float *x, long long n)
{
  if (n == 0) return;
  GB_LAUNCH(bond_x_kernel, (unsigned) n, 128, 0, b, rc, n_elements, x);
}

void launch_bond_fwd(int lmax, const BondsDev &b, const LayerDev &L, float *Q, int NA, int a0, int na)
{
  if (na == 0) return;
  switch (lmax) {
    case 1: launch_l<1>(b, L, Q, NA, a0, na); break;
    case 2: launch_l<2>(b, L, Q, NA, a0, na); break;
    case 3: launch_l<3>(b, L, Q, NA, a0, na); break;
    case 4: launch_l<4>(b, L, Q, NA, a0, na); break;
    default: throw Unsupported("lmax must be 1..4");
  }
}

}    // namespace gb
