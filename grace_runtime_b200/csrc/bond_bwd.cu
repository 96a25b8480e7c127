// Reverse bond kernel: from gQ = dE/dQ of the central atom, per bond
//   S[I, l]   = sum_{m} Y_lm gQ[(I, lm)]                      dE/dR[l] = sum_I S[I, l] msg_I,  dE/dmsg_I = sum_l S[I, l] R[l]
//   dE/dx     = sum_{l, n} dE/dR[n, l] dR[n, l]/dx
//   g         = sum_{I, lm, n} gQ[(I, lm)][n] R[n, l] msg_I[n] grad Y_lm
//   f         = (dE/dx / rcut) rhat + (g - (g . rhat) rhat) / r          (force on i; -f on j)
// as bond_scatter_bwd_t / bond_yi_bwd_g / bond_dEdx_t / bond_force of the reference
// (libgrace/include/grace/fused_cpu.h:836-942, 1027-1050) and add_bond_virial (libgrace/src/fused_1l.cpp:45-51).
//
// One block of 4 warps per atom; a lane owns channel n and keeps gQ of its channel in registers; warps (half-warps
// for C <= 16) take the bonds in turn and reduce the four bond scalars over the channels by shuffles.  The bond force
// is stored at the bond's slot of the neighbour list (no atomics; forces are gathered afterwards through the
// reverse-bond index), the virial as one fp64 row per atom.  A bond's share of dE/dmsg of its neighbour goes to the
// bond's slot too and is summed per neighbour by msg_grad_gather_kernel (chain.cu); only when that buffer could not be
// allocated the shares are added with fp32 atomics, as the reference does.
#include "bond_common.cuh"

namespace gb {

namespace {

constexpr int EBB = 96;    // bonds staged per round: most atoms in one round, every thread of the block staging one bond

template<int LMAX, int NIT, int NCH, int LPE, bool EXACT>
__global__ void __launch_bounds__(128) bond_bwd_kernel(BondsDev b, LayerDev L, SHTable sht,
                                                       const float *__restrict__ gQ, int NA, int a0,
                                                       float *__restrict__ fv, double *__restrict__ vir_atom, int add)
{
  constexpr int NL = LMAX + 1, NLM = NL * NL, EPW = 32 / LPE;
  __shared__ float4 YG[EBB][NLM];
  __shared__ float su[EBB][4];     // rhat, r
  __shared__ float srci[EBB], st[EBB];
  __shared__ int sk[EBB], smu[EBB], sj[EBB], scs[EBB];
  __shared__ float fe[EBB][4];     // g (3), dE/dx
  __shared__ double vred[4][6];

  const int a = blockIdx.x, i = b.ilist ? b.ilist[a0 + a] : a0 + a, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int ln = lane % LPE, esub = lane / LPE;
  const long long base = b.off[i];
  const int nb = b.cnt[i];
  const int mui = b.mu[i];
  const int C = L.C, nel = L.n_elements;
  const int tiles = (L.n_msg + 1 + NIT - 1) / NIT;
  const float fN = (float) L.N;
  double vir[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};

  for (int b0 = 0; b0 < nb; b0 += EBB) {
    const int nbat = min(EBB, nb - b0);
    for (int e = tid; e < nbat; e += 128) {
      const float4 rec = b.rec[base + b0 + e];
      const float r = sqrtf(rec.x * rec.x + rec.y * rec.y + rec.z * rec.z), ir = 1.0f / r;
      const int j = __float_as_int(rec.w);
      const int muj = b.mu[j];
      const float rc = L.rc[mui * nel + muj];
      int k;
      float t;
      spline_locate(r / rc, L.N, k, t);
      sk[e] = k; st[e] = t; smu[e] = muj; sj[e] = j;
      scs[e] = b.cslot[base + b0 + e];
      srci[e] = 1.0f / rc;
      su[e][0] = rec.x * ir; su[e][1] = rec.y * ir; su[e][2] = rec.z * ir; su[e][3] = r;
      float4 *yg = YG[e];
      sph_harm<LMAX, true>(sht, rec.x * ir, rec.y * ir, rec.z * ir,
                           [&](int lm, float v, float gx, float gy, float gz) { yg[lm] = make_float4(v, gx, gy, gz); });
      fe[e][0] = fe[e][1] = fe[e][2] = fe[e][3] = 0.0f;
    }
    __syncthreads();
    for (int tile = 0; tile < tiles; tile++) {
      const int Ibase = tile * NIT;
      float g[NIT][NLM][NCH];
#pragma unroll
      for (int I = 0; I < NIT; I++)
#pragma unroll
        for (int q = 0; q < NLM; q++)
#pragma unroll
          for (int ch = 0; ch < NCH; ch++) {
            const int n = ln + ch * LPE;
            g[I][q][ch] = (n < C && Ibase + I <= L.n_msg)
                              ? __ldg(gQ + ((size_t) ((Ibase + I) * NLM + q) * NA + a) * C + n) : 0.0f;
          }
      for (int e0 = w * EPW; e0 < nbat; e0 += 4 * EPW) {
        const int e = e0 + esub;
        const bool valid = e < nbat;
        float gx = 0.0f, gy = 0.0f, gz = 0.0f, dedx = 0.0f;
        if (valid) {
          const int k = sk[e], muj = smu[e], j = sj[e];
          const float t = st[e];
          const float4 *yg = YG[e];
#pragma unroll
          for (int ch = 0; ch < NCH; ch++) {
            const int n = ln + ch * LPE;
            if (n < C) {
              float R[NL], dR[NL];
              if (EXACT) {    // exact radial MLP, evaluated per slot beforehand
                const size_t ro = (size_t) (base + b0 + e) * (NL * C) + n;
#pragma unroll
                for (int l = 0; l < NL; l++) {
                  R[l] = __ldg(L.Rex + ro + l * C);
                  dR[l] = __ldg(L.dRex + ro + l * C);
                }
              } else {
                const float4 *cf = reinterpret_cast<const float4 *>(L.tab) + (size_t) k * NL * C + n;
#pragma unroll
                for (int l = 0; l < NL; l++) {
                  const float4 c = __ldg(cf + l * C);
                  R[l] = c.x + t * (c.y + t * (c.z + t * c.w));
                  dR[l] = (c.y + t * (2.0f * c.z + t * 3.0f * c.w)) * fN;
                }
              }
              if constexpr (NIT == 1) {    // one message function per pass: nothing to contract first
                const int Ig = Ibase;
                float m = 0.0f;
                if (Ig < L.n_msg) m = __ldg(L.msg + ((size_t) j * L.n_msg + Ig) * C + n);
                else if (Ig == L.n_msg) m = __ldg(L.z + (size_t) muj * C + n);
                float gm = 0.0f;
#pragma unroll
                for (int l = 0; l < NL; l++) {
                  const float rm = R[l] * m;
                  float S = 0.0f;
#pragma unroll
                  for (int q = l * l; q < (l + 1) * (l + 1); q++) {
                    const float4 y4 = yg[q];
                    const float gq = g[0][q][ch];
                    S = fmaf(y4.x, gq, S);
                    const float p = gq * rm;
                    gx = fmaf(p, y4.y, gx);
                    gy = fmaf(p, y4.z, gy);
                    gz = fmaf(p, y4.w, gz);
                  }
                  dedx = fmaf(S * m, dR[l], dedx);
                  gm = fmaf(S, R[l], gm);
                }
                if (Ig < L.n_msg) {
                  if (L.gmsg_slot) L.gmsg_slot[((size_t) scs[e] * L.n_msg + Ig) * C + n] = gm;
                  else atomicAdd(L.gmsg + ((size_t) j * L.n_msg + Ig) * C + n, gm);
                }
              } else {
                // messages of this tile first, then one contraction over them per lm: h[q] = sum_I msg_I gQ[I][q] carries
                // everything dE/dx and the direction gradient need, so the harmonics are applied once per bond and
                // channel instead of once per message function
                float m[NIT];
  #pragma unroll
                for (int I = 0; I < NIT; I++) {
                  const int Ig = Ibase + I;
                  m[I] = 0.0f;
                  if (Ig < L.n_msg) m[I] = __ldg(L.msg + ((size_t) j * L.n_msg + Ig) * C + n);
                  else if (Ig == L.n_msg) m[I] = __ldg(L.z + (size_t) muj * C + n);
                }
  #pragma unroll
                for (int l = 0; l < NL; l++) {
                  float T = 0.0f, vx = 0.0f, vy = 0.0f, vz = 0.0f;
  #pragma unroll
                  for (int q = l * l; q < (l + 1) * (l + 1); q++) {
                    float h = 0.0f;
  #pragma unroll
                    for (int I = 0; I < NIT; I++) h = fmaf(m[I], g[I][q][ch], h);
                    const float4 y4 = yg[q];
                    T = fmaf(y4.x, h, T);
                    vx = fmaf(h, y4.y, vx);
                    vy = fmaf(h, y4.z, vy);
                    vz = fmaf(h, y4.w, vz);
                  }
                  dedx = fmaf(T, dR[l], dedx);
                  gx = fmaf(R[l], vx, gx);
                  gy = fmaf(R[l], vy, gy);
                  gz = fmaf(R[l], vz, gz);
                }
  #pragma unroll
                for (int I = 0; I < NIT; I++) {    // dE/dmsg_I = sum_l R_l sum_{m} Y_lm gQ[I][lm]
                  const int Ig = Ibase + I;
                  if (Ig < L.n_msg) {
                    float gm = 0.0f;
  #pragma unroll
                    for (int l = 0; l < NL; l++) {
                      float S = 0.0f;
  #pragma unroll
                      for (int q = l * l; q < (l + 1) * (l + 1); q++) S = fmaf(yg[q].x, g[I][q][ch], S);
                      gm = fmaf(S, R[l], gm);
                    }
                    if (L.gmsg_slot) L.gmsg_slot[((size_t) scs[e] * L.n_msg + Ig) * C + n] = gm;
                    else atomicAdd(L.gmsg + ((size_t) j * L.n_msg + Ig) * C + n, gm);
                  }
                }
              }
            }
          }
        }
        const float tot = group_sum4<LPE>(gx, gy, gz, dedx, ln);
        if (valid && (ln & (LPE / 4 - 1)) == 0) fe[e][ln / (LPE / 4)] += tot;    // one owner per bond, tile and component: no race
      }
      __syncthreads();
    }
    for (int e = tid; e < nbat; e += 128) {
      const float ux = su[e][0], uy = su[e][1], uz = su[e][2], r = su[e][3];
      const float gxx = fe[e][0], gyy = fe[e][1], gzz = fe[e][2];
      const float dEdr = fe[e][3] * srci[e];
      const float gr = gxx * ux + gyy * uy + gzz * uz, ir = 1.0f / r;
      const float f0 = dEdr * ux + (gxx - gr * ux) * ir;
      const float f1 = dEdr * uy + (gyy - gr * uy) * ir;
      const float f2 = dEdr * uz + (gzz - gr * uz) * ir;
      float *o = fv + 3 * (size_t) scs[e];
      if (add) { o[0] += f0; o[1] += f1; o[2] += f2; }
      else { o[0] = f0; o[1] = f1; o[2] = f2; }
      const double dx = -(double) ux * r, dy = -(double) uy * r, dz = -(double) uz * r;
      vir[0] += dx * f0; vir[1] += dy * f1; vir[2] += dz * f2;
      vir[3] += dx * f1; vir[4] += dx * f2; vir[5] += dy * f2;
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < 6; k++) {
    for (int s = 16; s > 0; s >>= 1) vir[k] += __shfl_xor_sync(0xffffffffu, vir[k], s);
    if (lane == 0) vred[w][k] = vir[k];
  }
  __syncthreads();
  if (tid < 6) {
    const double v = vred[0][tid] + vred[1][tid] + vred[2][tid] + vred[3][tid];
    double *o = vir_atom + 6 * (size_t) i + tid;
    *o = add ? *o + v : v;
  }
}

// What the kernels with two channels per lane stage per bond.  A row holds (y y gx gx) (gy gy gz gz) per harmonic, an odd number
// of 16-byte words so that the threads which write the rows of different bonds meet no bank conflict.
template<int ROW, int EB> struct BwdStage {
  float4 Y[EB][ROW];
  float4 u[EB], fe[EB];    // rhat, r;  g, dE/dx
  int4 meta[EB];           // interval, element, offset, neighbour
  float scale[EB];         // intervals per length: N / rcut of the pair
  int cs[EB];
  double vred[4][6];
};

template<int LMAX, class S, class Place>
__device__ __forceinline__ void bwd_stage(S &s, int e, const BondsDev &b, const LayerDev &L, const SHTable &sht, long long slot, int mui, Place place)
{
  const float4 rec = b.rec[slot];
  const float r = sqrtf(rec.x * rec.x + rec.y * rec.y + rec.z * rec.z), ir = 1.0f / r;
  const int j = __float_as_int(rec.w), muj = b.mu[j];
  const float rc = L.rc[mui * L.n_elements + muj];
  int k;
  float t;
  spline_locate(r / rc, L.N, k, t);
  s.meta[e] = make_int4(k, muj, __float_as_int(t), j);
  s.cs[e] = b.cslot[slot];
  s.scale[e] = (float) L.N / rc;
  s.u[e] = make_float4(rec.x * ir, rec.y * ir, rec.z * ir, r);
  float4 *y = s.Y[e];
  sph_harm<LMAX, true>(sht, rec.x * ir, rec.y * ir, rec.z * ir, [&](int lm, float v, float gx, float gy, float gz) {
    const int at = place(lm);
    y[at] = make_float4(v, v, gx, gx);
    y[at + 1] = make_float4(gy, gy, gz, gz);
  });
}

// bond force to its slot, virial of the bonds this thread finishes
template<class S>
__device__ __forceinline__ void bwd_finish(const S &s, int e, float *__restrict__ fv, int add, double (&vir)[6])
{
  const float4 u = s.u[e], g = s.fe[e];
  const float dEdr = g.w * s.scale[e], gr = g.x * u.x + g.y * u.y + g.z * u.z, ir = 1.0f / u.w;
  const float f0 = dEdr * u.x + (g.x - gr * u.x) * ir;
  const float f1 = dEdr * u.y + (g.y - gr * u.y) * ir;
  const float f2 = dEdr * u.z + (g.z - gr * u.z) * ir;
  float *o = fv + 3 * (size_t) s.cs[e];
  if (add) { o[0] += f0; o[1] += f1; o[2] += f2; }
  else { o[0] = f0; o[1] = f1; o[2] = f2; }
  const double dx = -(double) u.x * u.w, dy = -(double) u.y * u.w, dz = -(double) u.z * u.w;
  vir[0] += dx * f0; vir[1] += dy * f1; vir[2] += dz * f2;
  vir[3] += dx * f1; vir[4] += dx * f2; vir[5] += dy * f2;
}

__device__ __forceinline__ void bwd_virial(double (&vred)[4][6], double (&vir)[6], double *__restrict__ vir_atom, int i, int add)
{
  const int tid = threadIdx.x;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    for (int s = 16; s > 0; s >>= 1) vir[k] += __shfl_xor_sync(0xffffffffu, vir[k], s);
    if ((tid & 31) == 0) vred[tid >> 5][k] = vir[k];
  }
  __syncthreads();
  if (tid < 6) {
    const double v = vred[0][tid] + vred[1][tid] + vred[2][tid] + vred[3][tid];
    double *o = vir_atom + 6 * (size_t) i + tid;
    *o = add ? *o + v : v;
  }
}

// Blocks per SM the kernels are compiled for, and bonds per round: as many as fit the shared memory of that many blocks, at most
// one per thread (lmax 3: 97 and, with messages, 124; lmax 4: 65 and 115).  They wait for the table and for shared memory most of the
// time: warps in flight count for more than a few spilled registers.  An atom that needs a second round pays two more barriers;
// that the larger stage leaves less L1 does not show.  ns per bond at 60, 83, 94 and 104 neighbours, lmax 3: 0.300, 0.279, 0.258, 0.276
// (with 78 bonds 0.301, 0.319, 0.303, 0.292, with 64 0.301, 0.321, 0.303, 0.292), with messages 0.470, 0.440, 0.407, 0.406 (80 bonds
// 0.468, 0.460, 0.461, 0.447); lmax 4 at 60, 66, 73 and 81: 0.404, 0.375, 0.348, 0.381 (60 bonds 0.404, 0.407, 0.388, 0.385).
constexpr size_t SM_SHARED = 228 * 1024, BLOCK_RESERVED = 1024;
template<int ROW> __host__ __device__ constexpr int stage_bonds(int blocks)
{
  constexpr size_t fixed = sizeof(BwdStage<ROW, 1>) - (sizeof(BwdStage<ROW, 17>) - sizeof(BwdStage<ROW, 1>)) / 16;    // 16 bonds: no padding
  constexpr size_t per = (sizeof(BwdStage<ROW, 17>) - sizeof(BwdStage<ROW, 1>)) / 16;
  const size_t n = (SM_SHARED / blocks - BLOCK_RESERVED - fixed) / per;
  return n < 128 ? (int) n : 128;
}
template<int LMAX> __host__ __device__ constexpr int pair_blocks() { return 4; }
template<int LMAX> __host__ __device__ constexpr int msg_blocks() { return LMAX <= 3 ? 3 : 2; }
// The four 16-byte words a load instruction of the message kernel reads, (bond, group of harmonics), lie in different banks: the
// groups are an odd number of words apart and the bonds three.
template<int LMAX> __host__ __device__ constexpr int msg_half() { return 2 * LmSplit<LMAX>::NK + 1; }
template<int LMAX> __host__ __device__ constexpr int msg_row() { return 2 * msg_half<LMAX>() + (8 + 3 - 2 * msg_half<LMAX>() % 8) % 8; }
template<int LMAX> __host__ __device__ constexpr int pair_row() { return 2 * (LMAX + 1) * (LMAX + 1) + 1; }
template<int LMAX> __host__ __device__ constexpr int pair_bonds() { return stage_bonds<pair_row<LMAX>()>(pair_blocks<LMAX>()); }
template<int LMAX> __host__ __device__ constexpr int msg_bonds() { return stage_bonds<msg_row<LMAX>()>(msg_blocks<LMAX>()); }
template<int LMAX> using PairStage = BwdStage<pair_row<LMAX>(), pair_bonds<LMAX>()>;
template<int LMAX> using MsgStage = BwdStage<msg_row<LMAX>(), msg_bonds<LMAX>()>;
static_assert(pair_bonds<3>() == 97 && msg_bonds<3>() == 124 && pair_bonds<4>() == 65 && msg_bonds<4>() == 115, "");
static_assert(4 * (sizeof(PairStage<3>) + BLOCK_RESERVED) <= SM_SHARED && 3 * (sizeof(MsgStage<3>) + BLOCK_RESERVED) <= SM_SHARED, "");
static_assert(4 * (sizeof(PairStage<4>) + BLOCK_RESERVED) <= SM_SHARED && 2 * (sizeof(MsgStage<4>) + BLOCK_RESERVED) <= SM_SHARED, "");

// Layers without message functions and with an even number of channels: LPB lanes per bond, two channels per lane, 32 / LPB
// bonds per warp at a time, with the gradients of its channels in a lane's registers.  With the chemical weight folded into
// the radial functions a harmonic costs four packed FMAs per lane and bond.  Bound by the shared-memory reads of the harmonics
// and, at 16 warps per SM, by their latency.  Against one channel per lane: GRACE-2L, 1,024,000 atoms, lmax 3: 29.9 -> 23.0 ms;
// GRACE-1L, 128,000 atoms, lmax 4: 3.81 -> 3.10 ms.
template<int LMAX, int LPB>
__global__ void __launch_bounds__(128, pair_blocks<LMAX>()) bond_bwd_pair_kernel(BondsDev b, LayerDev L, SHTable sht, const float *__restrict__ gQ, int NA, int a0,
                                                            float *__restrict__ fv, double *__restrict__ vir_atom, int add)
{
  constexpr int NL = LMAX + 1, NLM = NL * NL, BPW = 32 / LPB, EB = pair_bonds<LMAX>();
  extern __shared__ __align__(16) char smem[];
  PairStage<LMAX> &s = *reinterpret_cast<PairStage<LMAX> *>(smem);
  const int a = blockIdx.x, i = b.ilist ? b.ilist[a0 + a] : a0 + a, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int c = lane % LPB, sub = lane / LPB;
  const long long base = b.off[i];
  const int nb = b.cnt[i], mui = b.mu[i], C = L.C, C2 = C >> 1;
  const int rounds = max(1, (nb + EB - 1) / EB), per = (nb + rounds - 1) / rounds;
  double vir[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  float2 g[NLM];
#pragma unroll
  for (int q = 0; q < NLM; q++)
    g[q] = c < C2 ? __ldg(reinterpret_cast<const float2 *>(gQ + ((size_t) q * NA + a) * C) + c) : make_float2(0.f, 0.f);

  for (int b0 = 0; b0 < nb; b0 += per) {
    const int nbat = min(per, nb - b0);
    for (int e = tid; e < nbat; e += 128) bwd_stage<LMAX>(s, e, b, L, sht, base + b0 + e, mui, [](int lm) { return 2 * lm; });
    __syncthreads();
    for (int e0 = w * BPW; e0 < nbat; e0 += 4 * BPW) {
      const int e = e0 + sub;
      float2 gx = make_float2(0.f, 0.f), gy = gx, gz = gx, dedx = gx;
      if (e < nbat && c < C2) {
        const int4 m = s.meta[e];
        const float tt = __int_as_float(m.z);
        const float2 t = pair_of(tt), t_2 = pair_of(2.0f * tt), t_15 = pair_of(1.5f * tt);
        const float4 *cf = reinterpret_cast<const float4 *>(L.tab) + (size_t) m.x * NL * C + c;
        const float2 z = __ldg(reinterpret_cast<const float2 *>(L.z + (size_t) m.y * C) + c);
        const float4 *y = s.Y[e];
#pragma unroll
        for (int l = 0; l < NL; l++) {
          const float4 xy = __ldg(cf + l * C), zw = __ldg(cf + l * C + C2);
          float2 T = make_float2(0.f, 0.f), vx = T, vy = T, vz = T;
#pragma unroll
          for (int q = l * l; q < (l + 1) * (l + 1); q++) {
            const float4 A = y[2 * q], B = y[2 * q + 1];
            T = __ffma2_rn(lo2(A), g[q], T);
            vx = __ffma2_rn(hi2(A), g[q], vx);
            vy = __ffma2_rn(lo2(B), g[q], vy);
            vz = __ffma2_rn(hi2(B), g[q], vz);
          }
          const float2 R = pair_value(xy, zw, t);
          dedx = __ffma2_rn(T, pair_slope(xy, zw, t_2, t_15), dedx);
          gx = __ffma2_rn(R, vx, gx);
          gy = __ffma2_rn(R, vy, gy);
          gz = __ffma2_rn(R, vz, gz);
        }
        gx = __fmul2_rn(gx, z);
        gy = __fmul2_rn(gy, z);
        gz = __fmul2_rn(gz, z);
        dedx = __fmul2_rn(dedx, z);
      }
      const float tot = group_sum4<LPB>(gx.x + gx.y, gy.x + gy.y, gz.x + gz.y, dedx.x + dedx.y, c);
      if (e < nbat && (c & (LPB / 4 - 1)) == 0) reinterpret_cast<float *>(s.fe + e)[c / (LPB / 4)] = tot;
    }
    __syncthreads();
    for (int e = tid; e < nbat; e += 128) bwd_finish(s, e, fv, add, vir);
    __syncthreads();
  }
  bwd_virial(s.vred, vir, vir_atom, i, add);
}

// Layers with four message functions and at most 16 channels (an even number): 16 lanes per bond, lane = (group h of
// harmonics, channel pair c), two bonds per warp at a time; the gradients of 5 message functions x NK harmonics x two channels
// in a lane's registers.  Per harmonic the lane forms h = sum_I msg_I gQ[I][lm] once; with R and dR/dx of the harmonic's degree
// everything is linear in h:
//   dE/dx += dR_l Y_lm h,   g += R_l h grad Y_lm,   dE/dmsg_I += R_l Y_lm gQ[I][lm].
// One channel per lane took 447 issued instructions per bond and was bound by them; this takes 228, at 12 warps per SM (168
// registers; compiled for 16 warps it spills: 43 ms).  GRACE-2L, 1,024,000 atoms: 53.8 -> 36.7 ms.
template<int LMAX>
__global__ void __launch_bounds__(128, msg_blocks<LMAX>()) bond_bwd_msg_kernel(BondsDev b, LayerDev L, SHTable sht, const float *__restrict__ gQ, int NA, int a0,
                                                           float *__restrict__ fv, double *__restrict__ vir_atom, int add)
{
  using SP = LmSplit<LMAX>;
  constexpr int NL = LMAX + 1, NLM = NL * NL, NI = 5, NK = SP::NK, EB = msg_bonds<LMAX>(), HALF = msg_half<LMAX>();
  extern __shared__ __align__(16) char smem[];
  MsgStage<LMAX> &s = *reinterpret_cast<MsgStage<LMAX> *>(smem);
  const int a = blockIdx.x, i = b.ilist ? b.ilist[a0 + a] : a0 + a, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int c = lane & 7, h = (lane >> 3) & 1, sub = lane >> 4;
  const long long base = b.off[i];
  const int nb = b.cnt[i], mui = b.mu[i], C = L.C, C2 = C >> 1;
  const int rounds = max(1, (nb + EB - 1) / EB), per = (nb + rounds - 1) / rounds;
  double vir[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  float2 g[NI][NK];
#pragma unroll
  for (int k = 0; k < NK; k++) {
    const int q = h ? SP::lm(1, k) : SP::lm(0, k);
#pragma unroll
    for (int I = 0; I < NI; I++)
      g[I][k] = q >= 0 && c < C2 ? __ldg(reinterpret_cast<const float2 *>(gQ + ((size_t) (I * NLM + q) * NA + a) * C) + c)
                                 : make_float2(0.f, 0.f);
  }

  for (int b0 = 0; b0 < nb; b0 += per) {
    const int nbat = min(per, nb - b0);
    for (int e = tid; e < nbat; e += 128) {
      constexpr LmPlaces<LMAX> places;
      bwd_stage<LMAX>(s, e, b, L, sht, base + b0 + e, mui, [&](int lm) {
        const int at = places.v[lm];
        return at < NK ? 2 * at : HALF + 2 * (at - NK);
      });
#pragma unroll
      for (int hk = 0; hk < 2 * NK; hk++)    // positions without a harmonic
        if (SP::lm(hk / NK, hk % NK) < 0) {
          float4 *none = s.Y[e] + hk / NK * HALF + hk % NK * 2;
          none[0] = none[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __syncthreads();
    for (int e0 = 2 * w; e0 < nbat; e0 += 8) {
      const int e = e0 + sub;
      const bool work = e < nbat && c < C2;
      float2 gx = make_float2(0.f, 0.f), gy = gx, gz = gx, dedx = gx, gm[4] = {gx, gx, gx, gx};
      int j = 0;
      if (work) {
        const int4 m = s.meta[e];
        j = m.w;
        const float tt = __int_as_float(m.z);
        const float2 t = pair_of(tt), t_2 = pair_of(2.0f * tt), t_15 = pair_of(1.5f * tt);
        const float4 *cf = reinterpret_cast<const float4 *>(L.tab) + (size_t) m.x * NL * C + c;
        const float2 *msg = reinterpret_cast<const float2 *>(L.msg + (size_t) j * 4 * C) + c;
        float2 R[SP::NS], dR[SP::NS], mm[NI];
#pragma unroll
        for (int q = 0; q < SP::NS; q++) {
          constexpr auto some = [](int l) { return l < 0 ? 0 : l; };
          const int l = h ? some(SP::degree(1, q)) : some(SP::degree(0, q));
          const float4 xy = __ldg(cf + l * C), zw = __ldg(cf + l * C + C2);
          R[q] = pair_value(xy, zw, t);
          dR[q] = pair_slope(xy, zw, t_2, t_15);
        }
#pragma unroll
        for (int I = 0; I < 4; I++) mm[I] = __ldg(msg + I * C2);
        mm[4] = __ldg(reinterpret_cast<const float2 *>(L.z + (size_t) m.y * C) + c);
        const float4 *y = s.Y[e] + h * HALF;
#pragma unroll
        for (int k = 0; k < NK; k++) {
          constexpr auto bound = [](int q) { return q < SP::NS ? q : SP::NS - 1; };
          const int s0 = bound(SP::slot(0, k)), s1 = bound(SP::slot(1, k));
          const float2 Rk = s0 == s1 ? R[s0] : h ? R[s1] : R[s0], dRk = s0 == s1 ? dR[s0] : h ? dR[s1] : dR[s0];
          const float4 A = y[2 * k], B = y[2 * k + 1];
          float2 hq = __fmul2_rn(mm[0], g[0][k]);
#pragma unroll
          for (int I = 1; I < NI; I++) hq = __ffma2_rn(mm[I], g[I][k], hq);
          const float2 p = __fmul2_rn(Rk, hq), ry = __fmul2_rn(Rk, lo2(A));
          dedx = __ffma2_rn(__fmul2_rn(dRk, lo2(A)), hq, dedx);
          gx = __ffma2_rn(p, hi2(A), gx);
          gy = __ffma2_rn(p, lo2(B), gy);
          gz = __ffma2_rn(p, hi2(B), gz);
#pragma unroll
          for (int I = 0; I < 4; I++) gm[I] = __ffma2_rn(ry, g[I][k], gm[I]);
        }
      }
      // dE/dmsg: each group of harmonics takes two of the message functions and gets the other group's part of them
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const float2 give = h ? gm[q] : gm[2 + q];
        float2 keep = h ? gm[2 + q] : gm[q];
        keep.x += __shfl_xor_sync(0xffffffffu, give.x, 8);
        keep.y += __shfl_xor_sync(0xffffffffu, give.y, 8);
        if (work) {
          const int at = (2 * h + q) * C + 2 * c;
          if (L.gmsg_slot) *reinterpret_cast<float2 *>(L.gmsg_slot + (size_t) s.cs[e] * 4 * C + at) = keep;
          else {
            atomicAdd(L.gmsg + (size_t) j * 4 * C + at, keep.x);
            atomicAdd(L.gmsg + (size_t) j * 4 * C + at + 1, keep.y);
          }
        }
      }
      const float tot = group_sum4<16>(gx.x + gx.y, gy.x + gy.y, gz.x + gz.y, dedx.x + dedx.y, lane & 15);
      if (e < nbat && (lane & 3) == 0) reinterpret_cast<float *>(s.fe + e)[(lane & 15) >> 2] = tot;
    }
    __syncthreads();
    for (int e = tid; e < nbat; e += 128) bwd_finish(s, e, fv, add, vir);
    __syncthreads();
  }
  bwd_virial(s.vred, vir, vir_atom, i, add);
}

template<class Stage, class F> size_t pair_smem(F *kernel, size_t &attr)
{
  const size_t n = sizeof(Stage);
  if (n > attr) {
    GB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) n));
    attr = n;
  }
  return n;
}

template<int LMAX, int LPB>
void launch_pair(const BondsDev &b, const LayerDev &L, const float *gQ, int NA, int a0, int na, float *fv, double *vir_atom, int add)
{
  static size_t attr = 48 * 1024;
  const size_t smem = pair_smem<PairStage<LMAX>>(bond_bwd_pair_kernel<LMAX, LPB>, attr);
  GB_LAUNCH((bond_bwd_pair_kernel<LMAX, LPB>), na, 128, smem, b, L, sh_table_host(), gQ, NA, a0, fv, vir_atom, add);
}

template<int LMAX, int NIT, int NCH, int LPE>
void launch_t(const BondsDev &b, const LayerDev &L, const float *gQ, int NA, int a0, int na, float *fv,
              double *vir_atom, int add)
{
  if (L.Rex) GB_LAUNCH((bond_bwd_kernel<LMAX, NIT, NCH, LPE, true>), na, 128, 0, b, L, sh_table_host(), gQ, NA, a0, fv, vir_atom, add);
  else GB_LAUNCH((bond_bwd_kernel<LMAX, NIT, NCH, LPE, false>), na, 128, 0, b, L, sh_table_host(), gQ, NA, a0, fv, vir_atom, add);
}

template<int LMAX>
void launch_l(const BondsDev &b, const LayerDev &L, const float *gQ, int NA, int a0, int na, float *fv,
              double *vir_atom, int add)
{
  const int C = L.C, nI = L.n_msg + 1;
  if (C > 64) throw Unsupported("bond sums with more than 64 channels are not supported");
  if (L.pairs) {
    if (L.n_msg) {
      static size_t attr = 48 * 1024;
      const size_t smem = pair_smem<MsgStage<LMAX>>(bond_bwd_msg_kernel<LMAX>, attr);
      GB_LAUNCH(bond_bwd_msg_kernel<LMAX>, na, 128, smem, b, L, sh_table_host(), gQ, NA, a0, fv, vir_atom, add);
    } else if (C > 32) launch_pair<LMAX, 32>(b, L, gQ, NA, a0, na, fv, vir_atom, add);
    else if (C > 16) launch_pair<LMAX, 16>(b, L, gQ, NA, a0, na, fv, vir_atom, add);
    else launch_pair<LMAX, 8>(b, L, gQ, NA, a0, na, fv, vir_atom, add);
    return;
  }
  if (C > 32) launch_t<LMAX, 1, 2, 32>(b, L, gQ, NA, a0, na, fv, vir_atom, add);
  else if (C > 16) { if (nI == 5) launch_t<LMAX, 5, 1, 32>(b, L, gQ, NA, a0, na, fv, vir_atom, add); else launch_t<LMAX, 1, 1, 32>(b, L, gQ, NA, a0, na, fv, vir_atom, add); }
  else { if (nI == 5) launch_t<LMAX, 5, 1, 16>(b, L, gQ, NA, a0, na, fv, vir_atom, add); else launch_t<LMAX, 1, 1, 16>(b, L, gQ, NA, a0, na, fv, vir_atom, add); }
}

}    // namespace

void launch_bond_bwd(int lmax, const BondsDev &b, const LayerDev &L, const float *gQ, int NA, int a0, int na,
                     float *fv, double *vir_atom, int add)
{
  if (na == 0) return;
  switch (lmax) {
    case 1: launch_l<1>(b, L, gQ, NA, a0, na, fv, vir_atom, add); break;
    case 2: launch_l<2>(b, L, gQ, NA, a0, na, fv, vir_atom, add); break;
    case 3: launch_l<3>(b, L, gQ, NA, a0, na, fv, vir_atom, add); break;
    case 4: launch_l<4>(b, L, gQ, NA, a0, na, fv, vir_atom, add); break;
    default: throw Unsupported("lmax must be 1..4");
  }
}

}    // namespace gb
