// GRACE-3L evaluation: three message-passing layers (libgrace/src/fused_3l.cpp:1204-1637).  Per layer: the bond sums of
// the single-particle basis (per-pair radial tables, spherical harmonics, the normalised message of the layer before
// coupled in through the sparse cg_W), the dense chain of the layer as MV / PROD operations of the plan (cp_l
// projections, couples, reduces, FCs: the same kernels as GRACE-1L / 2L), EquivariantRMSNorm of the message and RMSNorm
// of the density; the readout on the sum of the three densities; then everything in reverse.  While they fit, the
// tensors of the three layers of all atoms are kept for the reverse pass; larger structures run every layer in passes
// over atom chunks and recompute a chunk's forward tensors when it is reversed.  Checked
// against the reference's CPU engine.
#include "engine.h"

#include "bond_common.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

namespace gb {

namespace {

struct Spbf3Dev {
  const float *tab;          // [pair][N][nl][C][4] cubic Hermite coefficients
  const int *pair_slot;      // [n_elements^2] table of the element pair (centre, neighbour), -1: none
  long long tab_stride;      // floats per pair
  const float *rc;           // [n_elements^2]
  const float *msg;          // [n][nlmi][C] normalised message of the layer before (null: layer 1)
  float *gmsg;               // [n][nlmi][C] its gradient, added to atomically (null: layer 1)
  const float *zproj;        // [n_elements][C]
  const float *l0mask;       // [nlmi]
  // the couple as flat lists, one after the other for each round and warp (s3_list): cg in the order of the output
  // functions, cgt in the order of the (harmonic, message function) pairs of the warp
  const int2 *cg, *cgt;
  const int *cg_off, *cgt_off;    // where the list of (round, warp) starts, [rounds warps + 1]
  int N, C, nl, nlm, nlmi, nfA, nel;
};


constexpr int S3_BB = 64;     // bonds whose harmonics and geometry are staged at once
constexpr int S3_NBS = 4;     // bonds whose radial functions and messages travel together
constexpr int S3_LIT = 7;     // message functions of a thread
constexpr int S3_WARPS = 4;   // most warps of a CTA
// warps of a CTA, and the message functions it holds at a time
int s3_warps(int nlmi) { return nlmi == 1 ? 4 : std::min(S3_WARPS, (nlmi + S3_LIT - 1) / S3_LIT); }
int s3_pitch(int nlmi) { return nlmi == 1 ? 1 : s3_warps(nlmi) * S3_LIT; }

__device__ __forceinline__ void s3_cp16(void *dst_smem, const void *src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned) __cvta_generic_to_shared(dst_smem)), "l"(src) : "memory");
}
__device__ __forceinline__ void s3_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void s3_cp_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Geometry of a bond, worked out once per batch of bonds by one thread per bond (a chain of dependent global loads: record
// -> element of the neighbour -> table of the pair) and kept in shared memory.
struct __align__(16) S3Bond {
  long long tab;    // offset of the bond's table row in floats, < 0: no table for this element pair, the bond is left out
  long long row;    // offset of the neighbour's message row in floats
  int muj;
  float t, r, rc;
};
__device__ __forceinline__ S3Bond s3_bond(const BondsDev &b, const Spbf3Dev &L, const float4 &rec, int mui)
{
  S3Bond o;
  const int j = __float_as_int(rec.w);
  o.muj = b.mu[j];
  o.r = sqrtf(rec.x * rec.x + rec.y * rec.y + rec.z * rec.z);
  o.rc = L.rc[mui * L.nel + o.muj];
  int k0;
  spline_locate(o.r / o.rc, L.N, k0, o.t);
  const int slot = L.pair_slot[mui * L.nel + o.muj];
  o.tab = slot < 0 ? -1 : (long long) slot * L.tab_stride + (long long) k0 * L.nl * L.C * 4;
  o.row = (long long) j * L.nlmi * L.C;
  return o;
}

// Bond sums of GRACE-3L and their reverse.  With U[ly] = Y_ly R_l(ly)[c] and I[li] = msg_j[li][c] + mask[li] zproj[mu_j][c] a
// channel c of an atom is a small outer-product sum over the bonds j,
//     P[ly][li] = sum_j U[ly] I[li]         (forward),
//     W[ly] = sum_li gP[ly][li] I[li],  dE/dmsg_j[li] = sum_ly gP[ly][li] U[ly]      (reverse, per bond),
// 625 multiply-adds per bond and channel at lmax 4 (three times that in reverse).  A CTA works on one atom and 32 channels,
// lane = channel; a warp owns 7 message functions and ALL harmonics of them, so that a thread keeps 25 x 7 sums (or their
// gradient) in registers and one bond costs it 7 messages, 5 radial values and the harmonics (16-byte broadcast reads) for
// 175 multiply-adds (350 in reverse), where tiles of 5 x 5 over 25 warps needed 10 shared-memory reads for 25.  That fills
// the register file with two warps per scheduler, balanced over the four of them; what the bonds need travels by asynchronous
// copies a group of bonds ahead, and the number of instructions is what counts: no index arithmetic per bond, the couple as
// flat lists read eight entries at a time, and in reverse pairs of harmonics through two-wide multiply-adds (forward they
// gain nothing: the compiler copies the paired sums apart in every iteration).
// A layer without messages has one function: the warps share the bonds instead (LIT = 1).
// 31,250 atoms, lmax 4, 64 channels, three layers (ms per evaluation, forward / reverse): tiles of 5 x 5 with staged operands
// 84.6 / 260; 5 functions per warp, couple term by term 43.4 / 87.9; this form 26.3 / 72.2.

template<int LMAX> struct S3 {
  static constexpr int NLM = (LMAX + 1) * (LMAX + 1), NL = LMAX + 1, NP = (NLM + 1) / 2;    // NP: pairs of harmonics
  static constexpr int YLD = (NP + 1) / 2 * 4;                                             // floats of a bond's harmonics
  __host__ __device__ static constexpr int l_of(int lm) { return lm < 1 ? 0 : lm < 4 ? 1 : lm < 9 ? 2 : lm < 16 ? 3 : 4; }
};

// Radial functions (and derivatives) of the bonds of a group: a thread owns one channel of the functions l = warp, warp +
// nw, ..; the coefficients travel to its own piece of `raw` by asynchronous copies issued a group ahead.  tabc: the table
// from the thread's channel on.
template<int NL>
__device__ __forceinline__ void s3_issue(const float *tabc, int C, const S3Bond *meta, int ns, float4 *raw, int warp, int nw, int lane)
{
  for (int l = warp; l < NL; l += nw)
#pragma unroll
    for (int s = 0; s < S3_NBS; s++)
      if (s < ns) s3_cp16(raw + (s * NL + l) * 32 + lane, tabc + max(meta[s].tab, 0LL) + 4 * l * C);
  s3_cp_commit();
}
template<int NL, bool GRAD>
__device__ __forceinline__ void s3_radial(float N, const S3Bond *meta, int ns, const float4 *raw, float *R, float *dR, int warp, int nw,
                                          int lane)
{
  for (int l = warp; l < NL; l += nw)
#pragma unroll
    for (int s = 0; s < S3_NBS; s++) {
      if (s >= ns) break;
      const int e = (s * NL + l) * 32 + lane;
      const float4 cf = raw[e];
      const float t = meta[s].t;
      const bool have = meta[s].tab >= 0;
      R[e] = have ? cf.x + t * (cf.y + t * (cf.z + t * cf.w)) : 0.0f;
      if (GRAD) dR[e] = have ? (cf.y + t * (2.0f * cf.z + t * 3.0f * cf.w)) * N : 0.0f;
    }
}

// The warp's part of the message rows of a group of bonds: LIT functions (and the chemical weights, where the mask asks for
// them) of 32 channels, by asynchronous copies into shared memory of the warp's own, a group ahead of their use.  Functions
// beyond the model's repeat the last one; channels beyond the layer's (16 or 48 channels: half of the last slice) are not copied,
// and in the reverse pass, which adds over the lanes, the lanes that have none get zeros in place of what lies there.
template<int LIT> struct S3Msg {
  static constexpr int ROWS = LIT + 1, GROUP = S3_NBS * ROWS * 32;    // floats of a group
  float mask[LIT];
  bool masked;
  __device__ void setup(const Spbf3Dev &L, int li0)
  {
    masked = false;
#pragma unroll
    for (int q = 0; q < LIT; q++) {
      mask[q] = li0 + q < L.nlmi ? L.l0mask[li0 + q] : 0.0f;
      masked = masked || mask[q] != 0.0f;
    }
  }
  // chunk of 4 channels (lane & 7) of the rows lane >> 3, lane >> 3 + 4, ..
  __device__ __forceinline__ void issue(const Spbf3Dev &L, const S3Bond *meta, int ns, int li0, int c0, float *buf, int lane) const
  {
    const int k = 4 * (lane & 7), r0 = lane >> 3;
    if (c0 + k >= L.C) return;
#pragma unroll
    for (int s = 0; s < S3_NBS; s++) {
      if (s >= ns) break;
      const S3Bond &B = meta[s];
      const float *m = L.msg + B.row + c0 + k;
#pragma unroll
      for (int r = 0; r < ROWS; r += 4) {
        const int row = r + r0;
        if (row < LIT && L.msg) s3_cp16(buf + (s * ROWS + row) * 32 + k, m + min(li0 + row, L.nlmi - 1) * L.C);
        else if (row == LIT && masked) s3_cp16(buf + (s * ROWS + row) * 32 + k, L.zproj + B.muj * L.C + c0 + k);
      }
    }
  }
  // have: the layer has messages; in: the lane has a channel, or what it computes goes nowhere
  __device__ __forceinline__ void get(const float *buf, int s, bool have, bool in, int lane, float (&ic)[LIT]) const
  {
#pragma unroll
    for (int q = 0; q < LIT; q++) ic[q] = have && in ? buf[(s * ROWS + q) * 32 + lane] : 0.0f;
    if (masked) {    // the same for the whole warp
      const float z = in ? buf[(s * ROWS + LIT) * 32 + lane] : 0.0f;
#pragma unroll
      for (int q = 0; q < LIT; q++) ic[q] = fmaf(mask[q], z, ic[q]);
    }
  }
};

// A flat list of the couple: entries (source row | target + 1 << 16 where the target's sum ends, coefficient); target[32 lane]
// of the sums go to `out`.  Eight entries at a time: their reads are in flight together, where a loop over the terms of one
// target after the other is a chain of dependent reads (a third of the forward kernel's time).
template<class Out>
__device__ __forceinline__ void s3_list(const int2 *__restrict__ list, int k0, int k1, const float *src, int lane, Out &&out)
{
  float v = 0.0f;
  for (int k = k0; k < k1; k += 8) {
    int2 t[8];
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; u++) t[u] = __ldg(list + min(k + u, k1 - 1));
#pragma unroll
    for (int u = 0; u < 8; u++) x[u] = src[(t[u].x & 0xffff) * 32 + lane];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      if (k + u >= k1) break;
      v = fmaf(__int_as_float(t[u].y), x[u], v);
      if (t[u].x >> 16) {
        out((t[u].x >> 16) - 1, v);
        v = 0.0f;
      }
    }
  }
}

// pairs of fp32 values in a 64-bit register, for the two-wide multiply-add (as float2 the accumulators of a loop are copied
// apart and together again)
typedef unsigned long long s3_pair;
__device__ __forceinline__ s3_pair s3_pack(float x, float y)
{
  s3_pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void s3_fma(s3_pair &d, s3_pair a, s3_pair b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ s3_pair s3_mul(s3_pair a, s3_pair b)
{
  s3_pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ s3_pair s3_dup(float v) { return s3_pack(v, v); }
__device__ __forceinline__ float s3_sum(s3_pair p)
{
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(p));
  return x + y;
}

// A[f][a][c] = sum_q cg[q, f] P[q][c]
template<int LMAX, int LIT>
__global__ void __launch_bounds__(32 * S3_WARPS, 2) spbf3_fwd_kernel(BondsDev b, Spbf3Dev L, SHTable sht, float *__restrict__ A, int NA,
                                                                     int a0)
{
  constexpr int NLM = S3<LMAX>::NLM, NL = S3<LMAX>::NL, YLD = S3<LMAX>::YLD;
  extern __shared__ __align__(16) float sm[];
  float *Ps = sm;                                                  // [nlm][functions of a round][32], after the bond loop
  float4 *raw = reinterpret_cast<float4 *>(sm);                    // during it: [NBS][nl][32]
  float *Rs = sm + 4 * S3_NBS * NL * 32;                           // [2][NBS][nl][32]
  float *Ys = Rs + 2 * S3_NBS * NL * 32;                           // [BB][YLD]
  S3Bond *meta = reinterpret_cast<S3Bond *>(Ys + S3_BB * YLD);     // [BB]
  const int nth = blockDim.x, nw = nth >> 5, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float *msg = reinterpret_cast<float *>(meta + S3_BB) + warp * 2 * S3Msg<LIT>::GROUP;    // [2] groups of the warp
  const int C = L.C, slices = (C + 31) / 32, ap = blockIdx.x / slices, i = a0 + ap, c0 = blockIdx.x % slices * 32, c = c0 + lane;
  const long long base = b.off[i];
  const int nb = b.cnt[i], mui = b.mu[i];
  const int pitch = LIT == 1 ? 1 : nw * LIT, nround = (L.nlmi + pitch - 1) / pitch;
  const float *tabc = L.tab + 4 * min(c, C - 1);
  for (int round = 0; round < nround; round++) {
    const int li0 = LIT == 1 ? 0 : round * pitch + warp * LIT;
    S3Msg<LIT> M;
    M.setup(L, li0);
    float acc[NLM][LIT];
#pragma unroll
    for (int a = 0; a < NLM; a++)
#pragma unroll
      for (int q = 0; q < LIT; q++) acc[a][q] = 0.0f;
    for (int q0 = 0; q0 < nb; q0 += S3_BB) {
      const int nq = min(S3_BB, nb - q0);
      __syncthreads();    // what the batch before (the sums of the round before) left is no longer read
      for (int e = tid; e < nq; e += nth) {
        const float4 rec = b.rec[base + q0 + e];
        const float ir = rsqrtf(rec.x * rec.x + rec.y * rec.y + rec.z * rec.z);
        sph_harm<LMAX, false>(sht, rec.x * ir, rec.y * ir, rec.z * ir, [&](int lm, float v, float, float, float) { Ys[e * YLD + lm] = v; });
        meta[e] = s3_bond(b, L, rec, mui);
      }
      __syncthreads();
      M.issue(L, meta, min(S3_NBS, nq), li0, c0, msg, lane);
      s3_issue<NL>(tabc, C, meta, min(S3_NBS, nq), raw, warp, nw, lane);
      for (int q = 0, k = 0; q < nq; q += S3_NBS, k ^= 1) {
        const int ns = min(S3_NBS, nq - q);
        float *R = Rs + k * S3_NBS * NL * 32;
        const float *mg = msg + k * S3Msg<LIT>::GROUP;
        s3_cp_wait();
        s3_radial<NL, false>((float) L.N, meta + q, ns, raw, R, nullptr, warp, nw, lane);
        __syncthreads();    // R of this group is complete; the other half was last read before the barrier of the group before
        if (q + S3_NBS < nq) {
          const int nn = min(S3_NBS, nq - q - S3_NBS);
          M.issue(L, meta + q + S3_NBS, nn, li0, c0, msg + (k ^ 1) * S3Msg<LIT>::GROUP, lane);
          s3_issue<NL>(tabc, C, meta + q + S3_NBS, nn, raw, warp, nw, lane);
        }
#pragma unroll 1
        for (int s = LIT == 1 ? warp : 0; s < ns; s += LIT == 1 ? nw : 1) {
          float ic[LIT];
          M.get(mg, s, L.msg != nullptr, true, lane, ic);    // lanes without a channel write nothing
          const float4 *Y4 = reinterpret_cast<const float4 *>(Ys + (q + s) * YLD);
          float Rl[NL];
#pragma unroll
          for (int l = 0; l < NL; l++) Rl[l] = R[(s * NL + l) * 32 + lane];
#pragma unroll
          for (int y = 0; y < (NLM + 3) / 4; y++) {
            const float4 yv = Y4[y];
            const float ya[4] = {yv.x, yv.y, yv.z, yv.w};
#pragma unroll
            for (int h = 0; h < 4; h++) {
              const int ly = 4 * y + h;
              if (ly >= NLM) continue;
              const float u = ya[h] * Rl[S3<LMAX>::l_of(ly)];
#pragma unroll
              for (int x = 0; x < LIT; x++) acc[ly][x] = fmaf(u, ic[x], acc[ly][x]);
            }
          }
        }
      }
    }
    // the couple: the sums of this round go to shared memory, and each function collects the pairs it is made of (a function
    // is added up by one thread per channel, across the rounds in global memory)
    __syncthreads();
#pragma unroll
    for (int a = 0; a < NLM; a++)
#pragma unroll
      for (int q = 0; q < LIT; q++) Ps[(LIT == 1 ? warp * NLM + a : a * pitch + warp * LIT + q) * 32 + lane] = acc[a][q];
    __syncthreads();
    if (LIT == 1) {    // the warps' shares of the bonds
      for (int a = warp; a < NLM; a += nw) {
        float p = 0.0f;
        for (int w = 0; w < nw; w++) p += Ps[(w * NLM + a) * 32 + lane];
        Ps[a * 32 + lane] = p;
      }
      __syncthreads();
    }
    const int at = round * nw + warp;
    s3_list(L.cg, L.cg_off[at], L.cg_off[at + 1], Ps, lane, [&](int f, float v) {
      float *o = A + ((size_t) f * NA + ap) * C + c;
      if (c < C) *o = round > 0 ? *o + v : v;
    });
  }
}

// Reverse of the above from gA: bond forces and per-atom virial (added: the caller clears them before the first layer is
// reversed), dE/dmsg of the neighbours.  Per bond a thread needs, beside W and dE/dmsg, its share of
//     sum_ly,c W R_l dY_ly/du   and   dE/dx = sum_ly,c W Y_ly dR_l/dx,
// both summed over the functions of its warp as they come, so that only four numbers per bond and warp are added over the
// lanes and none of W leaves the registers.
template<int LMAX, int LIT>
__global__ void __launch_bounds__(32 * S3_WARPS, 2) spbf3_bwd_kernel(BondsDev b, Spbf3Dev L, SHTable sht, const float *__restrict__ gA,
                                                                     int NA, float *__restrict__ fv, double *__restrict__ vir_atom,
                                                                     int a0)
{
  constexpr int NLM = S3<LMAX>::NLM, NL = S3<LMAX>::NL, NP = S3<LMAX>::NP;
  extern __shared__ __align__(16) float sm[];
  float *gAs = sm;                                                   // [nfA][32]
  float *gPs = gAs + 32 * L.nfA;                                     // [warps][half of nlm, LIT][32], before the bond loop; during it:
  float4 *G4 = reinterpret_cast<float4 *>(gPs);                      // [BB][NP][2]: (x0 x1 y0 y1), (z0 z1 Y0 Y1) of a pair
  float4 *raw = G4 + S3_BB * NP * 2;                                 // [NBS][nl][32]
  float *Rs = reinterpret_cast<float *>(raw + S3_NBS * NL * 32);     // [2][NBS][nl][32], then the derivatives
  float *dRs = Rs + 2 * S3_NBS * NL * 32;
  S3Bond *meta = reinterpret_cast<S3Bond *>(dRs + 2 * S3_NBS * NL * 32);    // [BB]
  float *msg = reinterpret_cast<float *>(meta + S3_BB) + (threadIdx.x >> 5) * 2 * S3Msg<LIT>::GROUP;    // [2] groups of the warp
  __shared__ float red[2][S3_NBS * 4];
  __shared__ double vir[S3_NBS][6];
  const int nth = blockDim.x, nw = nth >> 5, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int C = L.C, slices = (C + 31) / 32, ap = blockIdx.x / slices, i = a0 + ap, c0 = blockIdx.x % slices * 32, c = c0 + lane;
  const bool in = c < C;
  const long long base = b.off[i];
  const int nb = b.cnt[i], mui = b.mu[i];
  const int pitch = LIT == 1 ? 1 : nw * LIT, nround = (L.nlmi + pitch - 1) / pitch;
  const float *tabc = L.tab + 4 * min(c, C - 1);
  for (int f = warp; f < L.nfA; f += nw) gAs[f * 32 + lane] = in ? __ldg(gA + ((size_t) f * NA + ap) * C + c) : 0.0f;
  if (tid < S3_NBS)
    for (int k = 0; k < 6; k++) vir[tid][k] = 0.0;
  for (int e = tid; e < 2 * S3_NBS * 4; e += nth) (&red[0][0])[e] = 0.0f;
  // force and virial share of bond `tid` of the group at `at` of the batch q0, from the four sums of its warps
  auto finish = [&](int q0, int at, int ns, float *r4) {
    if (tid >= ns) return;
    const S3Bond B = meta[at + tid];
    const float gx = r4[4 * tid], gy = r4[4 * tid + 1], gz = r4[4 * tid + 2], dedx = r4[4 * tid + 3];
    r4[4 * tid] = r4[4 * tid + 1] = r4[4 * tid + 2] = r4[4 * tid + 3] = 0.0f;
    const long long slot = base + q0 + at + tid;
    const float4 rec = b.rec[slot];
    const float r = B.r, ir = 1.0f / r, ux = rec.x * ir, uy = rec.y * ir, uz = rec.z * ir;
    const float dEdr = dedx / B.rc, gr = gx * ux + gy * uy + gz * uz;
    const float f0 = dEdr * ux + (gx - gr * ux) * ir, f1 = dEdr * uy + (gy - gr * uy) * ir, f2 = dEdr * uz + (gz - gr * uz) * ir;
    float *o = fv + 3 * (size_t) b.cslot[slot];
    atomicAdd(o, f0);
    atomicAdd(o + 1, f1);
    atomicAdd(o + 2, f2);
    const double dx = -(double) ux * r, dy = -(double) uy * r, dz = -(double) uz * r;
    double *v = vir[tid];
    v[0] += dx * f0; v[1] += dy * f1; v[2] += dz * f2;
    v[3] += dx * f1; v[4] += dx * f2; v[5] += dy * f2;
  };
  for (int round = 0; round < nround; round++) {
    const int li0 = LIT == 1 ? 0 : round * pitch + warp * LIT;
    S3Msg<LIT> M;
    M.setup(L, li0);
    // gP of the warp's functions from gA, through its own piece of shared memory
    s3_pair gp[NP][LIT];
    __syncthreads();    // gA is staged; what the round before left is no longer read
    {
      constexpr int HP = (NP + 1) / 2;    // half of the harmonics at a time
      float *mine = gPs + warp * (2 * HP * LIT) * 32 + lane;
#pragma unroll
      for (int half = 0; half < 2; half++) {
        const int at = ((LIT == 1 ? 0 : round * nw + warp)) * 2 + half;
        s3_list(L.cgt, L.cgt_off[at], L.cgt_off[at + 1], gAs, lane, [&](int p, float v) { mine[p * 32] = v; });
#pragma unroll
        for (int a = half * HP; a < (half ? NP : HP); a++)
#pragma unroll
          for (int q = 0; q < LIT; q++)
            gp[a][q] = s3_pack(mine[((2 * a - half * 2 * HP) * LIT + q) * 32], mine[((2 * a + 1 - half * 2 * HP) * LIT + q) * 32]);
      }
    }
    for (int q0 = 0; q0 < nb; q0 += S3_BB) {
      const int nq = min(S3_BB, nb - q0);
      __syncthreads();    // what the batch before left is no longer read
      for (int e = tid; e < nq; e += nth) {
        const float4 rec = b.rec[base + q0 + e];
        const float ir = rsqrtf(rec.x * rec.x + rec.y * rec.y + rec.z * rec.z);
        float *g = reinterpret_cast<float *>(G4 + e * NP * 2);
        sph_harm<LMAX, true>(sht, rec.x * ir, rec.y * ir, rec.z * ir, [&](int lm, float v, float gx, float gy, float gz) {
          float *o = g + 8 * (lm >> 1) + (lm & 1);
          o[0] = gx;
          o[2] = gy;
          o[4] = gz;
          o[6] = v;
        });
        if (NLM & 1)
          for (int k = 1; k < 8; k += 2) g[8 * (NP - 1) + k] = 0.0f;
        meta[e] = s3_bond(b, L, rec, mui);
      }
      __syncthreads();
      M.issue(L, meta, min(S3_NBS, nq), li0, c0, msg, lane);
      s3_issue<NL>(tabc, C, meta, min(S3_NBS, nq), raw, warp, nw, lane);
      int k = 0;
      for (int q = 0; q < nq; q += S3_NBS, k ^= 1) {
        const int ns = min(S3_NBS, nq - q);
        float *R = Rs + k * S3_NBS * NL * 32, *dR = dRs + k * S3_NBS * NL * 32;
        const float *mg = msg + k * S3Msg<LIT>::GROUP;
        s3_cp_wait();
        s3_radial<NL, true>((float) L.N, meta + q, ns, raw, R, dR, warp, nw, lane);
        __syncthreads();    // R of this group is complete, and so are the sums of the group before
        if (q + S3_NBS < nq) {
          const int nn = min(S3_NBS, nq - q - S3_NBS);
          M.issue(L, meta + q + S3_NBS, nn, li0, c0, msg + (k ^ 1) * S3Msg<LIT>::GROUP, lane);
          s3_issue<NL>(tabc, C, meta + q + S3_NBS, nn, raw, warp, nw, lane);
        }
        if (q > 0) finish(q0, q - S3_NBS, S3_NBS, red[k ^ 1]);
#pragma unroll 1
        for (int s = LIT == 1 ? warp : 0; s < ns; s += LIT == 1 ? nw : 1) {
          float ic[LIT];
          M.get(mg, s, L.msg != nullptr, in, lane, ic);
          const ulonglong2 *G = reinterpret_cast<const ulonglong2 *>(G4 + (q + s) * NP * 2);
          float Rl[NL], dRl[NL];
#pragma unroll
          for (int l = 0; l < NL; l++) {
            Rl[l] = R[(s * NL + l) * 32 + lane];
            dRl[l] = dR[(s * NL + l) * 32 + lane];
          }
          s3_pair i2[LIT], v2[LIT], gx = s3_dup(0.0f), gy = gx, gz = gx, gr = gx;
#pragma unroll
          for (int x = 0; x < LIT; x++) {
            i2[x] = s3_dup(ic[x]);
            v2[x] = s3_dup(0.0f);
          }
#pragma unroll
          for (int p = 0; p < NP; p++) {
            const int l0 = S3<LMAX>::l_of(2 * p), l1 = 2 * p + 1 < NLM ? S3<LMAX>::l_of(2 * p + 1) : l0;
            const ulonglong2 g0 = G[2 * p], g1 = G[2 * p + 1];
            const s3_pair Rp = s3_pack(Rl[l0], Rl[l1]), u = s3_mul(g1.y, Rp);
            s3_pair w = s3_mul(gp[p][0], i2[0]);
            s3_fma(v2[0], gp[p][0], u);
#pragma unroll
            for (int x = 1; x < LIT; x++) {
              s3_fma(w, gp[p][x], i2[x]);
              s3_fma(v2[x], gp[p][x], u);
            }
            const s3_pair wr = s3_mul(w, Rp), wd = s3_mul(w, s3_pack(dRl[l0], dRl[l1]));
            s3_fma(gx, wr, g0.x);
            s3_fma(gy, wr, g0.y);
            s3_fma(gz, wr, g1.x);
            s3_fma(gr, wd, g1.y);
          }
          if (L.gmsg && in) {
            float *o = L.gmsg + meta[q + s].row + c;
#pragma unroll
            for (int x = 0; x < LIT; x++)
              if (li0 + x < L.nlmi) atomicAdd(o + (li0 + x) * C, s3_sum(v2[x]));
          }
          // the four sums over the lanes by one tree: two exchanges leave each lane one of them, three more add it up
          {
            const bool h = lane & 16, g = lane & 8;
            const float sx = s3_sum(gx), sy = s3_sum(gy), sz = s3_sum(gz), sr = s3_sum(gr);
            const float p0 = (h ? sz : sx) + __shfl_xor_sync(0xffffffffu, h ? sx : sz, 16);
            const float p1 = (h ? sr : sy) + __shfl_xor_sync(0xffffffffu, h ? sy : sr, 16);
            float t = (g ? p1 : p0) + __shfl_xor_sync(0xffffffffu, g ? p0 : p1, 8);
            t += __shfl_xor_sync(0xffffffffu, t, 4);
            t += __shfl_xor_sync(0xffffffffu, t, 2);
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            if ((lane & 7) == 0) atomicAdd(&red[k][4 * s + (h ? 2 : 0) + (g ? 1 : 0)], t);
          }
        }
      }
      __syncthreads();
      const int last = (nq - 1) / S3_NBS * S3_NBS;
      finish(q0, last, nq - last, red[k ^ 1]);
    }
  }
  if (tid < S3_NBS)
    for (int k = 0; k < 6; k++)
      if (vir[tid][k] != 0.0) atomicAdd(vir_atom + 6 * (size_t) i + k, vir[tid][k]);
}

struct EqNormDev {
  const float *dw, *mask, *aff;
  const int *e;
  int nf, C, center;
  double eps;
};

// The norms and the readout: a CTA (norms of the messages) or a warp (densities, readout) per atom, lanes along the channels.
// A thread per atom, which read 1600 values of its row one after the other, left all but a few SMs idle at hundreds of atoms
// (250 atoms: 2.0 ms for the two reverse norms, 0.8 ms forward).
constexpr int EQ_WARPS = 8;

__device__ __forceinline__ double warp_sum(double v)
{
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}
__device__ __forceinline__ double block_sum(double v, double *sh)    // v: the same on all lanes of a warp
{
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < EQ_WARPS; w++) s += sh[w];
  return s;
}

// EquivariantRMSNorm (libgrace/include/grace/fused_3l_cpu.h:346-370): x [f][NA][C] -> y rows [i][f][C]
__global__ void __launch_bounds__(32 * EQ_WARPS) eqnorm_fwd_kernel(EqNormDev E, const float *__restrict__ x, float *__restrict__ y, int NA,
                                                                   int a0)
{
  __shared__ double sh[EQ_WARPS];
  const int i = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto mean = [&](int f) {
    if (!E.center || E.mask[f] == 0.0f) return 0.0;
    double m = 0.0;
    for (int c = lane; c < E.C; c += 32) m += x[((size_t) f * NA + i) * E.C + c];
    return warp_sum(m) / E.C * E.mask[f];
  };
  double S = 0.0;
  for (int f = warp; f < E.nf; f += EQ_WARPS) {
    const double m = mean(f);
    double s2 = 0.0;
    for (int c = lane; c < E.C; c += 32) {
      const float v = (float) (x[((size_t) f * NA + i) * E.C + c] - m);
      s2 += (double) v * v;
    }
    S += E.dw[f] * s2;
  }
  const double r = 1.0 / sqrt(block_sum(warp_sum(S), sh) / E.C + E.eps);
  for (int f = warp; f < E.nf; f += EQ_WARPS) {
    const double m = mean(f);
    for (int c = lane; c < E.C; c += 32)
      y[((size_t) (a0 + i) * E.nf + f) * E.C + c] =
          (float) ((float) (x[((size_t) f * NA + i) * E.C + c] - m) * r) * E.aff[(size_t) E.e[f] * E.C + c];
  }
}

// gx [f][NA][C] = adjoint of the above for dy rows [i][f][C] (:373-415)
__global__ void __launch_bounds__(32 * EQ_WARPS) eqnorm_bwd_kernel(EqNormDev E, const float *__restrict__ x, const float *__restrict__ dy,
                                                                   float *__restrict__ gx, int NA, int a0)
{
  __shared__ double sh[EQ_WARPS];
  const int i = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto mean = [&](int f) {
    if (!E.center || E.mask[f] == 0.0f) return 0.0;
    double m = 0.0;
    for (int c = lane; c < E.C; c += 32) m += x[((size_t) f * NA + i) * E.C + c];
    return warp_sum(m) / E.C * E.mask[f];
  };
  double S = 0.0, dot = 0.0;
  for (int f = warp; f < E.nf; f += EQ_WARPS) {
    const float *xf = x + ((size_t) f * NA + i) * E.C, *a = E.aff + (size_t) E.e[f] * E.C, *d = dy + ((size_t) (a0 + i) * E.nf + f) * E.C;
    const double m = mean(f);
    double s2 = 0.0;
    for (int c = lane; c < E.C; c += 32) {
      const float v = (float) (xf[c] - m);
      s2 += (double) v * v;
      dot += (double) d[c] * a[c] * v;
    }
    S += E.dw[f] * s2;
  }
  S = block_sum(warp_sum(S), sh);
  dot = block_sum(warp_sum(dot), sh);
  const double r = 1.0 / sqrt(S / E.C + E.eps), k3 = r * r * r * dot / E.C;
  for (int f = warp; f < E.nf; f += EQ_WARPS) {
    const float *xf = x + ((size_t) f * NA + i) * E.C, *a = E.aff + (size_t) E.e[f] * E.C, *d = dy + ((size_t) (a0 + i) * E.nf + f) * E.C;
    float *o = gx + ((size_t) f * NA + i) * E.C;
    const double m = mean(f), kf = k3 * E.dw[f];
    double gm = 0.0;
    if (E.center && E.mask[f] != 0.0f) {
      for (int c = lane; c < E.C; c += 32) gm += (float) (r * d[c] * a[c] - kf * (float) (xf[c] - m));
      gm = warp_sum(gm) / E.C * E.mask[f];
    }
    for (int c = lane; c < E.C; c += 32) o[c] = (float) ((float) (r * d[c] * a[c] - kf * (float) (xf[c] - m)) - gm);
  }
}

// RMSNorm of the density (:416-425): x [NA][wr] (one function) -> y rows [i][wr]; sum rows += y
__global__ void __launch_bounds__(128) rmsnorm_fwd_kernel(const float *__restrict__ x, const float *__restrict__ scale, int n0, int wr,
                                                          float *__restrict__ sum, int first, int n, int a0)
{
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= n) return;
  const float *xi = x + (size_t) i * wr;
  float *s = sum + (size_t) (a0 + i) * wr;
  double q = 0.0;
  for (int c = n0 + lane; c < wr; c += 32) q += (double) xi[c] * xi[c];
  const double r = 1.0 / sqrt(warp_sum(q) / (wr - n0) + 1e-10);
  for (int c = lane; c < wr; c += 32) {
    const float y = c < n0 ? xi[c] : (float) (xi[c] * r) * scale[c - n0];
    s[c] = first ? y : s[c] + y;
  }
}

__global__ void __launch_bounds__(128) rmsnorm_bwd_kernel(const float *__restrict__ x, const float *__restrict__ scale, int n0, int wr,
                                                          const float *__restrict__ dy, float *__restrict__ gx, int n, int a0)
{
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= n) return;
  const float *xi = x + (size_t) i * wr, *d = dy + (size_t) (a0 + i) * wr;
  float *o = gx + (size_t) i * wr;
  double q = 0.0, g = 0.0;
  for (int c = n0 + lane; c < wr; c += 32) {
    q += (double) xi[c] * xi[c];
    g += (double) d[c] * scale[c - n0] * xi[c];
  }
  const double r = 1.0 / sqrt(warp_sum(q) / (wr - n0) + 1e-10), k = r * r * r * warp_sum(g) / (wr - n0);
  for (int c = lane; c < wr; c += 32) o[c] = c < n0 ? d[c] : (float) (r * d[c] * scale[c - n0] - k * xi[c]);
}

constexpr int RO_IN = 128, RO_HIDDEN = 256;    // most inputs and hidden units (build_plan refuses more)
struct Readout3Dev {
  const double *W0, *W1, *shift;    // [nin][nh], [nh], [n_elements]
  double n0, n1, oscale;
  int nin, nh, act;
};

// E_i = (MLP(sum[1:]) + sum[0]) scale + shift (fp64, :1334-1374); d: dE/d(sum) rows [i][1 + nin]
__global__ void __launch_bounds__(128) readout3_kernel(Readout3Dev R, const float *__restrict__ sum, const int *__restrict__ mu,
                                                       double *__restrict__ e_atom, float *__restrict__ d, int want_grad, int n)
{
  __shared__ double s_ds[4][RO_HIDDEN];
  __shared__ float s_h[4][RO_IN];
  const int w = threadIdx.x >> 5, i = blockIdx.x * 4 + w, lane = threadIdx.x & 31;
  if (i >= n) return;
  const int wr = R.nin + 1;
  const float *h = sum + (size_t) i * wr;
  float *di = d + (size_t) i * wr;
  for (int c = lane; c < R.nin; c += 32) s_h[w][c] = h[c + 1];
  __syncwarp();
  double e = 0.0;
  for (int j = lane; j < R.nh; j += 32) {    // a lane per hidden unit
    double s = 0.0;
    for (int c = 0; c < R.nin; c++) s += (double) s_h[w][c] * R.W0[(size_t) c * R.nh + j];
    s *= R.n0;
    double act, dact;
    if (R.act == 1) {
      act = tanh(s);
      dact = 1.0 - act * act;
    } else {
      const double sg = 1.0 / (1.0 + exp(-s));
      act = s * sg;
      dact = sg * (1.0 + s * (1.0 - sg));
    }
    e += R.W1[j] * act;
    s_ds[w][j] = R.oscale * R.n1 * R.W1[j] * dact * R.n0;
  }
  e = warp_sum(e) * R.n1;
  __syncwarp();
  if (lane == 0) e_atom[i] = (e + (double) h[0]) * R.oscale + R.shift[mu[i]];
  if (!want_grad) return;
  if (lane == 0) di[0] = (float) R.oscale;
  for (int c = lane; c < R.nin; c += 32) {    // a lane per input
    double g = 0.0;
    for (int j = 0; j < R.nh; j++) g += R.W0[(size_t) c * R.nh + j] * s_ds[w][j];
    di[c + 1] = (float) g;
  }
}

}    // namespace

// device state of the three layers
struct State3L {
  LayerEngine E[3];
  DBuf<float> arena[3], tab[3], zproj[3], l0mask[3], rho_scale[3];
  DBuf<int> cg_off[3], cgt_off[3];
  DBuf<int2> cg[3], cgt[3];
  DBuf<float> eq_dw[2], eq_mask[2], eq_aff[2], msg[2], gmsg[2];
  DBuf<int> eq_e[2];
  DBuf<int> pair_slot;
  std::vector<int> pair_slot_host;
  std::vector<std::vector<float>> tab_host[3];    // per layer, per pair slot
  int npairs = 0;
  DBuf<float> rho_sum, drho;
  DBuf<double> eW0, eW1;
  const float *bound[3] = {nullptr, nullptr, nullptr};    // arena and atom stride the tensor tables point into
  int bound_NC[3] = {0, 0, 0};
};

void Engine::setup_3l()
{
  const Plan3L &Q = *plan_.p3;
  s3_ = std::make_shared<State3L>();
  State3L &S = *s3_;
  for (int k = 0; k < 3; k++) {
    const Layer3Plan &L = Q.L[k];
    // (the reference's CPU engine asks for multiples of 16 as well: libgrace/src/fused_3l.cpp:433)
    if (L.C > 64 || L.C % 16) throw Unsupported("GRACE-3L: channel counts must be multiples of 16 up to 64");
    setup_layer(S.E[k], L.dense);
    S.zproj[k].upload(L.zproj);
    S.l0mask[k].upload(L.l0mask);
    S.rho_scale[k].upload(L.rho_scale);
    for (size_t q = 0; q < L.lt.size(); q++)    // the kernels take the radial function of a harmonic from its place
      if (L.lt[q] != (int) std::sqrt((double) q)) throw Unsupported("GRACE-3L: harmonics are expected in the order lm = l (l + 1) + m");
    std::vector<int2> cg, cgt;
    auto bits = [](float v) {
      int u;
      std::memcpy(&u, &v, 4);
      return u;
    };
    const int nw = s3_warps(L.nlmi), pitch = s3_pitch(L.nlmi), nround = (L.nlmi + pitch - 1) / pitch, nlm = plan_.nlm;
    const int lit = L.nlmi == 1 ? 1 : S3_LIT, hp = (nlm / 2 + nlm % 2 + 1) / 2 * 2;    // hp: harmonics of a half
    if (nlm * pitch >= (1 << 16) || L.nfA >= (1 << 15)) throw Unsupported("GRACE-3L: the couple of a layer has too many functions");
    // a target's last entry carries it; a target without entries gets one with coefficient 0
    auto close = [&](std::vector<int2> &v, size_t from, int target) {
      if (v.size() == from) v.push_back(make_int2(0, 0));
      v.back().x |= (target + 1) << 16;
    };
    std::vector<int> cg_off, cgt_off;
    for (int r = 0; r < nround; r++)
      for (int w = 0; w < nw; w++) {
        cg_off.push_back((int) cg.size());
        for (int f = w; f < L.nfA; f += nw) {    // the output functions of the warp: sums of pairs
          const size_t from = cg.size();
          for (int t = L.cg_off[f]; t < L.cg_off[f + 1]; t++) {
            const int ly = L.cg_p[t] / L.nlmi, li = L.cg_p[t] % L.nlmi;
            if (li / pitch == r) cg.push_back(make_int2(ly * pitch + li % pitch, bits(L.cg_v[t])));
          }
          if (r == 0 || cg.size() > from) close(cg, from, f);
        }
        if (lit == 1 && w > 0) continue;
        for (int half = 0; half < 2; half++) {    // the pairs of the warp: sums of the functions they feed
          cgt_off.push_back((int) cgt.size());
          for (int p = 0; p < hp * lit; p++) {
            const int ly = half * hp + p / lit, li = (lit == 1 ? 0 : r * pitch + w * lit) + p % lit;
            const size_t from = cgt.size();
            if (ly < nlm && li < L.nlmi)
              for (int t = L.cgt_off[ly * L.nlmi + li]; t < L.cgt_off[ly * L.nlmi + li + 1]; t++)
                cgt.push_back(make_int2(L.cgt_f[t], bits(L.cgt_v[t])));
            close(cgt, from, p);
          }
        }
      }
    cg_off.push_back((int) cg.size());
    cgt_off.push_back((int) cgt.size());
    S.cg_off[k].upload(cg_off);
    S.cgt_off[k].upload(cgt_off);
    S.cg[k].upload(cg);
    S.cgt[k].upload(cgt);
    if (k < 2) {
      S.eq_dw[k].upload(L.eq_dw);
      S.eq_mask[k].upload(L.eq_mask);
      S.eq_aff[k].upload(L.eq_aff);
      S.eq_e[k].upload(L.eq_e);
    }
  }
  S.pair_slot_host.assign((size_t) plan_.n_elements * plan_.n_elements, -1);
  S.pair_slot.upload(S.pair_slot_host);
  if (Q.e_nin > RO_IN || Q.e_nh > RO_HIDDEN) throw Unsupported("GRACE-3L: the energy MLP is too wide");
  S.eW0.upload(Q.eW0);
  S.eW1.upload(Q.eW1);
  shift_.upload(plan_.shift);
  GB_CUDA(cudaStreamSynchronize(dev().stream));
}

// radial tables of every pair of the given elements (built once per pair)
void Engine::prepare_species(const std::vector<int> &elements)
{
  if (plan_.layers != 3) return;
  std::lock_guard<std::mutex> lk(mu);
  State3L &S = *s3_;
  const Plan3L &Q = *plan_.p3;
  const int nel = plan_.n_elements;
  bool grown = false;
  for (int a : elements)
    for (int b : elements) {
      int &slot = S.pair_slot_host[(size_t) a * nel + b];
      if (slot >= 0) continue;
      slot = S.npairs++;
      for (int k = 0; k < 3; k++) S.tab_host[k].push_back(radial_table_3l(*Q.model, k, a, b, Q.spline_n));
      grown = true;
    }
  if (!grown) return;
  for (int k = 0; k < 3; k++) {
    std::vector<float> all;
    for (const auto &t : S.tab_host[k]) all.insert(all.end(), t.begin(), t.end());
    S.tab[k].upload(all);
  }
  S.pair_slot.upload(S.pair_slot_host);
  GB_CUDA(cudaStreamSynchronize(dev().stream));
}

void Engine::evaluate_3l(NeighborList &nl, bool energy_only, StageTimer *tm)
{
  State3L &S = *s3_;
  const Plan3L &Q = *plan_.p3;
  const int n = (int) nl.n();
  const int NA = (n + 3) / 4 * 4;
  const BondsDev bonds = nl.bonds();
  const int *mu = bonds.mu;
  const SHTable sht = sh_table_host();
  tc_now_ = dense_ == Dense::Tc || dense_ == Dense::Auto;    // the projections, reduces and FCs as tensor-core grouped GEMMs (mv_tc.cu)
  // every bond needs the radial table of its element pair: the species of every System / Batch of this engine were
  // prepared when it was created (prepare_species); a bond of a pair without a table is left out by the kernels
  if (tm) tm->begin(StageTimer::FWD);
  const int wr = Q.L[0].wr;
  S.rho_sum.ensure((size_t) n * wr);
  S.drho.ensure((size_t) n * wr);
  auto spbf = [&](int k) {
    const Layer3Plan &L = Q.L[k];
    Spbf3Dev d{};
    d.tab = S.tab[k].get();
    d.pair_slot = S.pair_slot.get();
    d.tab_stride = (long long) Q.spline_n * (plan_.lmax + 1) * L.C * 4;
    d.rc = rcf_.get();
    d.msg = k > 0 ? S.msg[k - 1].get() : nullptr;
    d.gmsg = k > 0 ? S.gmsg[k - 1].get() : nullptr;
    d.zproj = S.zproj[k].get();
    d.l0mask = S.l0mask[k].get();
    d.cg_off = S.cg_off[k].get();
    d.cgt_off = S.cgt_off[k].get();
    d.cg = S.cg[k].get();
    d.cgt = S.cgt[k].get();
    d.N = Q.spline_n;
    d.C = L.C;
    d.nl = plan_.lmax + 1;
    d.nlm = plan_.nlm;
    d.nlmi = L.nlmi;
    d.nfA = L.nfA;
    d.nel = plan_.n_elements;
    return d;
  };
  // launches of the bond kernels: a warp per S3_LIT message functions (a layer without messages: 4 warps that share the bonds)
  auto bonds_forward = [&](int k, float *A, int NC, int a0, int na) {
    const Layer3Plan &L = Q.L[k];
    const bool one = L.nlmi == 1;
    const int nw = s3_warps(L.nlmi), nlm = plan_.nlm, nl = plan_.lmax + 1, np = (nlm + 1) / 2;
    const size_t group = (size_t) nw * 2 * S3_NBS * ((one ? 1 : S3_LIT) + 1) * 32;    // floats of the message buffers
    const size_t stage = sizeof(float) * (6 * (size_t) S3_NBS * nl * 32 + (size_t) S3_BB * ((np + 1) / 2 * 4) + group) + sizeof(S3Bond) * S3_BB;
    const size_t sums = sizeof(float) * 32 * (size_t) nlm * nw * (one ? 1 : S3_LIT), smem = std::max(stage, sums);
    const unsigned grid = (unsigned) ((L.C + 31) / 32) * (unsigned) na;    // the slices of an atom side by side
    auto go = [&](auto kernel) {
      GB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 110 * 1024));
      before_launch("spbf3_fwd_kernel");
      kernel<<<grid, 32 * nw, smem, dev().stream>>>(bonds, spbf(k), sht, A, NC, a0);
      after_launch("spbf3_fwd_kernel");
    };
    switch (plan_.lmax) {
      case 1: one ? go(spbf3_fwd_kernel<1, 1>) : go(spbf3_fwd_kernel<1, S3_LIT>); break;
      case 2: one ? go(spbf3_fwd_kernel<2, 1>) : go(spbf3_fwd_kernel<2, S3_LIT>); break;
      case 3: one ? go(spbf3_fwd_kernel<3, 1>) : go(spbf3_fwd_kernel<3, S3_LIT>); break;
      default: one ? go(spbf3_fwd_kernel<4, 1>) : go(spbf3_fwd_kernel<4, S3_LIT>); break;
    }
  };
  auto bonds_reverse = [&](int k, const float *gA, int NC, int a0, int na) {
    const Layer3Plan &L = Q.L[k];
    const bool one = L.nlmi == 1;
    const int nw = s3_warps(L.nlmi), nlm = plan_.nlm, nl = plan_.lmax + 1, np = (nlm + 1) / 2;
    const size_t group = (size_t) nw * 2 * S3_NBS * ((one ? 1 : S3_LIT) + 1) * 32;
    const size_t stage = sizeof(float) * (8 * (size_t) S3_BB * np + 8 * (size_t) S3_NBS * nl * 32 + group) + sizeof(S3Bond) * S3_BB;
    const size_t grads = sizeof(float) * 32 * (size_t) ((np + 1) / 2 * 2) * nw * (one ? 1 : S3_LIT);
    const size_t smem = sizeof(float) * 32 * (size_t) L.nfA + std::max(stage, grads);
    if (smem > 200 * 1024) throw Unsupported("GRACE-3L: the bond sums of a layer do not fit the shared memory");
    const unsigned grid = (unsigned) ((L.C + 31) / 32) * (unsigned) na;    // the slices of an atom side by side
    auto go = [&](auto kernel) {
      GB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
      before_launch("spbf3_bwd_kernel");
      kernel<<<grid, 32 * nw, smem, dev().stream>>>(bonds, spbf(k), sht, gA, NC, fv_.get(), vir_atom_.get(), a0);
      after_launch("spbf3_bwd_kernel");
    };
    switch (plan_.lmax) {
      case 1: one ? go(spbf3_bwd_kernel<1, 1>) : go(spbf3_bwd_kernel<1, S3_LIT>); break;
      case 2: one ? go(spbf3_bwd_kernel<2, 1>) : go(spbf3_bwd_kernel<2, S3_LIT>); break;
      case 3: one ? go(spbf3_bwd_kernel<3, 1>) : go(spbf3_bwd_kernel<3, S3_LIT>); break;
      default: one ? go(spbf3_bwd_kernel<4, 1>) : go(spbf3_bwd_kernel<4, S3_LIT>); break;
    }
  };
  // Passes.  When the tensors of all three layers of all atoms fit the memory they are kept from the forward to the
  // reverse pass (arena k holds layer k).  Otherwise every layer runs in passes over atom chunks through one arena, and
  // the reverse pass of a layer evaluates the forward operations of a chunk again before it reverses them: the messages,
  // their gradients and the densities live in per-atom rows outside the arenas either way.
  long long per_all = 0, per_max = 0;
  for (int k = 0; k < 3; k++) {
    per_all += S.E[k].per_atom;
    per_max = std::max(per_max, S.E[k].per_atom);
  }
  bool held = true;    // the arenas hold all layers already: no look at the free memory
  for (int k = 0; k < 3; k++) held = held && (double) S.E[k].per_atom * NA <= (double) S.arena[k].capacity();
  double budget = 0.0;
  for (int k = 0; k < 3; k++) budget += 4.0 * (double) S.arena[k].capacity();
  if (!held) budget += 0.7 * (double) device_free_bytes();
  if (const char *env = getenv("GRACE_B200_3L_CHUNK")) budget = std::min(budget, 4.0 * per_all * std::max(4, atoi(env)) - 1.0);
  const bool keep = 4.0 * (double) per_all * NA <= budget;
  int NC = NA;    // atoms per pass (a multiple of 4: the atom stride of the arena)
  if (!keep) {
    NC = (int) std::min<double>(NA, std::max(512.0, budget / (4.0 * per_max)));
    if (const char *env = getenv("GRACE_B200_3L_CHUNK")) NC = std::min(NC, std::max(4, atoi(env)));
    NC = std::max(4, NC / 4 * 4);
    for (int k = 1; k < 3; k++) S.arena[k].release();
  }
  // the arena of layer k bound for passes of NC atoms
  auto bind = [&](int k) {
    LayerEngine &E = S.E[k];
    DBuf<float> &ar = S.arena[keep ? k : 0];
    float *base = ar.ensure((size_t) (keep ? E.per_atom : per_max) * NC);
    if (S.bound[k] != base || S.bound_NC[k] != NC) {    // the tensor table on the device moves with the arena only
      bind_arena(E, base, NC);
      S.bound[k] = base;
      S.bound_NC[k] = NC;
    }
    return base;
  };
  // forward operations of layer k for the atoms [a0, a0 + na); outputs: the message rows and the density sums
  auto forward = [&](int k, int a0, int na, bool outputs) {
    const Layer3Plan &L = Q.L[k];
    LayerEngine &E = S.E[k];
    const std::vector<TensorDev> &T = E.tensors_host;
    bonds_forward(k, T[L.tA].p, NC, a0, na);
    run(E, true, nl, NeighborList::All, mu + a0, a0, na, NC);
    if (!outputs) return;
    if (k < 2) {
      const EqNormDev e{S.eq_dw[k].get(), S.eq_mask[k].get(), S.eq_aff[k].get(), S.eq_e[k].get(), L.nfEQ, L.cEQ, L.eq_center, L.eq_eps};
      GB_LAUNCH(eqnorm_fwd_kernel, na, 32 * EQ_WARPS, 0, e, T[L.tEQ].p, S.msg[k].get(), NC, a0);
    }
    GB_LAUNCH(rmsnorm_fwd_kernel, (na + 3) / 4, 128, 0, T[L.tRHO].p, S.rho_scale[k].get(), L.rho_n0, wr, S.rho_sum.get(), k == 0 ? 1 : 0, na, a0);
  };
  // reverse operations of layer k for the atoms [a0, a0 + na), whose forward tensors are in the bound arena
  auto reverse = [&](int k, int a0, int na, float *base) {
    const Layer3Plan &L = Q.L[k];
    LayerEngine &E = S.E[k];
    const std::vector<TensorDev> &T = E.tensors_host;
    if (L.dense.zero_grads)
      launch_fill_zero(base + (size_t) E.grad_begin * NC, sizeof(float) * (size_t) (E.grad_end - E.grad_begin) * NC);
    GB_LAUNCH(rmsnorm_bwd_kernel, (na + 3) / 4, 128, 0, T[L.tRHO].p, S.rho_scale[k].get(), L.rho_n0, wr, S.drho.get(), T[L.tGRHO].p, na, a0);
    if (k < 2) {
      const EqNormDev e{S.eq_dw[k].get(), S.eq_mask[k].get(), S.eq_aff[k].get(), S.eq_e[k].get(), L.nfEQ, L.cEQ, L.eq_center, L.eq_eps};
      GB_LAUNCH(eqnorm_bwd_kernel, na, 32 * EQ_WARPS, 0, e, T[L.tEQ].p, S.gmsg[k].get(), T[L.tGEQ].p, NC, a0);
    }
    run(E, false, nl, NeighborList::All, mu + a0, a0, na, NC);
    bonds_reverse(k, T[L.tGA].p, NC, a0, na);
  };
  for (int k = 0; k < 2; k++) S.msg[k].ensure((size_t) n * Q.L[k].nfEQ * Q.L[k].cEQ);
  for (int k = 0; k < 3; k++) {
    bind(k);
    for (int a0 = 0; a0 < n; a0 += NC) forward(k, a0, std::min(NC, n - a0), true);
  }
  const Readout3Dev ro{S.eW0.get(), S.eW1.get(), shift_.get(), Q.en0, Q.en1, plan_.out_scale, Q.e_nin, Q.e_nh, Q.e_act};
  GB_LAUNCH(readout3_kernel, (n + 3) / 4, 128, 0, ro, S.rho_sum.get(), mu, e_atom_.get(), S.drho.get(), energy_only ? 0 : 1, n);
  if (tm) tm->end(StageTimer::FWD);
  if (energy_only) return;
  if (tm) tm->begin(StageTimer::BWD);
  // the reverse bond kernels add their shares (three layers, channel slices) to the bond forces and the virial
  launch_fill_zero(fv_.get(), sizeof(float) * 3 * (size_t) std::max<int64_t>(nl.nslots(), 1));
  launch_fill_zero(vir_atom_.get(), sizeof(double) * 6 * (size_t) n);
  for (int k = 0; k < 2; k++) {
    const Layer3Plan &L = Q.L[k];
    S.gmsg[k].ensure((size_t) n * L.nfEQ * L.cEQ);
    launch_fill_zero(S.gmsg[k].get(), sizeof(float) * (size_t) n * L.nfEQ * L.cEQ);
  }
  for (int k = 2; k >= 0; k--) {
    float *base = bind(k);
    for (int a0 = 0; a0 < n; a0 += NC) {
      const int na = std::min(NC, n - a0);
      if (!keep) forward(k, a0, na, false);    // the chunk's forward tensors again
      reverse(k, a0, na, base);
    }
  }
  if (tm) tm->end(StageTimer::BWD);
}

}    // namespace gb
