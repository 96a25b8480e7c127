// Kernels of the dense per-atom network (FC, Clebsch-Gordan products, reduces and their adjoints as two table-driven
// kernels), the fp64 readouts, and the per-atom gathers and sums that leave the network.
// Mathematics: libgrace/include/grace/fused_cpu.h:349-364 (FC), 411-453 (products), 637-649 (reduces);
// libgrace/src/fused_1l.cpp:378-427 and libgrace/src/fused_2l.cpp:548-615 (readouts).
#include "kernels.h"
#include "readout.cuh"

#include <algorithm>
#include <cstdint>
#include <cstdlib>

namespace gb {

// ---- MV: out[row][a][k] (+)= sum_items scale * sum_n M[n][k] x[item][a][n] ----------------------------------
// block (KP, 128 / KP): threadIdx.x = output channel k, threadIdx.y = atom group; AT atoms per thread share each
// weight load.  grid (rows, atom blocks).
template<int AT, bool ELEM>
__global__ void __launch_bounds__(128) mv_kernel(MVDev op, const TensorDev *__restrict__ T, const int *__restrict__ mu,
                                                 int NA, int na)
{
  const int row = blockIdx.x;
  const int k = threadIdx.x;
  const int a_first = (blockIdx.y * blockDim.y + threadIdx.y) * AT;
  if (k >= op.n_out || a_first >= na) return;
  float acc[AT];
  long long tyo[AT];
#pragma unroll
  for (int i = 0; i < AT; i++) {
    acc[i] = 0.0f;
    const int a = min(a_first + i, na - 1);
    tyo[i] = ELEM ? (long long) mu[a] * op.ty_stride : 0;
  }
  const int i0 = op.item_off[row], i1 = op.item_off[row + 1];
  for (int it = i0; it < i1; it++) {
    const MVItem item = op.items[it];
    const TensorDev src = T[item.src];
    const float *x[AT];
#pragma unroll
    for (int i = 0; i < AT; i++) x[i] = src.p + ((size_t) item.irow * NA + min(a_first + i, na - 1)) * src.C;
    float part[AT];
#pragma unroll
    for (int i = 0; i < AT; i++) part[i] = 0.0f;
    if (ELEM) {
      for (int n = 0; n < item.n_in; n++) {
#pragma unroll
        for (int i = 0; i < AT; i++)
          part[i] = fmaf(__ldg(x[i] + n), __ldg(op.W + tyo[i] + item.mat + (size_t) n * op.ldw + k), part[i]);
      }
    } else {
      const float *M = op.W + item.mat + k;
#pragma unroll 4
      for (int n = 0; n < item.n_in; n++) {
        const float w = __ldg(M + (size_t) n * op.ldw);
#pragma unroll
        for (int i = 0; i < AT; i++) part[i] = fmaf(__ldg(x[i] + n), w, part[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < AT; i++) acc[i] = fmaf(item.scale, part[i], acc[i]);
  }
  const TensorDev dst = T[op.dst];
  const int orow = op.row_out[row];
#pragma unroll
  for (int i = 0; i < AT; i++) {
    const int a = a_first + i;
    if (a < na) {
      float *o = dst.p + ((size_t) orow * NA + a) * dst.C + k;
      *o = op.accumulate ? *o + acc[i] : acc[i];
    }
  }
}

void launch_mv(const MVDev &op, const TensorDev *tensors, const int *mu, int NA, int na)
{
  if (op.nrows == 0 || na == 0) return;
  int KP = 8;
  while (KP < op.n_out) KP *= 2;
  if (KP > 128) throw Unsupported("dense network: more than 128 channels are not supported");
  constexpr int AT = 4;
  const dim3 block(KP, 128 / KP);
  const dim3 grid(op.nrows, (na + block.y * AT - 1) / (block.y * AT));
  if (op.elem) GB_LAUNCH((mv_kernel<AT, true>), grid, block, 0, op, tensors, mu, NA, na);
  else GB_LAUNCH((mv_kernel<AT, false>), grid, block, 0, op, tensors, mu, NA, na);
}

// ---- PROD: out[row][i] (+)= sum_terms coef A[a][i] B[b][i], i over the NA * C values of a function row ---------
__global__ void __launch_bounds__(256) prod_kernel(ProdDev op, const TensorDev *__restrict__ T, long long row_len,
                                                   long long act_len)
{
  const int row = blockIdx.x;
  const long long i = (long long) blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= act_len) return;
  const float *A = T[op.srcA].p + i;
  const float *B = op.srcB >= 0 ? T[op.srcB].p + i : nullptr;
  const int t0 = op.term_off[row], t1 = op.term_off[row + 1];
  float acc = 0.0f;
  if (B) {
    for (int t = t0; t < t1; t++) {
      const ProdTerm tm = op.terms[t];
      acc = fmaf(tm.coef * __ldg(A + tm.a * row_len), __ldg(B + tm.b * row_len), acc);
    }
  } else {
    for (int t = t0; t < t1; t++) {
      const ProdTerm tm = op.terms[t];
      acc = fmaf(tm.coef, __ldg(A + tm.a * row_len), acc);
    }
  }
  float *o = T[op.dst].p + (long long) op.row_out[row] * row_len + i;
  *o = (op.accumulate && !(op.row_first && op.row_first[row])) ? *o + acc : acc;
}

// The same for a tile of TA atoms with the input rows staged in shared memory: every input value comes from global
// memory once (coalesced, TA x C contiguous floats per function) however many terms read it, and the term loop runs on
// shared memory.  srcB == srcA or srcB < 0: one staged tensor.
__global__ void __launch_bounds__(256) prod_tile_kernel(ProdDev op, const TensorDev *__restrict__ T, int NA, int na, int TA,
                                                        int nfA, int nfB, int C)
{
  extern __shared__ __align__(16) float psm[];
  const int C4 = C >> 2, TAC4 = TA * C4, t = threadIdx.x;
  const int a0 = blockIdx.x * TA, nta = min(TA, na - a0);
  const int per = (op.nrows + gridDim.y - 1) / gridDim.y, row_lo = per * blockIdx.y, row_hi = min(op.nrows, row_lo + per);
  if (row_lo >= row_hi) return;
  const int term0 = op.term_off[row_lo], nterms = op.term_off[row_hi] - term0;
  float4 *sA = reinterpret_cast<float4 *>(psm);
  float4 *sB = sA + (size_t) nfA * TAC4;
  int4 *sT = reinterpret_cast<int4 *>(sB + (size_t) nfB * TAC4);    // per term: row offsets of both operands, coefficient
  const bool two = op.srcB >= 0 && op.srcB != op.srcA;
  {
    // eight independent 16-byte loads per thread in flight: the tile's rows come from nf separate regions of the
    // tensor, and a CTA has nothing else to do until they are there
    auto stage = [&](const float *G, float4 *S, int nf) {
      const int total = nf * TAC4;
      for (int base = 0; base < total; base += 256 * 8) {
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int idx = base + j * 256 + t, f = idx / TAC4, r = idx - f * TAC4;
          v[j] = (idx < total && r / C4 < nta) ? __ldg(reinterpret_cast<const float4 *>(G + ((size_t) f * NA + a0) * C) + r)
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int idx = base + j * 256 + t;
          if (idx < total) S[idx] = v[j];
        }
      }
    };
    stage(T[op.srcA].p, sA, nfA);
    if (two) stage(T[op.srcB].p, sB, nfB);
    for (int idx = t; idx < nterms; idx += 256) {
      const ProdTerm tm = op.terms[term0 + idx];
      sT[idx] = make_int4(tm.a * TAC4, tm.b * TAC4, __float_as_int(tm.coef), 0);
    }
  }
  __syncthreads();
  const float4 *Bs = op.srcB < 0 ? nullptr : (two ? sB : sA);
  float *D = T[op.dst].p;
  const int nvalid = nta * C4, warp = t >> 5, lane = t & 31;
  // a warp takes an output row and walks its TA x C values 64 float4 at a time, two per lane, so that a term (one
  // broadcast 16-byte read) serves two positions; the products are packed two-wide FMAs (the same roundings as
  // fmaf(coef * a, b, acc) per channel)
  auto f2 = [](float x, float y) { return make_float2(x, y); };
  for (int row = row_lo + warp; row < row_hi; row += 8) {
    const int t0 = op.term_off[row] - term0, t1 = op.term_off[row + 1] - term0;
    const bool add = op.accumulate && !(op.row_first && op.row_first[row]);
    float4 *orow = reinterpret_cast<float4 *>(D + ((size_t) op.row_out[row] * NA + a0) * C);
    for (int r = lane; r < nvalid; r += 64) {
      const bool has1 = r + 32 < nvalid;
      const int r1 = has1 ? r + 32 : r;
      float2 a0l = f2(0.f, 0.f), a0h = a0l, a1l = a0l, a1h = a0l;
      if (Bs) {
        for (int q = t0; q < t1; q++) {
          const int4 tm = sT[q];
          const float cf = __int_as_float(tm.z);
          const float2 c2 = f2(cf, cf);
          const float4 av0 = sA[tm.x + r], bv0 = Bs[tm.y + r], av1 = sA[tm.x + r1], bv1 = Bs[tm.y + r1];
          a0l = __ffma2_rn(__fmul2_rn(c2, f2(av0.x, av0.y)), f2(bv0.x, bv0.y), a0l);
          a0h = __ffma2_rn(__fmul2_rn(c2, f2(av0.z, av0.w)), f2(bv0.z, bv0.w), a0h);
          a1l = __ffma2_rn(__fmul2_rn(c2, f2(av1.x, av1.y)), f2(bv1.x, bv1.y), a1l);
          a1h = __ffma2_rn(__fmul2_rn(c2, f2(av1.z, av1.w)), f2(bv1.z, bv1.w), a1h);
        }
      } else {
        for (int q = t0; q < t1; q++) {
          const int4 tm = sT[q];
          const float cf = __int_as_float(tm.z);
          const float2 c2 = f2(cf, cf);
          const float4 av0 = sA[tm.x + r], av1 = sA[tm.x + r1];
          a0l = __ffma2_rn(c2, f2(av0.x, av0.y), a0l);
          a0h = __ffma2_rn(c2, f2(av0.z, av0.w), a0h);
          a1l = __ffma2_rn(c2, f2(av1.x, av1.y), a1l);
          a1h = __ffma2_rn(c2, f2(av1.z, av1.w), a1h);
        }
      }
      float4 o0 = make_float4(a0l.x, a0l.y, a0h.x, a0h.y), o1 = make_float4(a1l.x, a1l.y, a1h.x, a1h.y);
      if (add) {
        const float4 old0 = orow[r], old1 = orow[r1];
        o0.x += old0.x; o0.y += old0.y; o0.z += old0.z; o0.w += old0.w;
        o1.x += old1.x; o1.y += old1.y; o1.z += old1.z; o1.w += old1.w;
      }
      orow[r] = o0;
      if (has1) orow[r1] = o1;
    }
  }
}

void launch_prod(const ProdDev &op, const TensorDev *tensors, int NA, int na, int C, int nfA, int nfB, int nterms)
{
  if (op.nrows == 0 || na == 0) return;
  // tiled form: channels a multiple of 4 and at least one atom of input rows in shared memory
  if ((C & 3) == 0 && nfA > 0) {
    const bool two = op.srcB >= 0 && op.srcB != op.srcA;
    const size_t per_atom = (size_t) (nfA + (two ? nfB : 0)) * C * 4, fixed = (size_t) nterms * sizeof(int4) + 64;
    // several CTAs per SM (the load, compute and store phases of a tile overlap only across CTAs): a quarter of the
    // shared memory when that holds 4+ atoms, else half, else all of it
    static const size_t first = getenv("GRACE_B200_PROD_KB") ? (size_t) atoi(getenv("GRACE_B200_PROD_KB")) * 1024 : 54 * 1024;
    const size_t quarter = first, half = 110 * 1024, large = 200 * 1024;
    size_t budget = quarter;
    if (fixed + 4 * per_atom > quarter) budget = half;
    if (fixed + 4 * per_atom > half) budget = large;
    int TA = fixed < budget ? (int) std::min<size_t>(32, (budget - fixed) / per_atom) : 0;
    {    // a warp walks a row 64 float4 at a time: tiles whose rows are a multiple of that leave no lane idle
      const int unit = std::max(1, 64 / (C >> 2));
      if (TA > unit) TA = TA / unit * unit;
      while (TA >= 2 * unit && (na + TA - 1) / TA < dev().sm_count) TA = TA / 2 / unit * unit;    // few atoms: more tiles
    }
    // and where the tiles alone leave the GPU idle, the rows of a tile go to several CTAs (54 atoms: 12 -> 7 us a product)
    const int tiles = TA >= 1 ? (na + TA - 1) / TA : 1;
    const int gy = std::max(1, std::min((op.nrows + 3) / 4, 2 * dev().sm_count / tiles));
    if (TA >= 1) {
      const size_t smem = fixed + (size_t) TA * per_atom;
      static size_t attr = 48 * 1024;
      if (smem > attr) {
        GB_CUDA(cudaFuncSetAttribute(prod_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) large));
        attr = large;
      }
      GB_LAUNCH(prod_tile_kernel, dim3(tiles, gy), 256, smem, op, tensors, NA, na, TA, nfA, two ? nfB : 0, C);
      return;
    }
  }
  const long long row_len = (long long) NA * C, act_len = (long long) na * C;
  const dim3 grid(op.nrows, (unsigned) ((act_len + 255) / 256));
  GB_LAUNCH(prod_kernel, grid, 256, 0, op, tensors, row_len, act_len);
}

// ---- readouts (fp64) -------------------------------------------------------------------------------------------
// A thread per atom is a chain of a thousand dependent fp64 instructions, 88 us however few the atoms; a warp per atom is
// done in 20 us but takes five times the machine (GRACE-2L, 1,024,000 atoms: 10.4 against 2.2 ms).  The line is where the two
// meet.
constexpr int READOUT_WARP_ATOMS = 8192;

template<bool WARP>
__global__ void __launch_bounds__(128) readout_1l_kernel(ReadoutDev r, const float *__restrict__ rho, float *grho,
                                                         const int *__restrict__ mu, double *e_atom, int NA, int na, int a0,
                                                         int want_grad, const int *__restrict__ ilist)
{
  const int a = WARP ? blockIdx.x * 4 + (threadIdx.x >> 5) : blockIdx.x * 128 + threadIdx.x;
  if (a >= na) return;
  const int i = ilist ? ilist[a0 + a] : a0 + a;    // the atom of chunk position a
  const float *x = rho + (size_t) a * r.nrho;
  float *g = grho + (size_t) a * r.nrho;
  if (WARP) {
    const double e = readout_1l_warp(r, x, mu[i], g, want_grad, r.owned(i));
    if ((threadIdx.x & 31) == 0) e_atom[i] = e;
  } else {
    e_atom[i] = readout_1l_atom(r, x, mu[i], g, want_grad, r.owned(i));
  }
}

void launch_readout_1l(const ReadoutDev &r, const float *rho, float *grho, const int *mu, double *e_atom, int NA,
                       int na, int a0, int want_grad, const int *ilist)
{
  if (na == 0) return;
  if (na < READOUT_WARP_ATOMS)
    GB_LAUNCH((readout_1l_kernel<true>), (na + 3) / 4, 128, 0, r, rho, grho, mu, e_atom, NA, na, a0, want_grad, ilist);
  else
    GB_LAUNCH((readout_1l_kernel<false>), (na + 127) / 128, 128, 0, r, rho, grho, mu, e_atom, NA, na, a0, want_grad, ilist);
}

template<bool WARP>
__global__ void __launch_bounds__(128) readout_2l_kernel(ReadoutDev r, const float *__restrict__ rho_rows,
                                                         const float *__restrict__ I2, double *grho_rows, float *gI2,
                                                         const int *__restrict__ mu, double *e_atom, int NA, int na, int a0,
                                                         int want_grad, const int *__restrict__ ilist)
{
  const int a = WARP ? blockIdx.x * 4 + (threadIdx.x >> 5) : blockIdx.x * 128 + threadIdx.x;
  if (a >= na) return;
  const int nr = r.nrho;
  const size_t i = ilist ? (size_t) ilist[a0 + a] : (size_t) (a0 + a);    // the atom of chunk position a
  const bool own = r.owned((long long) i);
  if (WARP) {
    const double e = readout_2l_warp(r, rho_rows + i * nr, I2 + (size_t) a * nr, mu[i], grho_rows + i * nr, gI2 + (size_t) a * nr,
                                     want_grad, own);
    if ((threadIdx.x & 31) == 0) e_atom[i] = e;
  } else {
    e_atom[i] = readout_2l_atom(r, rho_rows + i * nr, I2 + (size_t) a * nr, mu[i], grho_rows + i * nr, gI2 + (size_t) a * nr,
                                want_grad, own);
  }
}

void launch_readout_2l(const ReadoutDev &r, const float *rho_rows, const float *I2, double *grho_rows, float *gI2,
                       const int *mu, double *e_atom, int NA, int na, int a0, int want_grad, const int *ilist)
{
  if (na == 0) return;
  if (na < READOUT_WARP_ATOMS)
    GB_LAUNCH((readout_2l_kernel<true>), (na + 3) / 4, 128, 0, r, rho_rows, I2, grho_rows, gI2, mu, e_atom, NA, na, a0, want_grad, ilist);
  else
    GB_LAUNCH((readout_2l_kernel<false>), (na + 127) / 128, 128, 0, r, rho_rows, I2, grho_rows, gI2, mu, e_atom, NA, na, a0, want_grad,
              ilist);
}

// out[a] = v[list[a]]
__global__ void __launch_bounds__(256) gather_int_kernel(const int *__restrict__ v, const int *__restrict__ list, int *out, long long n)
{
  const long long a = (long long) blockIdx.x * blockDim.x + threadIdx.x;
  if (a < n) out[a] = v[list[a]];
}

void launch_gather_int(const int *v, const int *list, int *out, long long n)
{
  if (n == 0) return;
  GB_LAUNCH(gather_int_kernel, (unsigned) ((n + 255) / 256), 256, 0, v, list, out, n);
}

// ---- chunk tensor <-> per-atom rows ----------------------------------------------------------------------------
template<class TR, bool TO_ROWS>
__global__ void __launch_bounds__(256) rows_kernel(float *t, TR *rows, int nf, int C, int NA, int na, int a0,
                                                   const int *__restrict__ ilist)
{
  const long long idx = (long long) blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long) na * nf * C;
  if (idx >= total) return;
  const int c = (int) (idx % C);
  const int f = (int) ((idx / C) % nf);
  const int a = (int) (idx / ((long long) C * nf));
  float *tp = t + ((size_t) f * NA + a) * C + c;
  const size_t i = ilist ? (size_t) ilist[a0 + a] : (size_t) (a0 + a);    // the atom of chunk position a
  TR *rp = rows + (i * nf + f) * C + c;
  if (TO_ROWS) *rp = (TR) *tp;
  else *tp = (float) *rp;
}

void launch_rows_from_chunk(const float *t, float *rows, int nf, int C, int NA, int na, int a0, const int *ilist)
{
  const long long total = (long long) na * nf * C;
  if (total == 0) return;
  GB_LAUNCH((rows_kernel<float, true>), (unsigned) ((total + 255) / 256), 256, 0, const_cast<float *>(t), rows, nf, C,
            NA, na, a0, ilist);
}
void launch_chunk_from_rows(float *t, const float *rows, int nf, int C, int NA, int na, int a0, const int *ilist)
{
  const long long total = (long long) na * nf * C;
  if (total == 0) return;
  GB_LAUNCH((rows_kernel<float, false>), (unsigned) ((total + 255) / 256), 256, 0, t, const_cast<float *>(rows), nf, C,
            NA, na, a0, ilist);
}
void launch_chunk_from_rows_f64(float *t, const double *rows, int nf, int C, int NA, int na, int a0, const int *ilist)
{
  const long long total = (long long) na * nf * C;
  if (total == 0) return;
  GB_LAUNCH((rows_kernel<double, false>), (unsigned) ((total + 255) / 256), 256, 0, t, const_cast<double *>(rows), nf,
            C, NA, na, a0, ilist);
}

// one warp per atom j: lanes over the `width` floats of a row, the atom's bonds one after the other
__global__ void __launch_bounds__(128) msg_grad_gather_kernel(BondsDev b, const int *__restrict__ rev,
                                                              const float *__restrict__ gslot, float *gmsg, int width,
                                                              const int *__restrict__ ilist, long long n,
                                                              const int *__restrict__ perm, int nlocal)
{
  const long long a = (long long) blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x & 31;
  if (a >= n) return;
  const long long j = ilist ? ilist[a] : a;
  const long long base = b.off[j];
  const int nb = b.cnt[j];
  for (int c0 = 0; c0 < width; c0 += 128) {    // 4 floats per lane and pass
    const int c = c0 + 4 * lane;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < width) {
      for (int e = 0; e < nb; e++) {
        if (perm && perm[__float_as_int(b.rec[base + e].w)] >= nlocal) continue;
        const size_t p = (size_t) rev[b.cslot[base + e]];
        const float4 v = __ldg(reinterpret_cast<const float4 *>(gslot + p * width + c));
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
      *reinterpret_cast<float4 *>(gmsg + (size_t) j * width + c) = acc;
    }
  }
}

void launch_msg_grad_gather(const BondsDev &b, const int *rev, const float *gslot, float *gmsg, int width, const int *ilist,
                            long long n, const int *perm, int nlocal)
{
  if (n == 0) return;
  GB_LAUNCH(msg_grad_gather_kernel, (unsigned) ((n + 3) / 4), 128, 0, b, rev, gslot, gmsg, width, ilist, n, perm, nlocal);
}

// one warp per atom with bonds: own sum by shuffles, neighbours by atomics
__global__ void __launch_bounds__(128) force_scatter_kernel(BondsDev b, const float *__restrict__ fv, double *forces, long long n)
{
  const long long i = (long long) blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x & 31;
  if (i >= n) return;
  const long long base = b.off[i];
  const int nb = b.cnt[i];
  double f0 = 0.0, f1 = 0.0, f2 = 0.0;
  for (int e = lane; e < nb; e += 32) {
    const size_t q = (size_t) b.cslot[base + e];
    const size_t j = (size_t) __float_as_int(b.rec[base + e].w);
    const double x = fv[3 * q], y = fv[3 * q + 1], z = fv[3 * q + 2];
    f0 += x; f1 += y; f2 += z;
    atomicAdd(forces + 3 * j, -x);
    atomicAdd(forces + 3 * j + 1, -y);
    atomicAdd(forces + 3 * j + 2, -z);
  }
  for (int s = 16; s > 0; s >>= 1) {
    f0 += __shfl_xor_sync(0xffffffffu, f0, s);
    f1 += __shfl_xor_sync(0xffffffffu, f1, s);
    f2 += __shfl_xor_sync(0xffffffffu, f2, s);
  }
  if (lane == 0 && nb > 0) {
    atomicAdd(forces + 3 * (size_t) i, f0);
    atomicAdd(forces + 3 * (size_t) i + 1, f1);
    atomicAdd(forces + 3 * (size_t) i + 2, f2);
  }
}

void launch_force_scatter(const BondsDev &b, const float *fv, double *forces, long long n)
{
  if (n == 0) return;
  GB_LAUNCH(force_scatter_kernel, (unsigned) ((n + 3) / 4), 128, 0, b, fv, forces, n);
}

// Zero fill of a 16-byte aligned buffer whose size is a multiple of 4 bytes: 16-byte stores, a grid-stride loop over a
// grid that fills the GPU.  For buffers of hundreds of megabytes this is several times faster than the driver's memset.
__global__ void __launch_bounds__(256) fill_zero_kernel(float4 *__restrict__ p4, long long n4, float *__restrict__ tail, int ntail)
{
  const long long stride = (long long) gridDim.x * blockDim.x;
  for (long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) p4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (blockIdx.x == 0 && (int) threadIdx.x < ntail) tail[threadIdx.x] = 0.0f;
}

void launch_fill_zero(void *p, size_t bytes)
{
  if (bytes == 0) return;
  if ((reinterpret_cast<uintptr_t>(p) & 15) != 0 || (bytes & 3) != 0 || bytes < (1u << 20)) {
    GB_CUDA(cudaMemsetAsync(p, 0, bytes, dev().stream));
    return;
  }
  const long long n4 = (long long) (bytes / 16);
  const int ntail = (int) ((bytes % 16) / 4);
  const unsigned grid = (unsigned) std::min<long long>((n4 + 255) / 256, (long long) dev().sm_count * 16);
  GB_LAUNCH(fill_zero_kernel, grid, 256, 0, reinterpret_cast<float4 *>(p), n4, reinterpret_cast<float *>(p) + 4 * n4, ntail);
}

__global__ void __launch_bounds__(256) add_f64_kernel(const double *__restrict__ v, double *out, long long n)
{
  const long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += v[i];
}

void launch_add_f64(const double *v, double *out, long long n)
{
  if (n == 0) return;
  GB_LAUNCH(add_f64_kernel, (unsigned) ((n + 255) / 256), 256, 0, v, out, n);
}

// ---- per-structure sums (deterministic: fixed tree per segment) ------------------------------------------------
// few long segments (one large structure): NB blocks per (segment, component) write partial sums over equal slices
// of the segment, a second launch adds them in slice order - still a fixed tree
__global__ void __launch_bounds__(256) segment_partial_kernel(const double *__restrict__ v, int K,
                                                              const int *__restrict__ seg, double *partial)
{
  __shared__ double sh[256];
  const int s = blockIdx.x, k = blockIdx.y, b = blockIdx.z, NB = gridDim.z;
  const long long s0 = seg[s], len = seg[s + 1] - s0, per = (len + NB - 1) / NB;
  const long long lo = s0 + b * per, hi = min(s0 + len, lo + per);
  double acc = 0.0;
  for (long long i = lo + threadIdx.x; i < hi; i += blockDim.x) acc += v[(size_t) i * K + k];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if ((int) threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[((size_t) s * K + k) * NB + b] = sh[0];
}

__global__ void __launch_bounds__(32) segment_final_kernel(const double *__restrict__ partial, int NB, double *out)
{
  const int sk = blockIdx.x;    // segment * K + component
  if (threadIdx.x != 0) return;
  double acc = 0.0;
  for (int b = 0; b < NB; b++) acc += partial[(size_t) sk * NB + b];
  out[sk] = acc;
}

void launch_segment_sum(const double *v, int K, const int *seg, int nseg, double *out, double *scratch, int nb)
{
  if (nseg == 0) return;
  GB_LAUNCH(segment_partial_kernel, dim3(nseg, K, nb), 256, 0, v, K, seg, scratch);
  GB_LAUNCH(segment_final_kernel, nseg * K, 32, 0, scratch, nb, out);
}

// What leaves an evaluation, in one launch: blocks [0, nsum) add the per-atom energies and virial rows of a structure
// each (seven columns at once, by a fixed tree), the others give a warp per atom that gathers its
// force in list order and moves its per-atom values to the caller's order; the error words of the call are
// collected beside the sums so that one copy brings everything to the host.  Bound by launch latency for small
// structures, where this was up to nine launches and copies of 2 - 7 us each.
__global__ void __launch_bounds__(256) finish_kernel(FinishDev F, int nsum)
{
  const int t = threadIdx.x;
  if ((int) blockIdx.x < nsum) {
    __shared__ double sh[7][256];
    const int s = blockIdx.x, lo = F.seg[s], hi = F.seg[s + 1];
    double acc[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int i = lo + t; i < hi; i += 256) {
      acc[0] += F.e_atom[i];
      if (F.virial) {
#pragma unroll
        for (int k = 0; k < 6; k++) acc[1 + k] += F.vir_atom[6 * (size_t) i + k];
      }
    }
#pragma unroll
    for (int k = 0; k < 7; k++) sh[k][t] = acc[k];
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
      if (t < st)
#pragma unroll
        for (int k = 0; k < 7; k++) sh[k][t] += sh[k][t + st];
      __syncthreads();
    }
    if (t == 0 && F.energy) F.energy[s] = sh[0][0];
    if (t < 6 && F.virial) F.virial[6 * (size_t) s + t] = sh[1 + t][0];
    return;
  }
  const int b = (int) blockIdx.x - nsum, i = b * 8 + (t >> 5), lane = t & 31;
  if (b == 0 && t == 0 && F.status) {
    const int f = F.nl_flag[0] | F.nl_flag[1], e = F.tc_flag ? *F.tc_flag : 0;
    F.status[0] = F.first ? f : F.status[0] | f;
    F.status[1] = F.first ? e : F.status[1] | e;
  }
  if (i >= F.n) return;
  const size_t at = F.perm[i];
  if (F.forces) {
    double f0 = 0.0, f1 = 0.0, f2 = 0.0;
    for (long long q = F.off[i] + lane; q < F.off[i + 1]; q += 32) {
      const long long p = F.rev[q];
      f0 += (double) F.fv[3 * q] - (double) F.fv[3 * p];
      f1 += (double) F.fv[3 * q + 1] - (double) F.fv[3 * p + 1];
      f2 += (double) F.fv[3 * q + 2] - (double) F.fv[3 * p + 2];
    }
    for (int s = 16; s > 0; s >>= 1) {
      f0 += __shfl_xor_sync(0xffffffffu, f0, s);
      f1 += __shfl_xor_sync(0xffffffffu, f1, s);
      f2 += __shfl_xor_sync(0xffffffffu, f2, s);
    }
    if (lane < 3) F.forces[3 * at + lane] = lane == 0 ? f0 : lane == 1 ? f1 : f2;
  }
  if (lane == 0 && F.energies) F.energies[at] = F.e_atom[i];
  if (F.uq && lane < 3) (lane == 0 ? F.gamma : lane == 1 ? F.sigma : F.cluster)[at] = F.uq[(size_t) lane * F.n + i];
}

void launch_finish(const FinishDev &F, int nsum)
{
  const int atom_blocks = F.forces || F.energies || F.uq ? (F.n + 7) / 8 : 1;
  GB_LAUNCH(finish_kernel, nsum + atom_blocks, 256, 0, F, nsum);
}

}    // namespace gb
