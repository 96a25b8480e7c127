// FC layers, reduces and their adjoints of the dense network on the 5th-generation tensor cores.
//
// On chunk tensors [function][atom][channel] an operation  out[row] (+)= sum_items scale * W_item^T x[item]  is a
// grouped GEMM whose long dimension is the atoms: for an output row and a tile of 128 atoms,
//     D[128 atoms][n_out] = sum_items X_item[128 atoms][K] . W_item[K][n_out],
// with X_item a contiguous block of the source tensor.  A CTA owns up to 256 / n_out atom tiles at a time and keeps two
// sets of fp32 accumulators for them in tensor memory; for every item of the row its producer warps write the tile's
// activations as three bf16 operand images into a ring of shared-memory stages (canonical K-major layout, 8-row x 16-byte
// core matrices), the item's weight images (split once when the model is loaded) arrive by one bulk asynchronous copy, and
// one thread issues tcgen05.mma kind::f16 M = 128, N = n_out, K = 16.
// Accuracy.  x = x1 + x2 + x3, each part the bf16 nearest to what the ones before leave, is all 24 bits of an fp32 number, and
//     a b ~ a3 b1 + a1 b3 + a2 b2 + a2 b1 + a1 b2 + a1 b1
// leaves out 2^-26 of a b.  The accumulators cut off what does not fit their 24 bits, with a bias towards zero that a sum over
// many atoms keeps; the products a1 b1 have 16 bits, so that adding them among themselves cuts off little, and where fp32 sums are
// the measure the five small products go to an accumulator of their own (SEP), which the epilogue adds with rounding.
// Two tf32 parts take as many instructions (half as wide in K) and more shared memory, but are 22 bits of an operand with products of
// 22.  Errors against fp64 (2-norm, several structures; fp32 FMA kernels / two tf32 parts / this): per-atom energies of GRACE-1L of
// order 4, 588 atoms 3.9e-7 / 3.0e-7 / 2.6e-7, GRACE-2L, 600 atoms 3.8e-7 / 3.8e-7 / 3.5e-7, GRACE-3L, 54 atoms 2.9e-7 / 4.7e-7 /
// 2.4e-7, forces along random directions 7.0e-7 / 1.4e-6 / 6.5e-7; extrapolation grade of GRACE-2L, 600 atoms 3.0e-8 / 4.7e-7 / 2.6e-8;
// virial of GRACE-2L, 600 atoms 5.8e-7 / 2.0e-6 / 5.4e-7.  Above 18,944 atoms (no SEP): GRACE-2L energies 2.5e-7 / 2.7e-7 / 2.0e-7, forces
// 6.2e-7 / 6.1e-7 / 5.3e-7; GRACE-3L energies 1.22e-6 / 1.23e-6 / 1.17e-6 (the first figure with two tf32 parts in all but the
// per-element sums).  Times are those of two tf32 parts within 0.3 %; SEP at all sizes would bring the last figure to 3.0e-7 and costs 2 % (GRACE-2L,
// 1,024,000 atoms 222.6 -> 227.5 ms) to 5 % (GRACE-1L, 128,000 atoms).
// The global loads of the next two tiles are in flight in registers while a tile is written, all items of a
// row accumulate in tensor memory, and the epilogue warps write each output row once while the next row's matrix
// instructions run.
// Widths are padded with zeros to K = 16, 32 or 64 and N a multiple of 16, so every operation of up to 64 inputs runs here.
// Operations whose weights depend on the central atom's element (the reduces to densities and messages, their adjoints) take
// tiles of atoms of ONE element: the atoms are gathered through an index (ElemOrder) that groups them by element, a row of
// 9 - 64 channels each, and the weight images are chosen per tile.  With the elements mixed in a tile the weights of every
// element present passed through shared memory: 557,000 atoms of 89 elements 82 ms, 1,024,000 atoms of 3 elements 20.7 ms per
// evaluation of GRACE-2L; grouped 9.3 and 16.2 ms.
// Independent operations of the same shape are one launch (Engine::setup_steps): rows carry their tensor and whether they add.
// Same mathematics as mv_kernel (chain.cu); reference: fc_fwd / mv_batch, libgrace/include/grace/fused_cpu.h:294-356,
// GPU fc_fwd4 libgrace/include/grace/kk/fused_dense.h:441-495.
//
// Every wait on the tensor cores is bounded: a wait that runs out sets the error flag, the CTA frees its tensor memory
// and returns, and the host reports the failure.
#include "mv_tc.h"

#include <algorithm>
#include <cstring>
#include <map>

namespace gb {

namespace {

constexpr int TM = 128;         // atoms of a tile = rows of an MMA = tensor-memory lanes
constexpr int NTH = 256;
constexpr int NW = NTH / 32;
constexpr int TMEM_COLS = 512;
constexpr int MAX_TILES = 16;   // atom tiles a CTA holds accumulators for
constexpr int MAX_TENSORS = 64;
constexpr int MAX_ITEMS = MVTensorCore::MAX_ITEMS, MAX_ROWS = MVTensorCore::MAX_ROWS;    // tables of an operation staged in shared memory
constexpr long long WAIT_CYCLES = 40000000LL;    // ~20 ms: far beyond any tile, far below a watchdog

constexpr int LONG_ROW = 16;    // items of a row from which on it goes in parts while fp32 sums are the measure
constexpr int PARTS = 3;        // bf16 numbers an fp32 operand is split into
// the products of parts (activation, weight) that are formed, small ones first
__device__ constexpr int PRODUCTS[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};

// byte offset of element (r, k) of a K-major bf16 operand tile with K columns (canonical layout, no swizzle)
__host__ __device__ inline int tile_off(int r, int k, int K) { return (r >> 3) * (K >> 3) * 128 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2; }

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned) __cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long make_desc(unsigned addr, int K)
{
  const unsigned long long lbo = 128 >> 4, sbo = ((K >> 3) * 128) >> 4;
  return (unsigned long long) ((addr & 0x3ffff) >> 4) | (lbo << 16) | (sbo << 32) | (1ull << 46);
}

// fp32 accumulate, bf16 x bf16, both operands K-major, M = 128, N = n
__device__ __forceinline__ unsigned make_idesc(int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned) (n >> 3) << 17) | ((unsigned) (TM >> 4) << 24); }

__device__ __forceinline__ void mma_bf16_ss(unsigned tmem_d, unsigned long long da, unsigned long long db, unsigned idesc, bool accumulate)
{
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"((unsigned) accumulate) : "memory");
}

// four activations in their bf16 parts, 8 bytes per part; the differences are exact in fp32
__device__ __forceinline__ void split4(float4 x, float sc, uint2 (&part)[PARTS])
{
  float v[4] = {x.x * sc, x.y * sc, x.z * sc, x.w * sc};
#pragma unroll
  for (int p = 0; p < PARTS; p++) {
    unsigned r[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r[q]) : "f"(v[2 * q + 1]), "f"(v[2 * q]));    // the second operand to the lower half
      v[2 * q] -= __uint_as_float(r[q] << 16);
      v[2 * q + 1] -= __uint_as_float(r[q] & 0xffff0000u);
    }
    part[p] = make_uint2(r[0], r[1]);
  }
}

template<int NC> __device__ __forceinline__ void tmem_ld(unsigned taddr, float (&v)[NC]);

template<> __device__ __forceinline__ void tmem_ld<32>(unsigned taddr, float (&v)[32])
{
  unsigned r[32];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
               "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                 "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                 "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

template<> __device__ __forceinline__ void tmem_ld<16>(unsigned taddr, float (&v)[16])
{
  unsigned r[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// 16 columns of 32 tensor-memory lanes (two 16-lane loads and one wait).  A thread gets, for groups j of 8 columns, columns
// 8 j + 2 (lane & 3) and the next of the rows lane / 4 (v[4 j], v[4 j + 1]) and lane / 4 + 8 (v[4 j + 2], v[4 j + 3]), then the
// same of rows + 16 behind the first 8 values: a store of two columns by the warp fills whole 32-byte sectors of 8 rows.
__device__ __forceinline__ void tmem_ld_rows(unsigned taddr, float (&v)[16])
{
  unsigned r[16];
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n\t"
               "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];\n\t"
               "tcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr), "r"(taddr + (16u << 16)) : "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// position in the loop nest (round of tiles, output row, item of the row, tile of the round)
struct Cursor {
  int tile0, nt, row, it, i0, i1, tt;
  bool valid;
};

// Activation tile of a fill: K4 = K / 4 float4 per atom row.  A warp instruction covers 8 atom rows x 4 consecutive
// float4 (64 contiguous bytes of each row in global memory, 512 contiguous bytes = 4 core matrices in shared memory:
// no bank conflicts); the 16 x CG such units of a tile go round the producer warps.
template<int K> struct TileRegs {
  static constexpr int K4 = K / 4, CG = (K4 + 3) / 4, UNITS = 16 * CG, PER = (UNITS + NW - 1) / NW;
  float4 v[PER];
};

// Warp-specialised: warps 0-7 produce (global loads two tiles ahead in registers, the operand images of a tile
// into one of S shared-memory stages, the weight images of an item into a ring of S buffers), warp 8 issues the matrix
// instructions (one thread; nothing else runs on its critical path), the warps from 9 on move finished accumulators from tensor
// memory to global memory.  Two sets of accumulators (TB tiles x n_out columns each) take turns, so the epilogue of a
// row overlaps the matrix instructions of the next.  Hand-offs are mbarriers: full[s] (256 producer arrivals) / empty[s]
// (tcgen05.commit) per stage, accfull[set] (tcgen05.commit after the last item of a row) / accempty[set] (every
// epilogue thread).  A wait that runs out raises `abort`, which every other wait sees, and all roles leave together.
constexpr int NPROD = NTH;
// grouped atoms: two epilogue warps per quarter of the lanes (the sums over several accumulators and the scattered rows take longer
// than the matrix instructions of a row: 1,024,000 atoms, 16 inputs, 9.4 -> 6.3 ms; 7.1 with the accumulator of the small products).  17 warps leave 96 registers per thread, not
// enough for producers that hold two tiles of 64 channels (1.87 -> 2.13 ms) or for the other epilogue
__host__ __device__ constexpr int epilogue_threads(int K, bool elem) { return elem && K < 64 ? 256 : 128; }
__host__ __device__ constexpr int block_threads(int K, bool elem) { return NTH + 32 + epilogue_threads(K, elem); }

// SEP: the small products have an accumulator of their own behind the op.sub accumulators of a1 b1.
template<int K, int CB, int S, bool ELEM, bool SEP>
__global__ void __launch_bounds__(block_threads(K, ELEM), 1) mv_tc_kernel(MVTCDev op, const TensorDev *__restrict__ Tg, int ntensors, int NA,
                                                            int na, int TB, int tmem_cols, int *error)
{
  using TR = TileRegs<K>;
  constexpr int K4 = TR::K4, UNITS = TR::UNITS, PER = TR::PER;
  constexpr int NEPI = epilogue_threads(K, ELEM), NTHREADS = block_threads(K, ELEM);
  constexpr int A_BYTES = TM * K * 2;    // one image (part) of an activation tile
  extern __shared__ __align__(1024) char smem[];
  __shared__ unsigned long long s_full[S], s_empty[S], s_accfull[2], s_accempty[2];
  __shared__ unsigned s_tmem;
  __shared__ int s_abort;
  __shared__ TensorDev s_T[MAX_TENSORS];
  // the operation's tables: every role walks them once per fill, so they live in shared memory
  __shared__ MVItem s_items[MAX_ITEMS];
  __shared__ MVRowDev s_rows[MAX_ROWS];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int N = op.N;
  const int W_BYTES = N * K * 2;                         // one image of a weight matrix
  char *A_st = smem;                                     // stage s at s * PARTS * A_BYTES
  char *W_st = smem + (size_t) S * PARTS * A_BYTES;      // buffer b at b * PARTS * W_BYTES
  float *tr_all = reinterpret_cast<float *>(W_st + (size_t) S * PARTS * W_BYTES);    // transpose buffers of the epilogue warps
  for (int q = t; q < ntensors; q += NTHREADS) s_T[q] = Tg[q];
  for (int q = t; q < op.nrows; q += NTHREADS) s_rows[q] = op.rows[q];
  for (int q = t; q < op.nitems; q += NTHREADS) s_items[q] = op.items[q];
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    for (int s = 0; s < S; s++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s_full[s])), "r"(NPROD) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_empty[s])) : "memory");
    }
    for (int s = 0; s < 2; s++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_accfull[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s_accempty[s])), "r"(NEPI) : "memory");
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = s_tmem;
  const int ntiles = ELEM ? op.tiles[0] : (na + TM - 1) / TM, per_round = gridDim.x * TB;
  volatile int *abort_flag = &s_abort;

  // bounded wait that also gives up when another role did
  auto wait = [&](unsigned long long *bar, unsigned parity) -> bool {
    const unsigned addr = smem_u32(bar);
    const long long t0 = clock64();
    for (;;) {
      unsigned ok;
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(ok) : "r"(addr), "r"(parity), "r"(20000u) : "memory");
      if (ok) return true;
      if (*abort_flag) return false;
      if (clock64() - t0 > WAIT_CYCLES) {
        *abort_flag = 1;
        return false;
      }
    }
  };
  auto start = [&](Cursor &c, int tile0, int row) {
    c.tile0 = tile0;
    c.row = row;
    c.valid = tile0 < ntiles && row < op.nrows;
    if (!c.valid) return;
    c.nt = min(TB, ntiles - tile0);
    c.i0 = c.it = s_rows[row].i0;
    c.i1 = op.parts ? min(c.i0 + op.sub, s_rows[row].i1) : s_rows[row].i1;
    c.tt = 0;
  };
  // rows in parts: the next items of the same row, an accumulator each
  auto next_part = [&](Cursor &c) -> bool {
    if (c.i1 == s_rows[c.row].i1) return false;
    c.i0 = c.it = c.i1;
    c.i1 = min(c.i0 + op.sub, s_rows[c.row].i1);
    return true;
  };
  auto advance = [&](Cursor &c) {
    if (++c.tt < c.nt) return;
    c.tt = 0;
    if (++c.it < c.i1 || next_part(c)) return;
    int row = c.row + gridDim.y, tile0 = c.tile0;
    if (row >= op.nrows) {
      row = blockIdx.y;
      tile0 += per_round;
    }
    start(c, tile0, row);
  };
  auto next_row = [&](Cursor &c) {    // first fill of the row, or part of a row, after c's
    if (next_part(c)) return;
    int row = c.row + gridDim.y, tile0 = c.tile0;
    if (row >= op.nrows) {
      row = blockIdx.y;
      tile0 += per_round;
    }
    start(c, tile0, row);
  };

  if (warp < NW) {
    // ---------------- producers ----------------
    // grouped atoms: this thread's two rows of the tile at hand (the tile stays while the items of all rows pass)
    int tile_of_rows = -1, arow[2] = {-1, -1};
    auto load_tile = [&](const Cursor &c, TR &r) {
      const MVItem item = s_items[c.it];
      const TensorDev src = s_T[item.src];
      const int atom0 = (c.tile0 + c.tt) * TM, valid = ELEM ? TM : min(TM, na - atom0);
      const float *base = src.p + (size_t) item.irow * NA * src.C;
      const bool vec = ((src.C | item.n_in) & 3) == 0;
      if (ELEM && tile_of_rows != c.tile0 + c.tt) {
        tile_of_rows = c.tile0 + c.tt;
        arow[0] = __ldg(op.order + atom0 + warp * 8 + (lane & 7));
        arow[1] = __ldg(op.order + atom0 + (warp + NW) * 8 + (lane & 7));
      }
#pragma unroll
      for (int j = 0; j < PER; j++) {
        const int u = warp + NW * j, row = (u % 16) * 8 + (lane & 7), c4 = (u / 16) * 4 + (lane >> 3);
        r.v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (u >= UNITS || row >= valid || 4 * c4 >= item.n_in) continue;
        const int a = ELEM ? arow[j & 1] : atom0 + row;    // (16 groups of rows, NW = 8 warps: even and odd j)
        if (ELEM && a < 0) continue;
        const float *x = base + (size_t) a * src.C + 4 * c4;
        if (vec) r.v[j] = __ldg(reinterpret_cast<const float4 *>(x));
        else {
          r.v[j].x = __ldg(x);
          if (4 * c4 + 1 < item.n_in) r.v[j].y = __ldg(x + 1);
          if (4 * c4 + 2 < item.n_in) r.v[j].z = __ldg(x + 2);
          if (4 * c4 + 3 < item.n_in) r.v[j].w = __ldg(x + 3);
        }
      }
    };
    Cursor cur, nxt, nxt2;
    start(cur, blockIdx.x * TB, blockIdx.y);
    TR regsA, regsB;
    if (cur.valid) load_tile(cur, regsA);
    nxt = cur;
    if (cur.valid) advance(nxt);
    if (nxt.valid) load_tile(nxt, regsB);
    int fill = 0, item_no = -1;
    bool ok = true;
    // one fill: `mine` holds the tile at `cur`; after its conversion it receives the tile two fills ahead
    auto step = [&](TR &mine) {
      nxt2 = nxt;
      if (nxt.valid) advance(nxt2);
      const int s = fill % S;
      // the matrix instructions that read this stage S fills ago (and everything issued before them) are done
      if (fill >= S) {
        ok = wait(&s_empty[s], (unsigned) ((fill / S - 1) & 1));
        if (!ok) return;
      }
      const MVItem item = s_items[cur.it];
      if (ELEM || cur.tt == 0) {    // first tile of an item (every tile of its own element): its weight images
        item_no++;
        if (t == 0) {
          // one bulk asynchronous copy; its bytes are counted by this stage's `full` barrier, so the matrix instructions
          // of the fill start when the image and the 256 arrivals are there, and no producer waits for the copy
          const unsigned bar = smem_u32(&s_full[s]), dst = smem_u32(W_st + (size_t) (item_no % S) * PARTS * W_BYTES);
          const int e = ELEM ? __ldg(op.tiles + 1 + cur.tile0 + cur.tt) : 0;
          const char *src = op.images + ((size_t) e * op.nmat + item.mat) * PARTS * W_BYTES;
          asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"((unsigned) (PARTS * W_BYTES)) : "memory");
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                       ::"r"(dst), "l"(src), "r"((unsigned) (PARTS * W_BYTES)), "r"(bar) : "memory");
        }
      }
      {    // registers -> operand images of stage s
        char *img = A_st + (size_t) s * PARTS * A_BYTES;
#pragma unroll
        for (int j = 0; j < PER; j++) {
          const int u = warp + NW * j, c4 = (u / 16) * 4 + (lane >> 3);
          if (u < UNITS && c4 < K4) {
            const int off = ((u % 16) * (K4 / 2) + (c4 >> 1)) * 128 + (lane & 7) * 16 + (c4 & 1) * 8;
            uint2 part[PARTS];
            split4(mine.v[j], item.scale, part);
#pragma unroll
            for (int p = 0; p < PARTS; p++) *reinterpret_cast<uint2 *>(img + p * A_BYTES + off) = part[p];
          }
        }
      }
      if (nxt2.valid) load_tile(nxt2, mine);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&s_full[s])) : "memory");
      fill++;
      cur = nxt;
      nxt = nxt2;
    };
    while (cur.valid && ok) {
      step(regsA);
      if (!cur.valid || !ok) break;
      step(regsB);
    }
  } else if (warp == NW) {
    // ---------------- matrix-instruction issuer ----------------
    if (lane == 0) {
      const unsigned idesc = make_idesc(N);
      Cursor cur;
      start(cur, blockIdx.x * TB, blockIdx.y);
      int fill = 0, item_no = -1, rowc = 0;
      bool ok = true;
      while (cur.valid && ok) {
        const int s = fill % S, set = rowc & 1;
        if (ELEM || cur.tt == 0) item_no++;
        if (cur.it == cur.i0 && cur.tt == 0 && rowc >= 2) {    // first fill of a row: its accumulators were read out
          ok = wait(&s_accempty[set], (unsigned) ((rowc / 2 - 1) & 1));
          if (!ok) break;
        }
        ok = wait(&s_full[s], (unsigned) ((fill / S) & 1));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned long long dA = make_desc(smem_u32(A_st + (size_t) s * PARTS * A_BYTES), K);
        const unsigned long long dB = make_desc(smem_u32(W_st + (size_t) (item_no % S) * PARTS * W_BYTES), K);
        const int at = cur.it - cur.i0;    // items take the accumulators of a1 b1 in turn
        const unsigned base = tmem + (unsigned) ((set * TB + cur.tt) * op.cols), d1 = base + (unsigned) (at % op.sub * N);
        const unsigned ds = SEP ? base + (unsigned) (op.sub * N) : d1;
        const bool acc1 = at >= op.sub, accs = SEP ? at > 0 : acc1;
#pragma unroll
        for (int q = 0; q < 6; q++) {
          const bool big = SEP && q == 5;
          const unsigned long long a = dA + (unsigned long long) (PRODUCTS[q][0] * (A_BYTES >> 4));
          const unsigned long long b = dB + (unsigned long long) (unsigned) (PRODUCTS[q][1] * (W_BYTES >> 4));
#pragma unroll
          for (int ks = 0; ks < K / 16; ks++)
            mma_bf16_ss(big ? d1 : ds, a + (unsigned long long) (ks * 16), b + (unsigned long long) (ks * 16), idesc,
                        big ? acc1 || ks > 0 : accs || q > 0 || ks > 0);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&s_empty[s])) : "memory");
        Cursor nx = cur;
        advance(nx);
        if (!nx.valid || nx.row != cur.row || nx.tile0 != cur.tile0 || nx.i0 != cur.i0) {    // the row is complete once these are done
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&s_accfull[set])) : "memory");
          rowc++;
        }
        fill++;
        cur = nx;
      }
    }
  } else {
    // ---------------- epilogue: tensor memory -> global, once per output row ----------------
    // Each warp moves blocks of 32 atoms x CB columns of its tensor-memory lanes: registers (a lane holds one atom's
    // columns) -> a padded transpose buffer of its own -> global memory with whole 128-byte lines per store
    const int ew = warp & 3;    // the quarter of the tensor-memory lanes this warp may read (warp id modulo 4)
    const int half = (warp - NW - 1) >> 2;    // grouped atoms: the warps of a quarter take the blocks in turn
    float *tr = tr_all + ew * (32 * (CB + 4));
    constexpr int LPR = CB / 4, RPI = 32 / LPR;    // lanes per atom row, atom rows per store instruction
    Cursor cur;
    start(cur, blockIdx.x * TB, blockIdx.y);
    int rowc = 0;
    bool ok = true;
    while (cur.valid && ok) {
      const int set = rowc & 1;
      ok = wait(&s_accfull[set], (unsigned) ((rowc / 2) & 1));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const MVRowDev row = s_rows[cur.row];
      const TensorDev dstT = s_T[row.dst];
      float *const out = dstT.p + (size_t) row.out * NA * dstT.C;
      const int nblk = N / CB, nb = cur.nt * nblk;
      if constexpr (ELEM) {    // rows of single atoms, 32-byte sectors straight from registers
        // later parts of a row add to what this thread wrote before
        const bool add = row.accumulate || cur.i0 > row.i0;
        const bool vec = ((dstT.C | row.n_out) & 1) == 0;
        for (int b = half; b < nb; b += NEPI / 128) {
          const int tt = b / nblk, c0 = (b - tt * nblk) * CB;
          int at[4];    // atoms of the thread's rows lane / 4 + 8 q, -1: none
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const int r = (cur.tile0 + tt) * TM + ew * 32 + 8 * q + (lane >> 2);
            at[q] = __ldg(op.order + r);
          }
          float *const o = out + c0 + 2 * (lane & 3);
          // value pair p: columns c0 + 8 j + 2 (lane & 3) and the next of row q
          auto row_of = [](int p) { return p / (CB / 4) * 2 + (p & 1); };
          auto col_of = [](int p) { return p % (CB / 4) / 2 * 8; };
          float2 old[CB / 2];
          if (add && vec) {
#pragma unroll
            for (int p = 0; p < CB / 2; p++) {
              const int a = at[row_of(p)];
              old[p] = a >= 0 && c0 + col_of(p) + 2 * (lane & 3) < row.n_out
                           ? __ldcg(reinterpret_cast<const float2 *>(o + (size_t) a * dstT.C + col_of(p))) : make_float2(0.f, 0.f);
            }
          }
          float v[CB];
          const unsigned from = tmem + ((unsigned) (ew * 32) << 16) + (unsigned) ((set * TB + tt) * op.cols + c0);
          tmem_ld_rows(from, v);
          const int nacc = cur.i1 - cur.i0;
          for (int k = 1; k < nacc + (SEP ? 1 : 0); k++) {    // the other accumulators of the row, the one of the small products last
            float w[CB];
            tmem_ld_rows(from + (unsigned) ((k < nacc ? k : op.sub) * N), w);
#pragma unroll
            for (int q = 0; q < CB; q++) v[q] += w[q];
          }
#pragma unroll
          for (int p = 0; p < CB / 2; p++) {
            const int a = at[row_of(p)], c = c0 + col_of(p) + 2 * (lane & 3);
            if (a < 0 || c >= row.n_out) continue;
            float *const d = o + (size_t) a * dstT.C + col_of(p);
            float2 x = make_float2(v[2 * p], v[2 * p + 1]);
            if (vec) {
              if (add) {
                x.x += old[p].x;
                x.y += old[p].y;
              }
              *reinterpret_cast<float2 *>(d) = x;
            } else {    // rows of an odd width: value by value
              d[0] = add ? d[0] + x.x : x.x;
              if (c + 1 < row.n_out) d[1] = add ? d[1] + x.y : x.y;
            }
          }
        }
      } else {
        const bool add = row.accumulate || cur.i0 > row.i0, vec = ((dstT.C | row.n_out) & 3) == 0;
        // atom of row r of this warp's quarter of tile tt, -1: none
        auto atom_of = [&](int tt, int r) {
          const int at = (cur.tile0 + tt) * TM + ew * 32 + r;
          return at < na ? at : -1;
        };
        // the old values of an accumulating row are fetched one block ahead of the block being written (later parts of a row add to
        // what this thread wrote before)
        float4 old[32 / RPI], oldn[32 / RPI];
        auto load_old = [&](int b, float4 (&o)[32 / RPI]) {
          const int tt = b / nblk, c0 = (b - tt * nblk) * CB;
#pragma unroll
          for (int j = 0; j < 32 / RPI; j++) {
            const int cq = lane % LPR, a = b < nb && c0 + 4 * cq < row.n_out ? atom_of(tt, j * RPI + lane / LPR) : -1;
            o[j] = a >= 0 ? __ldcg(reinterpret_cast<const float4 *>(out + (size_t) a * dstT.C + c0) + cq) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        };
        if (add && vec) load_old(0, oldn);
        for (int b = 0; b < nb; b++) {
          const int tt = b / nblk, c0 = (b - tt * nblk) * CB;
          float v[CB];
          const unsigned at = tmem + ((unsigned) (ew * 32) << 16) + (unsigned) ((set * TB + tt) * op.cols + c0);
          tmem_ld<CB>(at, v);
          if constexpr (SEP) {    // the other accumulators, the one of the small products last
            const int nacc = min(op.sub, cur.i1 - cur.i0);
            for (int k = 1; k <= nacc; k++) {
              float w[CB];
              tmem_ld<CB>(at + (unsigned) ((k < nacc ? k : op.sub) * N), w);
#pragma unroll
              for (int q = 0; q < CB; q++) v[q] += w[q];
            }
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < CB / 4; q++)
            *reinterpret_cast<float4 *>(tr + lane * (CB + 4) + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          __syncwarp();
          if (!vec) {    // rows of a width that is no multiple of 4: value by value
            const int w = min(CB, row.n_out - c0);
            for (int e = lane; e < 32 * w; e += 32) {
              const int r = e / w, c = e - r * w, a = atom_of(tt, r);
              if (a < 0) continue;
              float *o = out + (size_t) a * dstT.C + c0 + c;
              const float x = tr[r * (CB + 4) + c];
              *o = add ? *o + x : x;
            }
            continue;
          }
          if (add) {
#pragma unroll
            for (int j = 0; j < 32 / RPI; j++) old[j] = oldn[j];
            load_old(b + 1, oldn);
          }
#pragma unroll
          for (int j = 0; j < 32 / RPI; j++) {
            const int r = j * RPI + lane / LPR, cq = lane % LPR, a = c0 + 4 * cq < row.n_out ? atom_of(tt, r) : -1;
            if (a >= 0) {
              float4 w = *reinterpret_cast<const float4 *>(tr + r * (CB + 4) + 4 * cq);
              if (add) {
                w.x += old[j].x; w.y += old[j].y; w.z += old[j].z; w.w += old[j].w;
              }
              reinterpret_cast<float4 *>(out + (size_t) a * dstT.C + c0)[cq] = w;
            }
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&s_accempty[set])) : "memory");
      rowc++;
      next_row(cur);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (t == 0 && s_abort) atomicExch(error, 1);
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
}

// activation stages, weight ring and the transpose buffers of the four epilogue warps
size_t smem_bytes(int K, int N, int S)
{
  const size_t cb = N % 32 == 0 ? 32 : 16;
  return (size_t) S * PARTS * (TM + N) * K * 2 + (size_t) 4 * 32 * (cb + 4) * 4;
}

int stages_for(int K, int N) { return smem_bytes(K, N, 4) <= 200 * 1024 ? 4 : 2; }

template<int K, int CB, int S, bool ELEM, bool SEP>
void launch_s(const MVTCDev &op, const TensorDev *T, int ntensors, int NA, int na, int TB, int tmem_cols, dim3 grid, int *error)
{
  const size_t smem = smem_bytes(K, op.N, S);
  static size_t attr = 0;
  if (smem > attr) {
    GB_CUDA(cudaFuncSetAttribute((mv_tc_kernel<K, CB, S, ELEM, SEP>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    attr = smem;
  }
  const char *name = ELEM ? "mv_tc_element_kernel" : "mv_tc_kernel";
  before_launch(name);
  mv_tc_kernel<K, CB, S, ELEM, SEP><<<grid, block_threads(K, ELEM), smem, dev().stream>>>(op, T, ntensors, NA, na, TB, tmem_cols, error);
  after_launch(name);
}

template<int K, bool ELEM> void launch_k(const MVTCDev &op, const TensorDev *T, int ntensors, int NA, int na, int TB, dim3 grid, int *error)
{
  int tmem_cols = 32;    // a power of two that holds two sets of accumulators of TB tiles
  while (tmem_cols < 2 * TB * op.cols) tmem_cols *= 2;
  const bool s4 = stages_for(K, op.N) == 4;
  if constexpr (ELEM) {
    if (s4 && op.sep) launch_s<K, 16, 4, true, true>(op, T, ntensors, NA, na, TB, tmem_cols, grid, error);
    else if (op.sep) launch_s<K, 16, 2, true, true>(op, T, ntensors, NA, na, TB, tmem_cols, grid, error);
    else launch_s<K, 16, 2, true, false>(op, T, ntensors, NA, na, TB, tmem_cols, grid, error);
  } else if (op.sep) {    // (16 columns at a time: 32 of both accumulators do not fit the registers)
    if (s4) launch_s<K, 16, 4, false, true>(op, T, ntensors, NA, na, TB, tmem_cols, grid, error);
    else launch_s<K, 16, 2, false, true>(op, T, ntensors, NA, na, TB, tmem_cols, grid, error);
  } else if (op.N % 32 == 0) {
    if (s4) launch_s<K, 32, 4, false, false>(op, T, ntensors, NA, na, TB, tmem_cols, grid, error);
    else launch_s<K, 32, 2, false, false>(op, T, ntensors, NA, na, TB, tmem_cols, grid, error);
  } else {
    if (s4) launch_s<K, 16, 4, false, false>(op, T, ntensors, NA, na, TB, tmem_cols, grid, error);
    else launch_s<K, 16, 2, false, false>(op, T, ntensors, NA, na, TB, tmem_cols, grid, error);
  }
}

template<bool ELEM> void launch_e(int K, const MVTCDev &op, const TensorDev *T, int ntensors, int NA, int na, int TB, dim3 grid, int *error)
{
  switch (K) {
    case 16: launch_k<16, ELEM>(op, T, ntensors, NA, na, TB, grid, error); break;
    case 32: launch_k<32, ELEM>(op, T, ntensors, NA, na, TB, grid, error); break;
    case 64: launch_k<64, ELEM>(op, T, ntensors, NA, na, TB, grid, error); break;
    default: throw DeviceError("tensor-core FC: unsupported input width");
  }
}

// operand images of the matrices of an operation: B[n][k] = W[k][n] in its bf16 parts, zero beyond the matrix;
// grid (matrices, elements)
__global__ void __launch_bounds__(256) mv_images_kernel(const float *__restrict__ W, const int4 *__restrict__ mats, long long ty_stride,
                                                        int K, int N, char *images, int nmat, int first)
{
  const int4 m = mats[blockIdx.x];    // offset, rows, row stride, columns
  const float *M = W + (long long) blockIdx.y * ty_stride + m.x;
  char *o = images + ((size_t) blockIdx.y * nmat + first + blockIdx.x) * PARTS * N * K * 2;
  for (int e = threadIdx.x; e < N * K; e += 256) {
    const int n = e / K, k = e - n * K;
    const float w = k < m.y && n < m.w ? M[(long long) k * m.z + n] : 0.0f;
    uint2 part[PARTS];
    split4(make_float4(w, 0.f, 0.f, 0.f), 1.0f, part);
    for (int p = 0; p < PARTS; p++) *reinterpret_cast<unsigned short *>(o + (size_t) p * N * K * 2 + tile_off(n, k, K)) = (unsigned short) part[p].x;
  }
}

// Atoms by element, every element padded to whole tiles.  order [tiles x 128]: atom or -1; tiles: their number, then the
// element of each.  One block, no barrier per atom: a warp owns a stretch of the atoms, counts its elements, and after a scan
// over the warps hands out its places in order (lanes that hold the same element take consecutive ones).
constexpr int ORDER_EL = 256;    // most elements
__global__ void __launch_bounds__(1024) elem_order_kernel(const int *__restrict__ mu, int na, int nel, int tiles_max, int *order, int *tiles)
{
  extern __shared__ int cnt[];    // [32 warps][nel]: counts, then the next place of the warp
  __shared__ int at[ORDER_EL + 1];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, seg = (na + 1023) / 1024 * 32;
  const int a_lo = warp * seg, a_hi = min(na, a_lo + seg);
  for (int q = t; q < 32 * nel; q += 1024) cnt[q] = 0;
  for (int q = t; q < tiles_max * TM; q += 1024) order[q] = -1;
  __syncthreads();
  for (int a = a_lo + lane; a < a_hi; a += 32) atomicAdd(&cnt[warp * nel + mu[a]], 1);
  __syncthreads();
  for (int e = t; e < nel; e += 1024) {
    int n = 0;
    for (int w = 0; w < 32; w++) {
      const int c = cnt[w * nel + e];
      cnt[w * nel + e] = n;
      n += c;
    }
    at[e] = (n + TM - 1) / TM;
  }
  __syncthreads();
  if (t == 0) {
    int tile = 0;
    for (int e = 0; e < nel; e++) {
      const int k = at[e];
      at[e] = tile;
      tile += k;
    }
    at[nel] = tile;
    tiles[0] = min(tile, tiles_max);
  }
  __syncthreads();
  for (int e = t; e < nel; e += 1024)
    for (int k = at[e]; k < min(at[e + 1], tiles_max); k++) tiles[1 + k] = e;
  for (int a0 = a_lo; a0 < a_hi; a0 += 32) {
    const int a = a0 + lane, e = a < a_hi ? mu[a] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int lead = __ffs(same) - 1;
    int base = 0;
    if (e >= 0 && lane == lead) {
      base = cnt[warp * nel + e];
      cnt[warp * nel + e] = base + __popc(same);
    }
    base = __shfl_sync(0xffffffffu, base, lead);
    const int place = e < 0 ? tiles_max * TM : at[e] * TM + base + __popc(same & ((1u << lane) - 1u));
    if (place < tiles_max * TM) order[place] = a;
    __syncwarp();
  }
}

// the same for many atoms: counts and places by blocks of 1024 atoms
__global__ void __launch_bounds__(1024) elem_count_kernel(const int *__restrict__ mu, int na, int nel, int *count)
{
  __shared__ int cnt[ORDER_EL];
  const int t = threadIdx.x, a = blockIdx.x * 1024 + t;
  for (int e = t; e < nel; e += 1024) cnt[e] = 0;
  __syncthreads();
  if (a < na) atomicAdd(&cnt[mu[a]], 1);
  __syncthreads();
  for (int e = t; e < nel; e += 1024)
    if (cnt[e]) atomicAdd(count + e, cnt[e]);
}
__global__ void __launch_bounds__(1024) elem_tiles_kernel(int *count, int nel, int tiles_max, int *tiles)
{
  __shared__ int at[ORDER_EL + 1];
  if (threadIdx.x == 0) {
    int tile = 0;
    for (int e = 0; e < nel; e++) {
      at[e] = tile;
      tile += (count[e] + TM - 1) / TM;
    }
    at[nel] = tile;
    tiles[0] = min(tile, tiles_max);
  }
  __syncthreads();
  for (int e = 0; e < nel; e++)
    for (int k = at[e] + threadIdx.x; k < min(at[e + 1], tiles_max); k += 1024) tiles[1 + k] = e;
  for (int e = threadIdx.x; e < nel; e += 1024) count[e] = at[e] * TM;    // where the next atom of the element goes
}
__global__ void __launch_bounds__(1024) elem_place_kernel(const int *__restrict__ mu, int na, int nel, int tiles_max, int *next, int *order)
{
  __shared__ int cnt[ORDER_EL], base[ORDER_EL];
  const int t = threadIdx.x, a = blockIdx.x * 1024 + t;
  for (int e = t; e < nel; e += 1024) cnt[e] = 0;
  __syncthreads();
  const int e = a < na ? mu[a] : 0;
  int rank = 0;
  if (a < na) rank = atomicAdd(&cnt[e], 1);
  __syncthreads();
  for (int q = t; q < nel; q += 1024)
    if (cnt[q]) base[q] = atomicAdd(next + q, cnt[q]);
  __syncthreads();
  if (a < na && base[e] + rank < tiles_max * TM) order[base[e] + rank] = a;
}

}    // namespace

void ElemOrder::make(const int *mu, int na, int nel, int kinds)
{
  if (nel > ORDER_EL) throw Unsupported("models with more than 256 elements are not supported");
  tiles_max = (na + TM - 1) / TM + std::min(kinds, na);
  order_.set_label("nlist:element_order");
  tiles_.set_label("nlist:element_order");
  order_.ensure((size_t) tiles_max * TM);
  tiles_.ensure((size_t) tiles_max + 1);
  if (na <= 8192) {    // one block of 10 us against four launches
    GB_LAUNCH(elem_order_kernel, 1, 1024, sizeof(int) * 32 * nel, mu, na, nel, tiles_max, order_.get(), tiles_.get());
    return;
  }
  next_.set_label("nlist:element_order");
  next_.ensure(ORDER_EL);
  GB_CUDA(cudaMemsetAsync(next_.get(), 0, sizeof(int) * ORDER_EL, dev().stream));
  GB_CUDA(cudaMemsetAsync(order_.get(), 0xff, sizeof(int) * (size_t) tiles_max * TM, dev().stream));
  const int nb = (na + 1023) / 1024;
  GB_LAUNCH(elem_count_kernel, nb, 1024, 0, mu, na, nel, next_.get());
  GB_LAUNCH(elem_tiles_kernel, 1, 1024, 0, next_.get(), nel, tiles_max, tiles_.get());
  GB_LAUNCH(elem_place_kernel, nb, 1024, 0, mu, na, nel, tiles_max, next_.get(), order_.get());
}

int MVTensorCore::padded_k(const MVOp &o)
{
  int k = 0;
  for (const MVItem &it : o.items) k = std::max(k, it.n_in);
  return k <= 16 ? 16 : k <= 32 ? 32 : k <= 64 ? 64 : 0;
}

bool MVTensorCore::eligible(const MVOp &o, const std::vector<TensorSpec> &tensors)
{
  if (o.items.empty() || o.row_out.empty()) return false;
  if ((int) tensors.size() > MAX_TENSORS || (int) o.items.size() > MAX_ITEMS || (int) o.row_out.size() > MAX_ROWS) return false;
  const int K = padded_k(o), N = padded_n(o.n_out);
  if (K == 0 || N > 256) return false;
  for (size_t r = 0; r + 1 < o.item_off.size(); r++)
    if (o.item_off[r + 1] == o.item_off[r]) return false;    // a row without items has no accumulator to write
  // beside the tables of an operation (17 KB of static shared memory)
  return smem_bytes(K, N, 2) <= 211 * 1024;
}

void MVTensorCore::setup(const std::vector<const MVOp *> &ops, const std::vector<const float *> &W, int n_elements)
{
  K_ = N_ = 0;
  elem_ = ops[0]->elem;
  odd_ = false;
  for (const MVOp *o : ops) {
    K_ = std::max(K_, padded_k(*o));
    N_ = std::max(N_, padded_n(o->n_out));
    odd_ = odd_ || o->n_out % 16 != 0;
    for (const MVItem &it : o->items) odd_ = odd_ || (it.n_in != 8 && it.n_in != 16 && it.n_in != 32 && it.n_in != 64);
  }
  // rows of all operations; a row that several of them write gets the items of all (the first decides whether it adds)
  std::map<std::pair<int, int>, int> index;
  std::vector<MVRowDev> rows;
  std::vector<std::vector<MVItem>> row_items;
  std::vector<std::vector<int4>> mats(ops.size());
  int first = 0;
  for (size_t q = 0; q < ops.size(); q++) {
    const MVOp &o = *ops[q];
    std::map<int, int> image;    // distinct matrices of the operation
    for (size_t r = 0; r < o.row_out.size(); r++) {
      auto key = std::make_pair(o.dst, o.row_out[r]);
      auto f = index.find(key);
      if (f == index.end()) {
        f = index.emplace(key, (int) rows.size()).first;
        rows.push_back(MVRowDev{(short) o.dst, (short) o.row_out[r], (short) (o.accumulate ? 1 : 0), (short) o.n_out, 0, 0});
        row_items.emplace_back();
      }
      for (int i = o.item_off[r]; i < o.item_off[r + 1]; i++) {
        MVItem it = o.items[i];
        auto g = image.find(it.mat);
        if (g == image.end()) {
          g = image.emplace(it.mat, first + (int) mats[q].size()).first;
          mats[q].push_back(make_int4(it.mat, it.n_in, o.ldw, o.n_out));
        }
        it.mat = g->second;    // image index instead of the offset in the fp32 weights
        row_items[f->second].push_back(it);
      }
    }
    first += (int) mats[q].size();
  }
  nmat_ = first;
  std::vector<MVItem> items;
  for (size_t r = 0; r < rows.size(); r++) {
    rows[r].i0 = (int) items.size();
    items.insert(items.end(), row_items[r].begin(), row_items[r].end());
    rows[r].i1 = (int) items.size();
  }
  nrows_ = (int) rows.size();
  long_ = false;
  for (const MVRowDev &r : rows) long_ = long_ || r.i1 - r.i0 > LONG_ROW;
  nitems_ = (int) items.size();
  images_.set_label("engine:weights_bf16");
  items_.set_label("engine:tables");
  rows_.set_label("engine:tables");
  const int ne = elem_ ? n_elements : 1;
  images_.ensure((size_t) ne * nmat_ * PARTS * N_ * K_ * 2);
  items_.upload(items);
  rows_.upload(rows);
  first = 0;
  DBuf<int4> d;
  for (size_t q = 0; q < ops.size(); q++) {
    d.upload(mats[q]);
    GB_LAUNCH(mv_images_kernel, dim3((unsigned) mats[q].size(), ne), 256, 0, W[q], d.get(), (long long) ops[q]->ty_stride, K_, N_,
              images_.get(), nmat_, first);
    first += (int) mats[q].size();
    GB_CUDA(cudaStreamSynchronize(dev().stream));
  }
  ready_ = true;
}

void MVTensorCore::launch(const TensorDev *tensors, int ntensors, int NA, int na, int *error, const ElemOrder *order) const
{
  if (!ready_) throw DeviceError("tensor-core FC used before its set-up");
  if (nrows_ == 0 || na == 0) return;
  MVTCDev op{};
  op.rows = rows_.get();
  op.items = items_.get();
  op.images = images_.get();
  op.N = N_;
  op.nrows = nrows_;
  op.nitems = nitems_;
  op.nmat = nmat_;
  int ntiles = (na + TM - 1) / TM;
  if (elem_) {
    if (!order) throw DeviceError("tensor-core FC: the order of the atoms by element is missing");
    op.order = order->order_.get();
    op.tiles = order->tiles_.get();
    ntiles = order->tiles_max;
  }
  // one CTA per SM; two sets of accumulators share the 512 tensor-memory columns
  const int G = dev().sm_count;
  // Separate accumulators: operations with per-element weights and widths other than 8, 16, 32 and 64 at any size and everything while
  // a CTA has at most one tile, where fp32 sums are the measure.  With more atoms the usual widths go without: a second read of the
  // epilogue and half as many tiles per CTA cost more (64 x 64, 1,024,000 atoms 27.8 -> 40.1 ms).
  // Rows of reduces over the element and of the UQ projection are sums of up to a hundred items; every item has an accumulator of its
  // own, as many at a time as there are columns for, and the epilogue adds them with rounding, part of a row after part.
  op.sep = 2 * N_ <= TMEM_COLS / 2 && (elem_ || odd_ || ntiles <= G);
  const int held = TMEM_COLS / 2 / N_ - (op.sep ? 1 : 0);
  op.sub = elem_ ? std::max(1, std::min(15, held)) : op.sep && ntiles <= G ? std::min(4, held) : 1;
  op.cols = (op.sub + (op.sep ? 1 : 0)) * N_;
  op.parts = elem_ || (op.sep && ntiles <= G && long_);
  const int tb_max = elem_ || ntiles <= G ? 1 : std::max(1, std::min(MAX_TILES, TMEM_COLS / 2 / op.cols));
  const int rounds = (ntiles + G * tb_max - 1) / (G * tb_max);
  const int TB = std::max(1, std::min(tb_max, (ntiles + G * rounds - 1) / (G * rounds)));
  const int gx = std::min(G, (ntiles + TB - 1) / TB);
  const int gy = std::max(1, std::min(nrows_, G / gx));
  if (elem_) launch_e<true>(K_, op, tensors, ntensors, NA, na, TB, dim3(gx, gy), error);
  else launch_e<false>(K_, op, tensors, ntensors, NA, na, TB, dim3(gx, gy), error);
}

}    // namespace gb
