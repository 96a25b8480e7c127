// Tensor-core form of the MV operations (FC layers, reduces, their adjoints) on chunk tensors in global memory: see
// mv_tc.cu.
#pragma once

#include "kernels.h"

#include <algorithm>

namespace gb {

struct MVRowDev {
  short dst, out;     // tensor and function the row goes to
  short accumulate, n_out;
  int i0, i1;         // its items
};

struct MVTCDev {
  const MVRowDev *rows;
  const MVItem *items;     // as MVDev::items with `mat` = index of the matrix's operand image
  const char *images;      // per element and matrix: the [N][K] images of its three bf16 parts (canonical K-major layout)
  const int *order, *tiles;    // per-element weights: ElemOrder
  int N, nrows, nitems, nmat;
  bool sep;                // an accumulator of its own for the small products
  bool parts;              // rows in parts of `sub` items, each with an accumulator of its own
  int sub;                 // accumulators of a1 b1 that the items of a row take in turn
  int cols;                // columns of a tile's accumulators
};

// The atoms of a chunk grouped by element, for operations with per-element weights: tiles of 128 atoms of one element.
class ElemOrder {
 public:
  // mu [na]: elements (device), below nel; kinds: most different elements among them
  void make(const int *mu, int na, int nel, int kinds);
  int tiles_max = 0;
  DBuf<int> order_;    // [tiles_max][128] atom, -1: none
  DBuf<int> tiles_;    // [0] tiles in use, then the element of each

 private:
  DBuf<int> next_;
};

class MVTensorCore {
 public:
  static constexpr int MAX_ITEMS = 512, MAX_ROWS = 256;    // tables of an operation staged in shared memory
  // shapes the kernel covers: up to 64 inputs per item, up to 256 outputs, every row with at least one item
  static bool eligible(const MVOp &o, const std::vector<TensorSpec> &tensors);
  // the widths the kernel runs an operation with
  static int padded_k(const MVOp &o);
  static int padded_n(int n_out) { return (n_out + 15) / 16 * 16; }
  // one launch for `ops` (same padded widths, all or none with per-element weights); W: their fp32 weights on the device
  void setup(const std::vector<const MVOp *> &ops, const std::vector<const float *> &W, int n_elements);
  bool ready() const { return ready_; }
  // tensors: device table of the chunk tensors; error: device flag set when a bounded wait ran out; order: the chunk's atoms
  // by element (operations with per-element weights)
  void launch(const TensorDev *tensors, int ntensors, int NA, int na, int *error, const ElemOrder *order) const;

 private:
  bool ready_ = false, elem_ = false, odd_ = false, long_ = false;    // odd_: a width other than 8, 16, 32, 64 (inputs), multiples of 16 (outputs); long_: LONG_ROW
  int K_ = 0, N_ = 0, nrows_ = 0, nitems_ = 0, nmat_ = 0;
  DBuf<char> images_;
  DBuf<MVItem> items_;
  DBuf<MVRowDev> rows_;
};

}    // namespace gb
