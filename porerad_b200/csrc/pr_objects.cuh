// Device-resident objects behind the opaque handles of porerad.h.
#pragma once
#include <memory>
#include <vector>

#include "pr_internal.cuh"

namespace pr {

// Switches to the object's device for the duration of a call.
struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

// Sorted CSR of integer first-hit counts: row = origin patch, col = receiver patch.
struct CountCsr {
  int64_t n_rows = 0, nnz = 0;
  DevBuf<int64_t> row_ptr;  // n_rows + 1
  DevBuf<int32_t> col;      // nnz, ascending within a row
  DevBuf<int32_t> cnt;      // nnz, > 0
};

// Symmetric exchange matrix S' = 0.5 (A F + F^T A) without the support diagonal
// (delta A, applied separately).  Entry storage, by mode:
//   kStream:  value factor * n, n = n_ij + n_ji on the union of the patterns of F and F^T (every patch
//             with the same area and ray count), as the word stream of SymStream;
//   kCounts:  col (int32) + n (int32) on the same union, columns ascending (where most counts are above
//             what a word holds, and for many patches with few entries per row);
//   kValues:  col (int32) + binary64 value 0.5 A n / R of the entry's origin patch; row i
//             holds row i of F followed by row i of F^T (two ascending runs).
enum SymMode { kStream = 0, kCounts = 1, kValues = 2 };

// A kStream matrix in the order its products read it.  Columns fall into `groups` groups of nb blocks
// of W <= 2^14 columns, so that the blocks of x in use fit in shared memory.  CTA c owns the rows
// [cta_row[c], cta_row[c + 1]) of one group, at most rows_cap of them, where row i of group g counts
// as g n + i; with more than one group a product leaves a sum per row and group, which a second kernel
// adds.  The entries of a CTA's rows in one column block (a stage), row after row and within a row in
// the order k_stream_fill gives them, are packed into quads of four 32-bit words, every row starting a new quad and
// having at least one, and dealt to the CTA's kStreamThreads lanes in runs of q quads, a multiple of
// `unroll`; quad t of lane l is quad base + t kStreamThreads + l, and a CTA's stages follow one
// another.  Words: stream_place(column within the block) << 18 | row start << 17 (first word of a
// row's first quad) | n.  The rest of a row's last quad and of the last lanes' runs have n = 0 and
// place W, which holds 0 in every block (so that no value of x meets a row without it).  start[l] is
// the number of rows begun before lane l's run, minus one.
constexpr int kStreamThreads = 1024;
constexpr int kStreamColBits = 14;
constexpr uint32_t kStreamRow = 1u << 17, kStreamCount = kStreamRow - 1u;
// Where a block's column lies in shared memory: its low four bits (the bank pair of an 8-byte value)
// are mixed with the higher ones, so that columns at a fixed stride, such as the patches of a flat
// sheet, do not share a few banks (a 160^3 layer operator: 247 instead of 410 us; mixing pairs of
// columns only, which halves the copies of x, took 280 us there and won 2 % on foam).
__host__ __device__ __forceinline__ uint32_t stream_place(uint32_t col) {
  return col ^ (((col >> 4) ^ (col >> 8) ^ (col >> 12)) & 15u);
}
struct SymStream {
  int W = 0, nb = 0, groups = 1, ctas = 0, rows_cap = 0, unroll = 1;
  DevBuf<uint4> quads;      // and unroll x kStreamThreads more, read ahead but not used
  DevBuf<int64_t> cta_row;  // ctas + 1
  DevBuf<int64_t> base;     // ctas x nb + 1: first quad of a stage
  DevBuf<int32_t> q;        // ctas x nb
  DevBuf<int16_t> start;    // ctas x nb x kStreamThreads
};

struct SymCsr {
  int64_t n_rows = 0, nnz = 0;
  DevBuf<int64_t> row_ptr;
  DevBuf<uint32_t> cols;   // the column of every entry (kCounts, kValues)
  DevBuf<int32_t> cnt;     // kCounts
  DevBuf<double> val;      // kValues
  int mode = kStream;
  double factor = 0.0;     // 0.5 A / R in the uniform modes
  SymStream stream;        // kStream
};

// Padded occupancy of a box for the traversal: kPadX layers of solid cells beyond each x wall, and
// kHalo periodic copies on each side of y and z; bit c = cell ((i + kPadX) (ny + 2 kHalo) + j +
// kHalo) (nz + 2 kHalo) + k + kHalo.
constexpr int kPadX = 8, kHalo = 16;

// Division of n < 2^31 by a constant: n / by = (n mul >> 32) >> shift, mul = ceil(2^(31 + s) / by)
// with s = ceil(log2 by) and shift = s - 1 (mul by - 2^(31 + s) < by <= 2^s, so the error stays
// below 1 / by).
struct PadDiv {
  uint32_t mul = 0;
  int32_t shift = 0, by = 1;
  void set(int64_t d) {  // 2 <= d < 2^31
    int s = 1;
    while (((int64_t)1 << s) < d) ++s;
    mul = (uint32_t)((((uint64_t)1 << (31 + s)) + (uint64_t)d - 1) / (uint64_t)d);
    shift = s - 1;
    by = (int32_t)d;
  }
};

// A box and the divisions by its padded plane (cells of one x) and row (cells of one x, y).
struct BoxMap {
  int32_t nx = 0, ny = 0, nz = 0, padded = 0;
  PadDiv plane, row;
};

}  // namespace pr

struct pr_case {
  int device = 0;
  int64_t nx = 0, ny = 0, nz = 0, n_cells = 0;
  int64_t n_patches = 0, n_wall = 0;
  double H = 0.0, area = 0.0;
  pr::DevBuf<uint8_t> solid;      // n_cells, 0/1
  pr::DevBuf<uint32_t> occ;       // bit-packed solid flags, bit c = cell c (flat)
  pr::DevBuf<uint32_t> pad;       // padded occupancy (kPadX, kHalo), or empty
  pr::BoxMap box;
  pr::DevBuf<int8_t> cls;         // patch class 0 hot, 1 cold, 2 internal
  pr::DevBuf<int8_t> face;        // patch face 0..5, -1 for walls
  pr::DevBuf<int8_t> code;        // emission normal: 0..5 as +x,-x,+y,-y,+z,-z
  pr::DevBuf<int32_t> cell;       // owning cell, -1 for walls
  pr::DevBuf<double> origin;      // (P, 3)
  // Face table: cell_face_patch (n_cells, 6), then the hot and the cold wall patch of each
  // (j, k) lattice site.  A first hit is recorded as an index into this table (its hit code).
  pr::DevBuf<int32_t> ftab;
  cudaStream_t last_stream = nullptr;
  int32_t* cfp() const { return ftab.ptr; }
  int32_t* hot() const { return ftab.ptr + 6 * n_cells; }
  int32_t* cold() const { return ftab.ptr + 6 * n_cells + ny * nz; }
  void rebind(cudaStream_t s) {
    solid.stream = occ.stream = pad.stream = s;
    cls.stream = face.stream = code.stream = s;
    cell.stream = origin.stream = ftab.stream = s;
  }
  size_t device_bytes() const {
    return solid.bytes() + occ.bytes() + pad.bytes() + cls.bytes() + face.bytes() + code.bytes() + cell.bytes() +
           origin.bytes() + ftab.bytes();
  }
};

struct pr_counts {
  int device = 0;
  std::shared_ptr<pr::CountCsr> csr;
  pr::DevBuf<int64_t> rays;  // rays per origin
  int64_t rays_traced = 0, dda_steps = 0;
  cudaStream_t last_stream = nullptr;
};

struct pr_operator {
  int device = 0;
  int64_t n = 0;
  std::shared_ptr<pr::CountCsr> F;
  pr::DevBuf<int64_t> rays;   // R_i
  pr::DevBuf<double> area;    // A_i
  pr::SymCsr S;
  pr::DevBuf<double> scale;   // d
  double delta = 0.0;
  int method = 0, iterations = 0;
  double row_sum_error = 0.0;
  mutable int64_t spmv_calls = 0;
  // transposed count CSR (kept from the assembly for raw_rmatvec)
  mutable std::shared_ptr<pr::CountCsr> FT;
  mutable cudaStream_t last_stream = nullptr;
};

// Cell-centred finite-volume conduction on an x-oriented grid (porerad/conduction.py): the
// conductance of each cell's +x, +y and +z face (harmonic mean times dx, 0 on the +x face of
// the last layer; y and z periodic), the diagonal of A, and the wall responses.
struct pr_conduction {
  int device = 0;
  int64_t nx = 0, ny = 0, nz = 0, n = 0;
  double H = 0.0, dx = 0.0;
  pr::DevBuf<double> k, gx, gy, gz, diag, hot, cold;
  cudaStream_t last_stream = nullptr;
};
