// Host side of the runtime-radix pass kernel (rx_kernel.cuh): stage radices,
// tile geometry, the twiddle table's layout and the launch.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "pb_internal.hpp"

namespace pb {

constexpr int kRxMaxStages = 12;
constexpr int kRxMaxThreads = 512;
constexpr int kRxMaxPieces = 64;
// largest radix with a butterfly in registers; larger primes take the
// direct-sum stage
constexpr int kRxRegRadix = 23;

// Tile geometry of one pass, a function of its PassArgs (rx_geometry).  Shared
// memory: two row buffers (row i of a buffer is element i of every sequence:
// G vectors of W sequences), the twiddle table, the staged input lines of the
// tile, tile descriptors and piece rows.
struct RxGeom {
  int len;       // FFT length of the stages: m, or the convolution length of a Bluestein pass
  int lgG;       // log2 of the vectors per row
  int P;         // row pitch in vectors
  int threads;
  int bufv;      // vectors per row buffer
  int pre;       // 1: a pass over the staged lines forms the FFT input rows first
  int tw_smem;   // twiddle vectors held in shared memory (0: read from global memory)
  int alias;     // 1: the staging area is the second row buffer (no prefetch overlap)
  int ip;        // 1: stages in place in one row buffer, lines read straight into registers
  int pad;       // rows written by a stage are padded by one after every `pad` (0: none)
  int sl, sq;    // staging strides of a line and of an element, in elements
  int off_tw, off_stage, off_desc;  // byte offsets in shared memory
  int smem;      // bytes
  int max_smem;  // the device's limit
  int twoff[kRxMaxStages];
};

struct RxArgs {
  PassArgs p;
  RxGeom g;
};

// Stage radices of an m-point transform (stage 0 first); empty when m has a
// prime factor above 31.
std::vector<int> rx_radices(int m);

// The per-stage twiddle table of a radix list: for stage s the (R-1)*NS
// entries W^{k r} of a (NS*R)-point transform, then for a prime radix above
// kRxRegRadix its R roots.  Each entry is a vector (c, c, s, s) in f32 and
// (c, s) in f64, taken from `roots`, the m-th roots (m the radices' product).
template <typename R>
std::vector<R> rx_twiddles(const std::vector<int>& radix, const R* roots);

// Geometry for tiles of A.lines lines; false when they do not fit in
// max_smem bytes of shared memory.
bool rx_geometry(const PassArgs& A, int real_bytes, int max_smem, RxGeom* g);

// Sets A.lines, radices and geometry-independent fields for a pass whose
// layout conditions hold; false when the length is not served.  max_chunk is
// the longest run of lines along the tile axis, total_lines the lines of the
// whole pass, sms the device's multiprocessors.
bool rx_choose(PassArgs& A, int real_bytes, int max_smem, long long max_chunk, long long total_lines, int sms);

cudaError_t launch_rx(const PassArgs& A, int real_bytes, cudaStream_t stream);
int rx_occupancy(const PassArgs& A, int real_bytes);

}  // namespace pb
