// uns_packed.hpp -- the padding rule of packed cases (uns_cc_create_packed),
// shared by the host code that lays them out and the kernels that read it.
#pragma once

#ifdef __CUDACC__
#define UNS_HOST_DEVICE __host__ __device__
#else
#define UNS_HOST_DEVICE
#endif

namespace uns {

// The interior cells of every case start at a multiple of kCasePad and are
// padded to the next one; a padding cell belongs to no case.
constexpr int kCasePad = 256;

UNS_HOST_DEVICE inline long long padded_cells(long long cells) { return (cells + kCasePad - 1) / kCasePad * kCasePad; }

// A real cell of the case that block `block` of `threads` threads (a power of
// two up to kCasePad, one thread per cell) works on: the first of its
// kCasePad cells.  The block's own first cell may be padding where it is
// narrower than that.
UNS_HOST_DEVICE inline int block_case_cell(int block, int threads) { return block * threads / kCasePad * kCasePad; }

}  // namespace uns
