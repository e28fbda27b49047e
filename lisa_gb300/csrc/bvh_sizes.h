// Sizes of a BVH build: what a node and a leaf triangle take, how many there
// can be, and the bytes of all arrays, so that a fixed scratch can be checked
// against them when the library is compiled.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace lisa {

constexpr int NODE_BYTES = 96;
constexpr int TRI_BYTES = 64;

// What a build leaves on the device, for the host and for kernels that
// follow it on the stream.
struct BvhDeviceInfo {
  uint32_t nodes;      // 8-wide nodes
  uint32_t tris;       // leaf triangles written
  uint32_t depth;
  uint32_t failed;     // a bounded wait ran out
  int bounds[12];      // scene min, max and centroid min, max, as order-preserving ints
  uint32_t level[3];   // nodes taken by the collapse's current level (in turn)
  uint32_t barrier;    // arrivals of the collapse's blocks
  uint32_t ticket[4];  // tiles started, per sort pass
  uint64_t begin_ns, end_ns;  // the GPU's clock in the first kernel and at the end of the last
};

constexpr int RS_THREADS = 256;
constexpr int RS_PASSES = 4;  // 8 bits each (BvhDeviceInfo has a ticket per pass)

// Keys per thread of a sort tile: 16, but 4 for up to 256 Ki keys, which would
// otherwise make too few tiles (8 of them at 30,000) to fill the GPU.
constexpr int rs_rounds(uint32_t n) { return n <= (1u << 18) ? 4 : 16; }
constexpr uint32_t sort_tiles(uint32_t n) {
  return (uint32_t)((n + (uint64_t)RS_THREADS * rs_rounds(n) - 1) / ((uint64_t)RS_THREADS * rs_rounds(n)));
}

// Words of the tables that a build counts up in: look-back states and digit
// histograms of the sort, arrival flags of the bottom-up pass.
constexpr uint64_t counted_words(uint32_t n) { return (uint64_t)RS_PASSES * 256 * (sort_tiles(n) + 1) + n; }

// Most 8-wide nodes that n triangles can give.  A node with an internal
// child has eight children (the collapse opens candidates until there are
// eight or none is left to open, whatever was planned), the others (T, below F such nodes) hold at
// least four triangles; the F nodes' own leaves number 8 F - (F + T - 1), so
// n >= 4 T + 7 F - T + 1 >= 3 (F + T) + 1.
constexpr uint32_t max_nodes(uint32_t n) { return n / 3 + 1; }

// Bytes as scratch sources hand them out (256-byte pieces).
constexpr uint64_t al256(uint64_t b) { return ((b < 16 ? 16 : b) + 255) & ~255ull; }

// Device bytes that a build without a plan takes for its temporaries, and that
// any build takes for its nodes and leaf triangles, from n triangles.
constexpr uint64_t bvh_temp_bytes(uint32_t n) {
  return 4 * al256(16ull * n)              // boxes: plo phi ilo ihi
         + 4 * al256(4ull * n)             // keys vals keys2 vals2
         + 6 * al256(4ull * n)             // tree links, counts and costs
         + al256(4ull * counted_words(n))  //
         + al256(4ull * max_nodes(n))      // collapse work list
         + al256(sizeof(BvhDeviceInfo));
}
constexpr uint64_t bvh_output_bytes(uint32_t n) {
  return al256((uint64_t)NODE_BYTES * max_nodes(n)) + al256((uint64_t)TRI_BYTES * n);
}

}  // namespace lisa
