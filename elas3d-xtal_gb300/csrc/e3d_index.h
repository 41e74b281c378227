// Where a node's values lie, for kernels that carry node numbers in 32 bits (2^32
// nodes of a solve would take 700 GB and more).  Byte offsets into a component and
// indices into a vector of three components take 64: a batched or served solve needs
// 179 bytes a node, so that one of 1100^3 = 1.33e9 nodes has room on the device.  They
// cost nothing: ten RVEs of 32^3 to 88^3 581 ms, 590 with offsets of 32 bits; one of
// 64^3 60.1 and 59.9; 50 iterations at 500^3 321.3 and 320.9.
#pragma once

#ifdef __CUDACC__
#define E3D_HD __host__ __device__ __forceinline__
#else
#define E3D_HD inline
#endif

namespace e3d {

// Node of column `col` (x + nx y) in plane z of nxy nodes.
E3D_HD unsigned node_of(unsigned col, unsigned nxy, int z) { return col + nxy * (unsigned)z; }

// Byte offset of node m in a component of 4-byte values.
E3D_HD unsigned long long node_bytes4(unsigned long long m) { return 4ull * m; }

// Index of component c of node m in a vector of components of ns values.
E3D_HD unsigned long long value_of(unsigned m, int c, long long ns) {
  return m + (unsigned long long)c * (unsigned long long)ns;
}

}  // namespace e3d
