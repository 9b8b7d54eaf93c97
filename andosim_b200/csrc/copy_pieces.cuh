// copy_pieces.cuh -- how an array of 4-byte elements is cut into the aligned
// 16-byte pieces of an asynchronous copy. Plain arithmetic, so that a host
// compiler can check it: nothing outside the array is read.
#pragma once

#ifdef __CUDACC__
#define ANDO_HD __host__ __device__
#else
#define ANDO_HD
#endif

namespace ando {

// An array of n elements that starts `off` elements (0 to 3) past a 16-byte
// boundary: the pieces [q0, q1), counted from that boundary on, are the array's as
// a whole; the `head` elements before them and the `tail` after share theirs with
// whatever lies beside the array and are copied one by one.
struct CopyPieces { int head, q0, q1, tail; };
ANDO_HD inline CopyPieces copy_pieces(int off, int n) {
  const int to_boundary = (4 - off) & 3, head = n < to_boundary ? n : to_boundary;
  const int q0 = off > 0 ? 1 : 0, end = (off + n) >> 2;
  return CopyPieces{head, q0, end > q0 ? end : q0, n > head ? (off + n) & 3 : 0};
}

}  // namespace ando
