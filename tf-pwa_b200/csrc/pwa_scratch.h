// Sizes of the scratch block of pwa_pieces_multi: counters (4 bytes each),
// arguments (bytes) and rows (doubles), side by side in one allocation.
//
// A service alternates between few large fits (many rows, few arguments) and
// many small ones (the reverse), so each part keeps the largest size that any
// batch has needed: the steady state allocates nothing.
#pragma once

#include <cstddef>

struct BatchScratch {
  long long counters = 0, rows = 0;
  size_t args = 0;

  size_t bytes() const {
    return sizeof(unsigned int) * (size_t)counters + args + sizeof(double) * (size_t)rows;
  }
  bool holds(long long n_count, size_t arg_bytes, long long n_rows) const {
    return n_count <= counters && arg_bytes <= args && n_rows <= rows;
  }
  // The sizes with which a batch fits: twice its need where it exceeds what
  // is there (counters in whole 256 bytes, so that the arguments stay
  // aligned), the others as they are.
  BatchScratch grown(long long n_count, size_t arg_bytes, long long n_rows) const {
    BatchScratch g = *this;
    if (n_count > counters) g.counters = (2 * n_count + 63) / 64 * 64;
    if (arg_bytes > args) g.args = 2 * ((arg_bytes + 255) / 256 * 256);
    if (n_rows > rows) g.rows = 2 * n_rows;
    return g;
  }
};
