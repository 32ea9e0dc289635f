// host_copy.cuh -- copies between the caller's (pageable) arrays and the
// device; results come back through page-locked chunks, with the host side's
// memcpy of large ones spread over threads.
#pragma once

#include "common.cuh"

namespace mdbas {

struct CopySpan {
  void *host;
  void *dev;
  size_t bytes;
  bool add;    // copy_out: doubles, added to the host array's
  bool joins;  // dev goes on where the previous span's array (one allocation) ends
  CopySpan(void *h = nullptr, void *d = nullptr, size_t b = 0, bool a = false, bool j = false)
      : host(h), dev(d), bytes(b), add(a), joins(j) {}
};

// Three arrays that follow one another on the device.
struct CopySpan3 {
  CopySpan s[3];
  CopySpan3(void *a, void *b, void *c, double *dev, size_t n, bool add = false)
      : s{CopySpan(a, dev, sizeof(double) * n, add),
          CopySpan(b, dev + n, sizeof(double) * n, add, true),
          CopySpan(c, dev + 2 * n, sizeof(double) * n, add, true)} {}
};

// Host arrays to the device on stream s, ordered there.  Pageable arrays have
// been read on return; page-locked ones are read by the copy engine and must
// stay as they are until the stream has got there (every call of the drop-in
// ends with a wait; of the engine's calls, those that return results do).
// (Both take at most 16 spans.)
int copy_in(const CopySpan *spans, int count, cudaStream_t s);
// Device arrays to the host: waits for the work already on s and returns with
// the data in the host arrays.  On an error their contents are undefined: work
// that failed before the copies is noticed before anything is written, but a
// device lost between two chunks leaves an array with `add` added to in part.
int copy_out(const CopySpan *spans, int count, cudaStream_t s);

// The page-locked chunks live while any user is registered (an engine, the
// drop-in and the standalone reciprocal sums once used); the last one to
// leave frees them.
void host_copy_enter();
void host_copy_leave();

}  // namespace mdbas
