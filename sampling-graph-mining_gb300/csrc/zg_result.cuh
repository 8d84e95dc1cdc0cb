// zg_result.cuh — pinned host memory for the reduced result of one synchronous run, written by the
// finalize kernel itself: the caller waits for the stream and reads it, without a device-to-host copy
// (a copy to pageable memory costs about 8 us, a third of the shortest run).
#pragma once

#include "zg_internal.cuh"

// One of a fixed number of slots (one allocation per process, made on first use), held from
// construction to destruction; p is null when all are taken or the allocation failed, and the caller
// copies from device memory then.  Safe from several threads; a slot belongs to one run at a time.
struct ZgResultSlot {
  ZgPartial* p;
  ZgResultSlot();
  ~ZgResultSlot();
  ZgResultSlot(const ZgResultSlot&) = delete;
  ZgResultSlot& operator=(const ZgResultSlot&) = delete;
};
