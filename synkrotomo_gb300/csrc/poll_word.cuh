// What the stopping rule's host check reads back, in plain integers so that a host
// test can evaluate it.
#pragma once

#ifndef SYNK_HD
#ifdef __CUDACC__
#define SYNK_HD __host__ __device__ __forceinline__
#else
#define SYNK_HD inline
#endif
#endif

namespace synk {

// Low half: the number of the call; high half: its slices still updating.  The pinned
// words belong to the context, and the copies of a call on another stream may still
// arrive: only a word of this call says that this call is done.
SYNK_HD bool poll_done(unsigned long long word, int call) { return word == (unsigned long long)(unsigned)call; }

}  // namespace synk
