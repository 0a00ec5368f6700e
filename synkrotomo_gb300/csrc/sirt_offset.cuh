// Byte offsets of the one-launch SIRT engine's detector gathers (sirt_small.cu),
// in plain integers so that a host test can evaluate them.
#pragma once

#ifndef SYNK_HD
#ifdef __CUDACC__
#define SYNK_HD __host__ __device__ __forceinline__
#else
#define SYNK_HD inline
#endif
#endif

namespace synk {

// The offsets are unsigned and count from the entry before the residual:
// candidate -1 of angle 0 lies there, and its neighbour, detector 0, is read at
// offset 4.  (Counted from the residual it would wrap to 4 GB - 4; signed
// offsets made N=128, 128 angles, 200 iterations 2.58 ms instead of 2.52.)  The
// problems the engine takes hold at most 1.3e8 entries a slice.
constexpr int kSmallLead = 1;

// Offset of angle k's row of D detectors, less the bits of the magic constant
// (floor_magic) and plus the middle detector zi that the coordinates count from.
SYNK_HD unsigned small_row_offset(int k, int D, int zi, int magic_bits) {
    return ((unsigned)k * (unsigned)D + (unsigned)zi + (unsigned)kSmallLead - (unsigned)magic_bits) * 4u;
}

// Offset of the first candidate detector, bits = the rounded coordinate's.
SYNK_HD unsigned small_gather_offset(unsigned bits, unsigned row) { return bits * 4u + row; }

}  // namespace synk
