// Pixel-driven backprojection of a tile: bp_chunk_pair on rows of detector pairs
// (the standalone backprojector, SIRT of one large slice), bp_chunk on plain rows
// (the persistent and phase SIRT kernels, the backprojector without scratch).
//
// A block of 256 threads owns a tile of 32 columns; a thread owns one column and
// PIX rows spaced apart.  The per-angle constants of the chord-length trapezoid are
// staged in shared memory kBpChunk angles at a time and read as one broadcast
// float4 + one float2 per angle; each (pixel, angle) then costs 9-10 warp
// instructions with one 8-byte gather, or ~14 with two 4-byte ones:
//   q    = x_c*cos - y_c*sin - rz_c               (rho of the centre from the middle
//                                                  detector position rz_c, ProbGeom)
//   s0   = ceil((q - sqrt(2)/2) / deltarho) + zi  (first candidate detector)
//   d_i  = s0*deltarho + i*deltarho - q           (signed distance ray -> centre)
//   w_i  = sat((h - |d_i|) / b)                   (chord / lbase)
//   acc += lbase * sum_i w_i * sino[k][s0 + i]
// which is the reference's per-pixel sum (backprojection.fut:48-65) with
// intersect_fact*lbase (22-33, 62) written as the exact chord length of the
// line through the unit pixel.  Near-axis angles (AngleGeom::exact) are staged
// with zero weight and summed afterwards with the reference's own expressions.
#pragma once

#include "f32x2.cuh"
#include "synk_internal.cuh"

namespace synk {

// Angles per staged chunk (and per partial sum before the compensated
// total).  Fewer chunks mean fewer staging barriers; the whole angle set of a
// problem of up to 256 angles is one chunk.  SIRT at N=128 / 128 angles, 200
// iterations: 4.08 ms with 64, 3.96 with 128; N=256 / 180 angles: 8.73 ms with
// 128, 8.53 with 256; dense backprojection 4.09 / 4.07 / 4.05 ms with 64 /
// 128 / 256.
constexpr int kBpChunk = 256;

struct BpStage {
    float4 cs[kBpChunk];   // cos, sin, h/b, 1/b
    float2 le[kBpChunk];   // lbase, h/b - (1 - sqrt(2)/2)/b
};

// Stages angles [k0, k0 + kBpChunk) of P (all threads of the block call it).
__device__ __forceinline__ void bp_stage(const ProbGeom &P, int k0, BpStage &st) {
    for (int i = threadIdx.x; i < kBpChunk; i += blockDim.x) {
        const int k = k0 + i;
        float4 v = make_float4(0.0f, 0.0f, -1.0f, 0.0f);   // zero weight
        float2 l = make_float2(0.0f, -1.0f);
        if (k < P.a) {
            const AngleGeom g = load_geom(P.geom, k);
            if (!g.exact && isfinite(g.c)) {               // an angle without a direction weighs nothing
                v = make_float4(g.c, g.s, g.h_over_b, g.inv_b);
                l = make_float2(g.lbase, fmaf(-(1.0f - fact_f32()), g.inv_b, g.h_over_b));
            }
        }
        st.cs[i] = v;
        st.le[i] = l;
    }
}

// Accumulates angles k in [kc, kend) with (k - kc) % kstride == kphase of the
// staged chunk into acc[m] for the PIX pixels (row0 + m*ystep, col) whose
// centres are (xc, yc0 + m*ystep).  sino: the problem's sinogram [a][D].
//
// UNIT (deltarho = 1): with q = rho_c - rz_c - sqrt(2)/2, the first
// candidate detector is ceil(q) + zi and e = ceil(q) - q is in [0, 1); the two
// candidates sit at signed distances e - sqrt(2)/2 and e + 1 - sqrt(2)/2
// from the centre (the second is never negative), so
//   w0 = sat(h/b - |e - sqrt(2)/2| / b),  w1 = sat(c1 - e/b),  c1 = h/b - (1 - sqrt(2)/2)/b.
// INRANGE: the host proved that every window [s0, s0+1] lies in [0, D).
// SCALED: the sinogram rows of the staged (non-near-axis) angles are already
// multiplied by their lbase (row_scale), which saves one multiply per
// (pixel, angle); near-axis rows stay unscaled for bp_exact_angles.
// UNR = 2 walks the angles two at a time, so that their gathers are in flight
// together; the sums stay in angle order, bit for bit those of UNR = 1.
// Measured on GB300: SIRT at N=128 6.20 -> 5.88 ms (200 iterations; few warps
// there hide the gathers' latency), the dense backprojector at N=2048 4.88 ->
// 4.73 ms.
template <int PIX, bool UNIT, bool INRANGE, bool SCALED, int UNR = 1>
__device__ __forceinline__ void bp_chunk(const ProbGeom &P, const BpStage &st, int kc, int kend, int kphase,
                                         int kstride, const float *__restrict__ sino, float xc, float yc0,
                                         float ystep, float (&acc)[PIX]) {
    const float fact = fact_f32();
    const int D = P.D;
    const unsigned uD = (unsigned)D;
    const int nk = min(kBpChunk, kend - kc);
    const float zoff = -P.rz_c - fact;        // centred: |q| stays below ~N/sqrt(2) + 1
    // INRANGE gather base: row + zi - kMagicBits (the magic constant's bits folded in)
    const uintptr_t zoffb = (uintptr_t)(((intptr_t)P.zi - (intptr_t)kMagicBits) * 4);
    auto angle = [&](int i) {
        const float4 g = st.cs[i];
        const float2 le = st.le[i];
        const float *__restrict__ row = sino + (size_t)(kc + i) * D;
        if constexpr (UNIT) {
            // q of pixel m from the angle's base value in one rounding
            // (fma(m, dq, q0)), not by repeated additions: those drift by up
            // to PIX-1 roundings of |q| ~ D/2, which near-axis-adjacent
            // angles (trapezoid edges 1/b steep) turn into visible weight errors
            const float q0 = fmaf(xc, g.x, fmaf(-yc0, g.y, zoff));
            const float dq = -ystep * g.y;
            // INRANGE: the address comes straight from the bits of the rounded
            // sum r = q + 1.5*2^23 (bits(r) = bits(1.5*2^23) + s0), that constant
            // folded into the row base: one wide multiply-add per gather pair
            const uintptr_t rowb = reinterpret_cast<uintptr_t>(row) + zoffb;
#pragma unroll
            for (int m = 0; m < PIX; ++m) {
                const float q = m ? fmaf((float)m, dq, q0) : q0;
                float v0, v1, e;
                if constexpr (INRANGE) {
                    const float r = __fadd_ru(q, kMagic);
                    e = __fsub_rn(r, kMagic) - q;
                    const float *p = reinterpret_cast<const float *>(
                        rowb + (uintptr_t)(unsigned)__float_as_int(r) * 4u);
                    v0 = __ldg(p);
                    v1 = __ldg(p + 1);
                } else {
                    int s0;
                    e = ceil_magic(q, s0) - q;
                    s0 += P.zi;
                    v0 = ((unsigned)s0 < uD) ? __ldg(row + s0) : 0.0f;
                    v1 = ((unsigned)(s0 + 1) < uD) ? __ldg(row + s0 + 1) : 0.0f;
                }
                const float w0 = __saturatef(fmaf(-fabsf(e - fact), g.w, g.z));
                const float w1 = __saturatef(fmaf(-e, g.w, le.y));
                if constexpr (SCALED) acc[m] = fmaf(w1, v1, fmaf(w0, v0, acc[m]));
                else acc[m] = fmaf(le.x, fmaf(w1, v1, w0 * v0), acc[m]);
            }
        } else {
            const float t0 = fmaf(-yc0, g.y, -P.rz_c);
            const float tstep = -ystep * g.y;
#pragma unroll
            for (int m = 0; m < PIX; ++m) {
                const float t = m ? fmaf((float)m, tstep, t0) : t0;
                const float qc = fmaf(xc, g.x, t);             // rho_c - rz_c
                int s0;
                float s0f = ceil_magic((qc - fact) * P.inv_deltarho, s0);
                float d = s0f * P.deltarho - qc;
                float a = 0.0f;
                for (int q2 = 0; q2 < P.rpp; ++q2, d += P.deltarho) {
                    const int det = s0 + P.zi + q2;
                    const float w = __saturatef(fmaf(-fabsf(d), g.w, g.z));
                    if ((unsigned)det < uD) a = fmaf(w, __ldg(row + det), a);
                }
                acc[m] = SCALED ? acc[m] + a : fmaf(le.x, a, acc[m]);
            }
        }
    };
    int i = kphase;
    if constexpr (UNR >= 2)
        for (; i + kstride < nk; i += 2 * kstride) {
            angle(i);
            angle(i + kstride);
        }
    for (; i < nk; i += kstride) angle(i);
}

// The same sums on detector pairs: entry pad + s of row k (W entries a row) holds
// detectors (s, s+1), already times the row's factor and zero outside [0, D), so
// one 8-byte gather serves two candidates of a pixel and angle, and one packed
// multiply-add (acc_0, acc_1) += (w0, w1) * (v0, v1).  Angles kphase, kphase +
// 2^lgstride, ... of the chunk staged from kc on go into out[m] (overwritten).  Two
// pixels' coordinates, ceilings and distances are computed at a time with packed
// instructions (the halves round as the scalar ones), and a gather's address is a
// 32-bit offset in the chunk's rows (the caller keeps 256 rows below 4 GB): the
// 64-bit wide multiply-add it replaces holds the FMA pipe for four to five cycles.
// UNIT: deltarho = 1 (bp_chunk's weights); otherwise RPP candidates, at most four.
// CLAMP: first candidates may lie outside the row's entries; those outside
// [-pad, D] are moved to its ends, which are zero (PairRows).
// Two angles at a time with 80 registers (3 blocks per SM), N=2048, 2048 angles:
// 4.05 -> 3.44 ms (one at a time 4.25; 64 registers 3.75; three with 128 registers
// 3.62; the tile's segments staged in shared memory 3.88).
template <int PIX, int RPP = 2, bool UNIT = true, bool CLAMP = false>
__device__ __forceinline__ void bp_chunk_pair(const ProbGeom &P, const BpStage &st, int kc,
                                              const float2 *__restrict__ pairs, int W, int pad, int kphase,
                                              int lgstride, float xc, float yc0, float ystep, float (&out)[PIX]) {
    static_assert(PIX % 2 == 0, "pixels go in pairs");
    static_assert(!UNIT || RPP == 2, "two candidates at deltarho = 1");
    const float fact = fact_f32();
    const f32x2 mg2 = pk2(kMagic, kMagic), nmg2 = pk2(-kMagic, -kMagic), m1 = pk2(-1.0f, -1.0f);
    const f32x2 nf2 = pk2(-fact, -fact);
    // not UNIT: coordinates are kept negated (-q), so that s0*deltarho - q is one multiply-add
    const f32x2 f2 = pk2(fact, fact), ninv2 = pk2(-P.inv_deltarho, -P.inv_deltarho), dr2 = pk2(P.deltarho, P.deltarho);
    const char *base = reinterpret_cast<const char *>(pairs + (size_t)kc * W);
    const unsigned step = ((unsigned)W * 8u) << lgstride;
    // gather offset in the chunk = bits(r)*8 + rowoff (mod 2^32), bits(r) = kMagicBits + s0 - zi
    unsigned rowoff = ((unsigned)(P.zi + pad) - (unsigned)kMagicBits) * 8u + (unsigned)W * 8u * (unsigned)kphase;
    // limits of r: the zero entries, or 2^21, which no pixel's window reaches
    const float rlo = kMagic + (float)max(-pad - P.zi, -(1 << 21));
    const float rhi = kMagic + (float)min(P.D - P.zi, 1 << 21);
    const int nk = (min(kBpChunk, P.a - kc) - kphase + (1 << lgstride) - 1) >> lgstride;   // this part's angles
    f32x2 acc[PIX];
#pragma unroll
    for (int m = 0; m < PIX; ++m) acc[m] = pk2(0.0f, 0.0f);
#pragma unroll 2
    for (int j = 0; j < nk; ++j) {
        const int i = (j << lgstride) + kphase;
        const float4 g = st.cs[i];
        auto entry = [&](float r) {
            if constexpr (CLAMP) r = fminf(fmaxf(r, rlo), rhi);
            return base + ((unsigned)__float_as_int(r) * 8u + rowoff);
        };
        if constexpr (UNIT) {
            const float c1 = st.le[i].y;
            // q of pixel m from the angle's base value in one rounding (see bp_chunk)
            const float q0 = fmaf(xc, g.x, fmaf(-yc0, g.y, -P.rz_c - fact));
            const float dq = -ystep * g.y;
            const f32x2 q02 = pk2(q0, q0), dq2 = pk2(dq, dq);
            float2 v[PIX], w[PIX];
#pragma unroll
            for (int h = 0; h < PIX / 2; ++h) {
                const f32x2 q = fma2(pk2((float)(2 * h), (float)(2 * h + 1)), dq2, q02);
                const f32x2 r = add2_ru(q, mg2);
                const f32x2 e = fma2(q, m1, add2(r, nmg2));            // ceil(q) - q
                const float2 ev = unpk2(e), dv = unpk2(add2(e, nf2)), rv = unpk2(r);
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    v[2 * h + o] = __ldg(reinterpret_cast<const float2 *>(entry(o ? rv.y : rv.x)));
                    w[2 * h + o].x = __saturatef(fmaf(-fabsf(o ? dv.y : dv.x), g.w, g.z));
                    w[2 * h + o].y = __saturatef(fmaf(-(o ? ev.y : ev.x), g.w, c1));
                }
            }
#pragma unroll
            for (int m = 0; m < PIX; ++m) acc[m] = fma2(pk2(w[m]), pk2(v[m]), acc[m]);
        } else {
            const float nt0 = fmaf(yc0, g.y, P.rz_c), dt = ystep * g.y;   // -(rho - rz_c) = -x*cos + y*sin + rz_c
            const f32x2 nc2 = pk2(-g.x, -g.x), xc2 = pk2(xc, xc), nt02 = pk2(nt0, nt0), dt2 = pk2(dt, dt);
#pragma unroll
            for (int h = 0; h < PIX / 2; ++h) {
                const f32x2 t = fma2(pk2((float)(2 * h), (float)(2 * h + 1)), dt2, nt02);
                const f32x2 nq = fma2(xc2, nc2, t);
                const f32x2 r = add2_ru(mul2(add2(nq, f2), ninv2), mg2);
                const float2 rv = unpk2(r);
                const char *p[2] = {entry(rv.x), entry(rv.y)};
                f32x2 d = fma2(add2(r, nmg2), dr2, nq);                  // distance of the first candidate
#pragma unroll
                for (int c = 0; c < RPP; c += 2) {
                    const float2 d0 = unpk2(d);
                    d = add2(d, dr2);
                    const float2 d1 = unpk2(d);
                    d = add2(d, dr2);
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        const float w0 = __saturatef(fmaf(-fabsf(o ? d0.y : d0.x), g.w, g.z));
                        if (c + 1 < RPP) {
                            const float w1 = __saturatef(fmaf(-fabsf(o ? d1.y : d1.x), g.w, g.z));
                            const float2 v = __ldg(reinterpret_cast<const float2 *>(p[o] + c * 8));
                            acc[2 * h + o] = fma2(pk2(w0, w1), pk2(v), acc[2 * h + o]);
                        } else {
                            const float v = __ldg(reinterpret_cast<const float *>(p[o] + c * 8));
                            float2 a = unpk2(acc[2 * h + o]);
                            a.x = fmaf(w0, v, a.x);
                            acc[2 * h + o] = pk2(a);
                        }
                    }
                }
            }
        }
        rowoff += step;
    }
#pragma unroll
    for (int m = 0; m < PIX; ++m) {
        const float2 t = unpk2(acc[m]);
        out[m] = t.x + t.y;
    }
}

// Factor of sinogram row k in a SCALED backprojection: lbase, or 1 for a
// near-axis angle (summed from the unscaled row by bp_exact_angles).
__device__ __forceinline__ float row_scale(const AngleGeom *__restrict__ geom, int k) {
    return __ldg(&geom[k].exact) ? 1.0f : __ldg(&geom[k].lbase);
}

// True when every pixel's two candidate detectors of the UNIT path lie in
// [0, D) (deltarho = 1 and a detector row covering the image's circumcircle,
// as the reference's D >= ceil(N*sqrt(2)) with centred rhozero does).  The
// tiles cover columns [0, 32*ceil(N/32)) and rows [0, tile_rows*ceil(N/tile_rows))
// (pixels past N are computed, not stored), so the bound takes the padded
// extent, and it keeps a margin for the float rounding of q.  A launch whose
// tile height divides tile_rows never reaches further.
inline bool bp_windows_in_range(const ProbGeom &P, int tile_rows) {
    if (P.deltarho != 1.0f) return false;
    const int ext_x = (P.N + 31) / 32 * 32;
    const int ext_y = (P.N + tile_rows - 1) / tile_rows * tile_rows;
    const int ext = ext_x > ext_y ? ext_x : ext_y;
    const double m = fmax(P.half - 0.5, ext - 0.5 - P.half);       // max |x_c|, |y_c| of a tile pixel
    const double R = m * 1.4142135623730951;                         // max |rho_c|
    const double f = 0.70710677;
    const double rz = (double)P.rhozero;
    const double margin = 1e-2 + 1e-5 * (R + fabs(rz));
    const double lo = -R - f - rz, hi = R - f - rz;
    return ceil(lo - margin) >= 0.0 && ceil(hi + margin) + 1.0 <= (double)P.D - 1.0;
}

// Rows of bp_chunk_pair: `pad` zero entries before detector 0, W = D + 2*pad - 1
// entries.  A first candidate s has its entries when -pad <= s <= D + pad - 2 (two
// less with a second pair).
struct PairRows {
    int pad, W;
    bool inrange;    // every tile pixel's first candidate has its entries: no CLAMP
};

// The pixels of a tile past the image's edge reach up to 63*sqrt(2) further than
// the image, so the rows are padded as far as they need (at most kBpMaxPad,
// else CLAMP, which costs a minimum and a maximum per gather: N=2046, 1999 angles
// 4.28 ms with it, 3.37 without).
constexpr int kBpMaxPad = 128;
inline PairRows bp_pair_rows(const ProbGeom &P, int tile_rows) {
    const int ext_x = (P.N + 31) / 32 * 32;
    const int ext_y = (P.N + tile_rows - 1) / tile_rows * tile_rows;
    const int ext = ext_x > ext_y ? ext_x : ext_y;
    const double R = fmax(P.half - 0.5, ext - 0.5 - P.half) * 1.4142135623730951;   // max |rho_c| of a tile pixel
    const double f = 0.70710677, rz = (double)P.rhozero, dr = (double)P.deltarho;
    const double margin = 1e-2 + 1e-5 * (R + fabs(rz)) / dr;
    const double lo = ceil((-R - f - rz) / dr - margin), hi = ceil((R - f - rz) / dr + margin);
    const int base = P.rpp > 2 ? 4 : 2;
    const double need = fmax((double)base, fmax(-lo, hi - P.D + (double)base));
    PairRows r;
    r.inrange = need <= (double)kBpMaxPad;
    r.pad = r.inrange ? (int)need : base;
    r.W = P.D + 2 * r.pad - 1;
    return r;
}

// The near-axis angles of list[0..nexact) for the PIX pixels, the reference's
// own expressions (bp_angle's exact branch).
template <int PIX>
__device__ __forceinline__ void bp_exact_angles(const ProbGeom &P, const int *__restrict__ list, int nexact,
                                                int kphase, int kstride, const float *__restrict__ sino, int row0,
                                                int rstep, int col, float (&acc)[PIX]) {
    for (int e = kphase; e < nexact; e += kstride) {
        const int k = __ldg(list + e);
        const AngleGeom g = load_geom(P.geom, k);
#pragma unroll
        for (int m = 0; m < PIX; ++m) {
            const int row = row0 + m * rstep;
            if (row < P.N && col < P.N) acc[m] += bp_angle<false>(P, g, sino + (size_t)k * P.D, row, col);
        }
    }
}

}  // namespace synk
