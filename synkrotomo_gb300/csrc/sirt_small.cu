// SIRT of one small problem (futhark/SIRT.fut:27-39) in one cooperative launch:
// one block of 32 warps per SM, two grid barriers per iteration.
//
// At these sizes an iteration's arithmetic is a microsecond or two, and what
// bounds it is the chain of latencies between its phases.  So every warp owns the same
// forward and backward items in all iterations: their decoding, geometry, row
// ranges, normaliser entries and measured values are loaded once, before the
// loop, and stay in registers (problems with more items than warps decode them again),
// the angle constants stay in shared memory, and a phase is then: one
// burst of independent gathers, a reduction through shared memory, one store,
// a barrier that costs an arrival without a reply and a poll.  N=128, 128 angles,
// 200 iterations: 3.49 ms with two chained launches per iteration, 2.56 here: 7000
// of an iteration's 27000 cycles are the forward walk (four bursts), 7000 the
// backward one, the rest the two barriers (at least 3500 each) and the reductions.
//
// Items.  Forward: a unit = (slice, 32 detectors, angle), S warps with a row part
// each; then one warp per near-axis ray and per listed corner ray.  Backward: a
// unit = (slice, 32 columns, image row), SB warps with an angle part each.  A block
// takes neighbouring units, so that what its warps read overlaps: chunks of
// consecutive angles' bands of the image, consecutive rows' detector windows.
// The forward chunks are dealt round with the detector groups varying fastest,
// because rays near the edge of the detector row are short: with one run of units per
// block the longest blocks took four times the shortest (N=256, 180 angles).
//
// Other blocks' stores are read after a barrier whose acquire invalidates the
// SM's L1; these reads are plain loads (not the read-only path).
#include <limits.h>
#include <math.h>

#include "synk_internal.cuh"
#include "sirt_internal.cuh"
#include "sirt_device.cuh"
#include "sirt_offset.cuh"
#include "poll_limit.cuh"
#include "fp_tile.cuh"
#include "bp_tile.cuh"

namespace synk {

namespace {

constexpr int kWarpsSmall = 32;

// A warp's near-axis or corner ray, decoded: its line, rows and data.
struct ExtraRay {
    float slope, intercept, lbase, Rk, b, scale;   // scale: row scale, or the chord of a corner ray
    int j0, j1;                                      // frame rows (none when the ray misses the image)
    const float *img;                                // frame image of the slice
    float *dst;                                      // where the residual (corner ray: its term) goes, null: nowhere
    int s, corner;
};

constexpr int kExactSmall = 8;        // near-axis angles whose geometry is kept in shared memory

struct SmallShared {
    ExtraRay extra[kWarpsSmall];
    AngleGeom exg[kExactSmall];
    int exk[kExactSmall];
    int goff[5];                      // offsets of the corners' lists
    // angle pairs (2j, 2j+1), near-axis angles with zero weight: cos and sin, h/b
    // and 1/b, c1 (bp_chunk's) and the row's byte offset less the magic constant's
    float4 cs[kSirtSmallAngles / 2], hb[kSirtSmallAngles / 2], cr[kSirtSmallAngles / 2];
    // forward units of the warps: (slice or -1, first row, end row, flat); per lane
    // x0, slope, 1/|slope|, lbase (0: no ray), and on the first row part b, R, row
    // scale, index of the residual
    int4 unit[kWarpsSmall];
    float4 line[kWarpsSmall][32], meas[kWarpsSmall][32];
    float red[kWarpsSmall][33];
    int flag, any;
};

__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid barrier number `epoch` (1, 2, ...): the counter only grows.  False in
// every thread once the wait ran out of time (PollLimit; the status word is then set).
__device__ __forceinline__ bool small_barrier(unsigned *count, unsigned target, int *status,
                                              unsigned long long timeout_ns, int *s_flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        if ((int)(ld_relaxed_u32(count) - target) < 0) {
            PollLimit limit;
            limit.start(global_ns());
            for (unsigned spin = 1; (int)(ld_relaxed_u32(count) - target) < 0; ++spin)
                if ((spin & 63u) == 0u && (limit.over(global_ns(), timeout_ns) || spin > (1u << 30))) {
                    atomicExch(status, SYNK_ETIMEOUT);
                    ok = 0;
                    break;
                }
        }
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        *s_flag = ok;
    }
    __syncthreads();
    return *s_flag != 0;
}

// Consecutive angles of a forward chunk: as many as leave a block about three chunks.
__host__ __device__ inline int small_chunk(long long units, int grid) {
    int c = 1;
    while (c < 8 && units >= 5LL * c * grid) c *= 2;
    return c;
}

// Decodes forward unit (slice s, angle slot, detector group d), s < 0: none, into
// the warp's entries of sh.
__device__ __forceinline__ void fp_unit(const SirtProblem &q, SmallShared &sh, int s, int slot, int d, int steep_slots,
                                        int part, int S) {
    const ProbGeom &P = q.P;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ka = s >= 0 ? __ldg(q.L.order + slot) : -1;               // -1: padding of an angle group
    const int r = d * 32 + lane;
    const bool in = ka >= 0 && r < P.D;
    const WarpRay R = warp_ray(P, in ? ka : -1, in ? r : 0, part * P.N / S, (part + 1) * P.N / S);
    __syncwarp();
    if (lane == 0) sh.unit[warp] = make_int4(ka >= 0 ? s : -1, R.J0, R.J1, slot < steep_slots ? 0 : 1);
    sh.line[warp][lane] = make_float4(R.x0, R.slope, R.ainv, R.valid ? R.lbase : 0.0f);
    if (part == 0) {
        float4 m = make_float4(0.0f, -1.0f, 0.0f, 0.0f);           // R < 0: no residual of this lane
        if (in) {
            const size_t ray = (size_t)ka * P.D + r, out = (size_t)s * P.a * P.D + ray;
            m = make_float4(__ldg(q.b + out), __ldg(q.R + ray), row_scale(P.geom, ka), __int_as_float((int)out));
        }
        sh.meas[warp][lane] = m;
    }
    __syncwarp();
}

// Sum of the unit's rows (fp_lane_walk's arithmetic, eight rows of gathers in
// flight): v0 = pixel c, v1 = pixel c+1 of the padded frame image, the index
// clamped to the zero entries N+1 and N+2 outside the image and past the last row.
// A lane without a ray walks pixels that are not its own: its sum is dropped, not
// multiplied by zero (the pixels may be infinite or NaN).
__device__ __forceinline__ float small_walk(const ProbGeom &P, const float4 L, int J0, int J1, const float *img) {
    const unsigned W = (unsigned)(P.N + 2), zix = (unsigned)P.N + 1u;
    const unsigned okbase = (unsigned)kMagicBits - 1u - (unsigned)P.half;   // bits(r) - okbase = c + 1
    const f32x2 sl2 = pk2(L.y, L.y), x02 = pk2(L.x, L.x);
    const f32x2 mg2 = pk2(kMagic, kMagic), m1 = pk2(-1.0f, -1.0f);
    const float ainv = L.z, omv = __fsub_rn(1.0f, L.z);
    float sum = 0.0f, comp = 0.0f, part = 0.0f;
    int n = 0;
    for (int j = J0; j < J1; j += 8) {
        float t[8], v0[8], v1[8];
        const float jf = (float)(j - P.half);
        const int left = J1 - j;                                            // warp-uniform
#pragma unroll
        for (int h = 0; h < 8; h += 2) {
            const f32x2 x = fma2(pk2(jf + (float)h, jf + (float)(h + 1)), sl2, x02);
            const f32x2 rr = add2_rd(x, mg2);
            const float2 f = unpk2(add2(x, fma2(rr, m1, mg2))), rv = unpk2(rr);      // x - floor(x)
            unsigned i0 = min((unsigned)__float_as_int(rv.x) - okbase, zix);
            unsigned i1 = min((unsigned)__float_as_int(rv.y) - okbase, zix);
            int j0 = j + h, j1 = j + h + 1;
            if (left < 8) {                                                    // rows past the last: a zero entry of row j
                if (h >= left) i0 = zix, j0 = j;
                if (h + 1 >= left) i1 = zix, j1 = j;
            }
            const float *p0 = img + (i0 + (unsigned)j0 * W), *p1 = img + (i1 + (unsigned)j1 * W);
            v0[h] = p0[0];
            v1[h] = p0[1];
            v0[h + 1] = p1[0];
            v1[h + 1] = p1[1];
            t[h] = __saturatef(__fmaf_rn(f.x, ainv, omv));
            t[h + 1] = __saturatef(__fmaf_rn(f.y, ainv, omv));
        }
#pragma unroll
        for (int h = 0; h < 8; ++h) part += fmaf(t[h], v1[h] - v0[h], v0[h]);
        if (++n == kSirtCompRows / 8) {
            comp_add(sum, comp, part);
            part = 0.0f;
            n = 0;
        }
    }
    comp_add(sum, comp, part);
    return L.w != 0.0f ? (sum + comp) * L.w : 0.0f;
}

// Decodes extra x of the problem: slice by slice the near-axis rays, then the
// listed corner rays (graze_ray of sirt.cu).
__device__ __forceinline__ ExtraRay extra_ray(const SirtProblem &q, long long x, int nexact, int ngraze) {
    const ProbGeom &P = q.P;
    const int per = nexact * P.D + ngraze;
    const size_t pr = (size_t)P.a * P.D, np = (size_t)P.N * (P.N + 2);
    ExtraRay e;
    e.s = (int)(x / per);
    const int i = (int)(x - (long long)e.s * per);
    int k, r, slot = -1;
    if (i < nexact * P.D) {
        k = __ldg(q.L.exact + i / P.D);
        r = i % P.D;
    } else {
        const int gidx = i - nexact * P.D;
        int c = 0;
        while (c < 3 && gidx >= __ldg(q.goff + c + 1)) ++c;
        slot = c * q.graze_capc + (gidx - __ldg(q.goff + c));
        const int2 ent = __ldg(q.graze + slot);
        k = ent.x;
        r = ent.y;
    }
    const AngleGeom g = load_geom(P.geom, k);
    const float rho = __fadd_rn(P.rhozero, __fmul_rn((float)r, P.deltarho));
    e.slope = g.slope;
    e.intercept = __fdiv_rn(rho, g.cost);
    e.lbase = g.lbase;
    e.img = (g.flat ? q.xTpad : q.xpad) + (size_t)e.s * np;
    e.j0 = 0;
    e.j1 = P.N;
    if (slot >= 0) lane_rows(P, g, ray_x0(g, e.intercept), e.j0, e.j1);
    if (fabsf(rho) > 0.75f * (float)P.N + 2.0f) e.j1 = e.j0;
    const size_t ray = (size_t)k * P.D + r;
    e.Rk = __ldg(q.R + ray);
    e.b = __ldg(q.b + (size_t)e.s * pr + ray);
    e.corner = slot >= 0;
    if (e.corner) {
        e.scale = __ldg(q.glen + slot);
        e.dst = q.gcontrib + (size_t)e.s * 4 * q.graze_capc + slot;
    } else {
        e.scale = row_scale(P.geom, k);
        e.dst = e.Rk < 0.0f ? nullptr : q.rr + (size_t)e.s * pr + ray;
    }
    return e;
}

// The ray's sum by the warp's lanes over its frame rows, the reference's own
// expressions (fp_exact_ray_warp on data that other blocks wrote).
__device__ __forceinline__ float extra_walk(const ProbGeom &P, const ExtraRay &e) {
    float acc = 0.0f;
    const int iend = min(P.half, -P.half + e.j1);
    for (int i = -P.half + e.j0 + (int)(threadIdx.x & 31); i < iend; i += 32) {
        const ExactRow w = fp_row_exact_terms(P.half, e.slope, e.intercept, e.lbase, i);
        const float *row = e.img + (size_t)(i + P.half) * (P.N + 2) + P.half + 1;
        const float b = w.botin ? __fmul_rn(w.lbot, row[w.xpb]) : 0.0f;
        const float t = w.topin ? __fmul_rn(w.ltop, row[w.xpt]) : 0.0f;
        acc = __fadd_rn(acc, __fadd_rn(b, t));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    return acc;
}

// Adds e^2 (lane values) of the warp's ray(s) of slice s to its residual sum.
__device__ __forceinline__ void small_add_e2(const SirtProblem &q, int s, int it, double e2) {
    const double w = warp_sum_d(e2);
    if ((threadIdx.x & 31) == 0 && w != 0.0) atomicAdd(q.res2 + (size_t)s * (q.iterations + 1) + it, w);
}

__device__ __forceinline__ bool small_fp_needed(const SirtSmall &p, int s, int it) {
    const SirtProblem &q = p.q;
    if (it > q.iterations || (it == q.iterations && !p.record_final)) return false;
    return !(p.tol2 > 0.0 && stop_of(q, s) < it);
}

template <bool INRANGE>
__global__ void __launch_bounds__(1024, 1) sirt_small_kernel(const SirtSmall p) {
    __shared__ SmallShared sh;
    const SirtProblem &q = p.q;
    const ProbGeom &P = q.P;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = gridDim.x;
    const int apairs = (P.a + 1) >> 1;
    for (int j = threadIdx.x; j < apairs; j += 1024) {
        float c[2], si[2], h[2], ib[2], c1[2], ro[2];
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const int k = min(2 * j + o, P.a - 1);
            const AngleGeom g = load_geom(P.geom, k);
            // no weight without a finite line, nor past the last angle, whose entries
            // the filler of an odd count reads again: a detector outside a pixel's
            // window must not enter it, not even times zero (it may be NaN)
            const bool line = !g.exact && fabsf(g.c) <= 2.0f, w = line && 2 * j + o < P.a;
            c[o] = line ? g.c : 0.0f;
            si[o] = line ? g.s : 0.0f;
            h[o] = w ? g.h_over_b : -1.0f;
            ib[o] = w ? g.inv_b : 0.0f;
            c1[o] = w ? fmaf(-(1.0f - fact_f32()), g.inv_b, g.h_over_b) : -1.0f;
            ro[o] = __uint_as_float(small_row_offset(k, P.D, P.zi, kMagicBits));
        }
        sh.cs[j] = make_float4(c[0], c[1], si[0], si[1]);
        sh.hb[j] = make_float4(h[0], h[1], ib[0], ib[1]);
        sh.cr[j] = make_float4(c1[0], c1[1], ro[0], ro[1]);
    }
    const int nsteep = __ldg(q.L.counts), ngroups = nsteep + __ldg(q.L.counts + 1), nexact = __ldg(q.L.counts + 2);
    const int ngraze = graze_count(q);
    const size_t np = (size_t)P.N * (P.N + 2), pr = (size_t)P.a * P.D;
    // forward: this block's chunks of CH units, G units at a time; the near-axis and
    // corner rays on the warps that are idle in every block's last round
    const int S = p.S, G = kWarpsSmall / S, part = warp % S;
    const int slots = ngroups * 32, dg = (P.D + 31) >> 5;
    const long long units = (long long)slots * dg * q.nslices;
    const int CH = small_chunk(units, nb);
    const long long nchunks = units / CH;                                     // slots is a multiple of 32
    const int umax = (int)((nchunks + nb - 1) / nb) * CH, frounds = (umax + G - 1) / G;
    const long long extras = (long long)(nexact * P.D + ngraze) * q.nslices;
    const int used = frounds > 0 ? (umax - (frounds - 1) * G) * S : 0;
    const int spare = used < kWarpsSmall ? kWarpsSmall - used : kWarpsSmall;
    const int ew = used < kWarpsSmall ? warp - used : warp;                 // this warp's extra slot, < 0: none
    auto funit = [&](int f) {
        const int l = f * G + warp / S;
        const long long chunk = (long long)(l / CH) * nb + blockIdx.x;
        const long long sc = chunk / dg;                                       // slice and slot chunk
        const int per = slots / CH;
        const int s = chunk < nchunks ? (int)(sc / max(per, 1)) : -1;
        fp_unit(q, sh, s, (int)(sc % max(per, 1)) * CH + l % CH, (int)(chunk - sc * dg), nsteep * 32, part, S);
    };
    // backward: this block's consecutive units, GB at a time
    const int SB = p.SB, GB = kWarpsSmall / SB, bpart = warp % SB;
    const int tx_n = (P.N + 31) >> 5;
    const long long bunits = (long long)tx_n * P.N * q.nslices;
    const long long bbeg = bunits * blockIdx.x / nb, bend = bunits * (blockIdx.x + 1) / nb;
    const int brounds = (int)(((bunits + nb - 1) / nb + GB - 1) / GB);
    struct BpUnit {
        int s, row, tx;
    };
    auto bunit = [&](int f) {
        BpUnit u = {-1, 0, 0};
        const long long x = bbeg + (long long)f * GB + warp / SB;
        if (x < bend) {
            u.s = (int)(x / ((long long)tx_n * P.N));
            const int rem = (int)(x - (long long)u.s * tx_n * P.N);
            u.tx = rem / P.N;
            u.row = rem - u.tx * P.N;
        }
        return u;
    };
    const float fact = fact_f32(), zoff = -P.rz_c - fact;

    const long long x0 = (long long)ew * nb + blockIdx.x;
    if (ew >= 0 && x0 < extras && lane == 0) sh.extra[warp] = extra_ray(q, x0, nexact, ngraze);
    for (int e = threadIdx.x; e < min(nexact, kExactSmall); e += 1024) {
        sh.exk[e] = __ldg(q.L.exact + e);
        sh.exg[e] = load_geom(P.geom, sh.exk[e]);
    }
    if (threadIdx.x < 5) sh.goff[threadIdx.x] = __ldg(q.goff + threadIdx.x);
    if (frounds > 0) funit(0);
    float C0 = 0.0f;                  // C of this lane's pixel when there is one backward round
    BpUnit bu = bunit(0);
    if (brounds == 1 && bpart == 0 && bu.s >= 0 && bu.tx * 32 + lane < P.N)
        C0 = __ldg(q.C + (size_t)bu.row * P.N + bu.tx * 32 + lane);
    __syncthreads();
    unsigned epoch = 0;
    const unsigned arrivals = (unsigned)nb;
    for (int it = 0; it <= q.iterations; ++it) {
        // ---- forward: e = b - FP(x), rr = R*e (residual() of sirt.cu) ----
        for (int f = 0; f < frounds; ++f) {
            if (frounds > 1) funit(f);
            const int4 u = sh.unit[warp];
            const bool on = u.x >= 0 && small_fp_needed(p, u.x, it);           // uniform over the unit's warps
            float v = 0.0f;
            if (on) v = small_walk(P, sh.line[warp][lane], u.y, u.z, (u.w ? q.xTpad : q.xpad) + (size_t)u.x * np);
            if (S > 1) {
                sh.red[warp][lane] = v;
                __syncthreads();
                if (part == 0)
                    for (int t = 1; t < S; ++t) v += sh.red[warp + t][lane];
                if (f + 1 < frounds) __syncthreads();
            }
            if (on && part == 0) {
                const float4 m = sh.meas[warp][lane];
                double e2 = 0.0;
                if (!(m.y < 0.0f)) {                                           // (negative: a listed corner ray)
                    const float e = __fsub_rn(m.x, v);
                    q.rr[__float_as_int(m.w)] = __fmul_rn(__fmul_rn(m.y, e), m.z);
                    e2 = (double)e * (double)e;
                }
                if (p.want_e2) small_add_e2(q, u.x, it, e2);
            }
        }
        if (ew >= 0)
            for (long long x = x0; x < extras; x += (long long)spare * nb) {
                if (x != x0 || extras > (long long)spare * nb) {                  // more than one: decode it again
                    __syncwarp();
                    if (lane == 0) sh.extra[warp] = extra_ray(q, x, nexact, ngraze);
                    __syncwarp();
                }
                const ExtraRay &e = sh.extra[warp];
                if (!small_fp_needed(p, e.s, it)) continue;
                const float v = extra_walk(P, e);
                double e2 = 0.0;
                if (lane == 0 && e.dst) {
                    const float d = __fsub_rn(e.b, v);
                    *e.dst = e.corner ? __fmul_rn(e.scale, __fmul_rn(-e.Rk, d)) : __fmul_rn(__fmul_rn(e.Rk, d), e.scale);
                    e2 = (double)d * (double)d;
                }
                if (p.want_e2) small_add_e2(q, e.s, it, e2);
            }
        if (it == q.iterations) break;             // the kernel's end publishes the last residuals
        if (!small_barrier(p.count, ++epoch * arrivals + p.extra, p.status, p.timeout_ns, &sh.flag)) return;
        // stopping rule (the same decision in every block)
        if (p.tol2 > 0.0) {
            if (threadIdx.x == 0) sh.any = 0;
            __syncthreads();
            for (int s = threadIdx.x; s < q.nslices; s += 1024) {
                if (bp_needed(p.tol2, q, s, it)) sh.any = 1;
                else if (blockIdx.x == 0 && stop_of(q, s) > it) q.stop_iter[s] = it;
            }
            __syncthreads();
            if (!sh.any) break;
        }
        // ---- backward: x + C*BP(rr) (SIRT.fut:38-39) ----
        for (int f = 0; f < brounds; ++f) {
            if (brounds > 1) bu = bunit(f);
            const int s = bu.s, row = bu.row, tx = bu.tx;
            const bool on = s >= 0 && bp_needed(p.tol2, q, s, it);              // uniform over the unit's warps
            const int col = tx * 32 + lane;
            const bool in = on && col < P.N;
            float acc = 0.0f;
            float x = 0.0f, C = 0.0f;
            float *xp = q.xpad + (size_t)(on ? s : 0) * np + (size_t)row * (P.N + 2) + col + 1;
            if (in && bpart == 0) {
                x = *xp;
                C = brounds == 1 ? C0 : __ldg(q.C + (size_t)row * P.N + col);
            }
            // the image corners add the terms of the rays that clip only them, every angle
            // part its share of the list (its first entries are fetched ahead of the walk)
            const bool crow = on && (row == 0 || row == P.N - 1);                // warp-uniform
            float ct[2] = {0.0f, 0.0f};
            const int ci = bpart * 32 + lane;
            if (crow) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = (row == P.N - 1 ? 2 : 0) + h;
                    if (tx == (h ? tx_n - 1 : 0) && ci < sh.goff[c + 1] - sh.goff[c])
                        ct[h] = q.gcontrib[((size_t)s * 4 + c) * q.graze_capc + ci];
                }
            }
            if (on) {
                const float *rr = q.rr + (size_t)s * pr;
                const char *rrb = reinterpret_cast<const char *>(rr - kSmallLead);
                const float xc = (float)(col - P.half) + 0.5f, yc = (float)(row - P.half) + 0.5f;
                const f32x2 xc2 = pk2(xc, xc), nyc2 = pk2(-yc, -yc), zo2 = pk2(zoff, zoff);
                const f32x2 mg2 = pk2(kMagic, kMagic), nmg2 = pk2(-kMagic, -kMagic), m1 = pk2(-1.0f, -1.0f);
                const f32x2 nf2 = pk2(-fact, -fact);
                const int jend = apairs * (bpart + 1) / SB;
                float sum = 0.0f, comp = 0.0f, psum = 0.0f;
                int n = 0;
                for (int j0 = apairs * bpart / SB; j0 < jend; j0 += 4) {
                    float v0[8], v1[8], w0[8], w1[8];
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const int j = min(j0 + h, jend - 1);
                        const float4 a4 = sh.cs[j], b4 = sh.hb[j], c4 = sh.cr[j];
                        const f32x2 qv = fma2(xc2, pk2(a4.x, a4.y), fma2(nyc2, pk2(a4.z, a4.w), zo2));
                        const f32x2 r2 = add2_ru(qv, mg2);
                        const f32x2 e2v = fma2(qv, m1, add2(r2, nmg2));         // ceil(q) - q
                        const float2 ev = unpk2(e2v), dv = unpk2(add2(e2v, nf2)), rv = unpk2(r2);
#pragma unroll
                        for (int o = 0; o < 2; ++o) {
                            const int i = 2 * h + o;
                            const float ib = o ? b4.w : b4.z;
                            const unsigned off = small_gather_offset(__float_as_uint(o ? rv.y : rv.x),
                                                                     __float_as_uint(o ? c4.w : c4.z));
                            w0[i] = __saturatef(fmaf(-fabsf(o ? dv.y : dv.x), ib, o ? b4.y : b4.x));
                            w1[i] = __saturatef(fmaf(-(o ? ev.y : ev.x), ib, o ? c4.y : c4.x));
                            if (j0 + h >= jend) w0[i] = w1[i] = 0.0f;            // past the part's last pair
                            const float *pv = reinterpret_cast<const float *>(rrb + off);
                            if (INRANGE) {
                                v0[i] = pv[0];
                                v1[i] = pv[1];
                            } else {
                                const int det = __float_as_int(o ? rv.y : rv.x) - kMagicBits + P.zi;
                                v0[i] = (unsigned)det < (unsigned)P.D ? pv[0] : 0.0f;
                                v1[i] = (unsigned)(det + 1) < (unsigned)P.D ? pv[1] : 0.0f;
                            }
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 8; ++h) psum = fmaf(w1[h], v1[h], fmaf(w0[h], v0[h], psum));
                    if (++n == kBpChunk / 8) {
                        comp_add(sum, comp, psum);
                        psum = 0.0f;
                        n = 0;
                    }
                }
                comp_add(sum, comp, psum);
                acc = sum + comp;
                // near-axis angles, the reference's own expressions (bp_exact_angles)
                float ex = 0.0f;
                for (int e = bpart; e < nexact; e += SB) {
                    const int k = e < kExactSmall ? sh.exk[e] : __ldg(q.L.exact + e);
                    const AngleGeom g = e < kExactSmall ? sh.exg[e] : load_geom(P.geom, k);
                    if (!in) continue;
                    float a1 = 0.0f;
                    bp_exact_terms(P, g, row, col, [&](int det, float l) {
                        a1 = __fadd_rn(a1, __fmul_rn(l, rr[(size_t)k * P.D + det]));
                    });
                    ex += a1;
                }
                acc += ex;
                if (crow) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int c = (row == P.N - 1 ? 2 : 0) + h;
                        if (tx != (h ? tx_n - 1 : 0)) continue;
                        const int n = sh.goff[c + 1] - sh.goff[c];
                        for (int i = ci + 32 * SB; i < n; i += 32 * SB)
                            ct[h] = __fadd_rn(ct[h], q.gcontrib[((size_t)s * 4 + c) * q.graze_capc + i]);
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) ct[h] = __fadd_rn(ct[h], __shfl_xor_sync(0xffffffffu, ct[h], o));
                        if (col == (h ? P.N - 1 : 0)) acc = __fadd_rn(acc, ct[h]);
                    }
                }
            }
            if (SB > 1) {
                if (f > 0) __syncthreads();
                sh.red[warp][lane] = acc;
                __syncthreads();
                if (bpart == 0)
                    for (int t = 1; t < SB; ++t) acc += sh.red[warp + t][lane];
            }
            if (on && bpart == 0) {
                if (in) {
                    const float xi = __fadd_rn(x, __fmul_rn(C, acc));
                    *xp = xi;
                    q.xTpad[(size_t)s * np + (size_t)col * (P.N + 2) + row + 1] = xi;
                }
            }
        }
        if (!small_barrier(p.count, ++epoch * arrivals + p.extra, p.status, p.timeout_ns, &sh.flag)) return;
    }
}

}  // namespace

int sirt_small_grid() {
    int dev = 0, sms = 0, b = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, sirt_small_kernel<true>, 1024, 0);
    int c = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, sirt_small_kernel<false>, 1024, 0);
    return b > 0 && c > 0 ? sms : 0;
}

void sirt_small_splits(const ProbGeom &P, int nslices, int grid, int *S, int *SB) {
    const long long fu = (long long)((P.a + 31) / 32 + 1) * 32 * ((P.D + 31) / 32) * nslices;
    const long long bu = (long long)((P.N + 31) / 32) * P.N * nslices;
    const int ch = small_chunk(fu, grid);
    const long long fb = ((fu / ch + grid - 1) / grid) * ch, bb = (bu + grid - 1) / grid;      // most units of a block
    int s = 1;
    while (s < 8 && fb * s * 2 <= kWarpsSmall && P.N / (2 * s) >= 8) s *= 2;
    int b = 1;
    while (b < 32 && bb * b * 2 <= kWarpsSmall && P.a / (2 * b) >= 4) b *= 2;
    *S = s;
    *SB = b;
}

cudaError_t launch_sirt_small(const SirtSmall &p, int grid, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(1024);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return p.q.bp_inrange ? cudaLaunchKernelEx(&cfg, sirt_small_kernel<true>, p)
                          : cudaLaunchKernelEx(&cfg, sirt_small_kernel<false>, p);
}

}  // namespace synk
