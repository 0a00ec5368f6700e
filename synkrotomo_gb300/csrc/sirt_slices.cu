// SIRT phases of a slice stack (futhark/SIRT3D.fut:23-28): the slices share one
// geometry, so a thread evaluates a ray's (a pixel's) indices and weights once
// and applies them to the V slices of a group.
//
// Layout: groups of V = 4 slices interleaved as float4 (a last group of one or
// two slices as float2, V = 2; absent slices are zero).  Group g at 4*g times
// the per-slice size holds the padded iterate xpad[N][N+2][V] and its transpose
// xTpad (a zero entry on each side of a row, more after the last), and the
// weighted residual rr[a*D][V].  One gather then serves V slices.
//
// What bounds them: the L1's return path.  A gather returns at most 128 bytes
// per cycle and SM to the registers, whatever its lanes share (a warp's 16-byte
// gather takes at least four cycles, measured 4.06), so a step's two 16-byte
// gathers take 2.03 cycles per slice, while the shared index and weight
// arithmetic takes about 1.1; one slice at a time took 2.6-3.2 issue cycles.
// N=512, 360 angles: 16 slices x 10 iterations 18.6 -> 8.95 ms, 512 slices
// 105.7 -> 49.7 us per slice and iteration.
#include <math.h>

#include "synk_internal.cuh"
#include "sirt_internal.cuh"
#include "sirt_device.cuh"
#include "fp_tile.cuh"
#include "bp_tile.cuh"
#include "f32x2.cuh"

namespace synk {

namespace {

template <int V>
struct VecOf;
template <> struct VecOf<2> { typedef float2 T; };
template <> struct VecOf<4> { typedef float4 T; };
template <int V>
using Vec = typename VecOf<V>::T;

// the V values of an entry, as packed pairs or as an array
__device__ __forceinline__ void ld_pairs(const float2 *p, f32x2 (&v)[1]) { v[0] = pk2(__ldg(p)); }
__device__ __forceinline__ void ld_pairs(const float4 *p, f32x2 (&v)[2]) {
    const float4 u = __ldg(p);
    v[0] = pk2(u.x, u.y);
    v[1] = pk2(u.z, u.w);
}
__device__ __forceinline__ void to_array(const float2 &u, float (&a)[2]) { a[0] = u.x; a[1] = u.y; }
__device__ __forceinline__ void to_array(const float4 &u, float (&a)[4]) { a[0] = u.x; a[1] = u.y; a[2] = u.z; a[3] = u.w; }
__device__ __forceinline__ float2 to_vec(const float (&a)[2]) { return make_float2(a[0], a[1]); }
__device__ __forceinline__ float4 to_vec(const float (&a)[4]) { return make_float4(a[0], a[1], a[2], a[3]); }

// Group of slices s0 .. s0+V-1 of the stack.  A clamped gather of an image's
// last row reads one entry past the group: the zero entry that starts the
// next group of four, or kGroupPad zero floats before the last group of two (whose entries
// are narrower) and at the end.
constexpr int kGroupPad = 8;
template <int V>
__device__ __forceinline__ Vec<V> *group_ptr(float *base, int s0, size_t per_slice) {
    return reinterpret_cast<Vec<V> *>(base + (size_t)s0 * per_slice + (V == 2 ? kGroupPad : 0));
}

constexpr int kSlotsExact = 4;      // near-axis angle slots of the exact kernel (repeats loop)

// The ray's sums over rows [J0, J1) of the group's V slices on its padded
// frame image (32-bit byte offsets: below 4 GB, checked by the host).  Per
// row: x = (j - half)*slope + x0, c = floor(x) + half, t = share of column c+1,
// sum += (1 - t)*v[c] + t*v[c+1].  Plain float32 over kSirtCompRows rows,
// compensated across chunks.
template <int V>
__device__ __forceinline__ void group_walk(const ProbGeom &P, const WarpRay &R, const char *__restrict__ img,
                                           float (&out)[V]) {
    constexpr unsigned EB = 4u * V;                                           // bytes of an entry
    const unsigned rowbytes = (unsigned)(P.N + 2) * EB;
    const unsigned okbase = (unsigned)kMagicBits - 1u - (unsigned)P.half;   // bits(r) - okbase = c + 1
    const unsigned zix = (unsigned)P.N + 1u;                                 // entries N+1, N+2 are zero
    const f32x2 sl2 = pk2(R.slope, R.slope), x02 = pk2(R.x0, R.x0);
    const f32x2 mg2 = pk2(kMagic, kMagic), m1 = pk2(-1.0f, -1.0f), two2 = pk2(2.0f, 2.0f);
    const float ainv = R.ainv, omv = __fsub_rn(1.0f, R.ainv);
    float sum[V], comp[V];
#pragma unroll
    for (int i = 0; i < V; ++i) sum[i] = comp[i] = 0.0f;
    f32x2 part[V / 2];

    auto gather = [&](unsigned off, float t) {
        const f32x2 t2 = pk2(t, t);
        const float u = __fsub_rn(1.0f, t);
        const f32x2 u2 = pk2(u, u);
        const Vec<V> *e = reinterpret_cast<const Vec<V> *>(img + off);
        f32x2 a[V / 2], b[V / 2];
        ld_pairs(e, a);
        ld_pairs(e + 1, b);
#pragma unroll
        for (int p = 0; p < V / 2; ++p) {
            part[p] = fma2(u2, a[p], part[p]);
            part[p] = fma2(t2, b[p], part[p]);
        }
    };
    auto rows = [&](int ja, int jz, bool clamp) {
        for (int j = ja; j < jz;) {
            const int jend = min(j + kSirtCompRows, jz);
#pragma unroll
            for (int p = 0; p < V / 2; ++p) part[p] = pk2(0.0f, 0.0f);
            const float jf = (float)(j - P.half);
            f32x2 jf2 = pk2(jf, jf + 1.0f);
            // unclamped offset: bits*EB + rowoff (mod 2^32)
            unsigned rowoff = (unsigned)j * rowbytes - (clamp ? 0u : okbase * EB);
            auto two = [&](bool second) {
                const f32x2 x = fma2(jf2, sl2, x02);
                const f32x2 rr = add2_rd(x, mg2);
                const f32x2 f = add2(x, fma2(rr, m1, mg2));         // x - floor(x)
                const float2 fv = unpk2(f), rv = unpk2(rr);
                unsigned ia = (unsigned)__float_as_int(rv.x), ib = (unsigned)__float_as_int(rv.y);
                if (clamp) {
                    ia = min(ia - okbase, zix);
                    ib = min(ib - okbase, zix);
                }
                gather(ia * EB + rowoff, __saturatef(__fmaf_rn(fv.x, ainv, omv)));
                if (second) gather(ib * EB + rowoff + rowbytes, __saturatef(__fmaf_rn(fv.y, ainv, omv)));
                jf2 = add2(jf2, two2);
                rowoff += 2u * rowbytes;
            };
            for (; j + 3 < jend; j += 4) {
                two(true);
                two(true);
            }
            for (; j < jend; j += 2) two(j + 1 < jend);
            j = jend;
#pragma unroll
            for (int p = 0; p < V / 2; ++p) {
                const float2 v = unpk2(part[p]);
                comp_add(sum[2 * p], comp[2 * p], v.x);
                comp_add(sum[2 * p + 1], comp[2 * p + 1], v.y);
            }
        }
    };
    rows(R.J0, R.I0, true);
    rows(R.I0, R.I1, false);
    rows(R.I1, R.J1, true);
#pragma unroll
    for (int i = 0; i < V; ++i) out[i] = R.valid ? (sum[i] + comp[i]) * R.lbase : 0.0f;
}

// Residuals of one ray for the group's slices (residual() of sirt.cu): e = b -
// fp, rr = R*e times the row's scale.  e2[i] += e^2 when wanted.
template <int V>
__device__ __forceinline__ void group_residual(const SirtProblem &q, int s0, int k, int r, const float (&v)[V],
                                               bool want_e2, double (&e2)[V]) {
    const size_t pr = (size_t)q.P.a * q.P.D;
    const size_t ray = (size_t)k * q.P.D + r;
    const float Rk = q.R[ray];
    if (Rk < 0.0f) return;                            // a listed corner ray (graze lists)
    const float sc = row_scale(q.P.geom, k);
    float w[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const float e = s0 + i < q.nslices ? __fsub_rn(q.b[(size_t)(s0 + i) * pr + ray], v[i]) : 0.0f;
        w[i] = __fmul_rn(__fmul_rn(Rk, e), sc);
        if (want_e2) e2[i] += (double)e * (double)e;
    }
    group_ptr<V>(q.rr, s0, pr)[ray] = to_vec(w);
}

// Any slice of the group still needs the forward phase of iteration it.
template <int V>
__device__ __forceinline__ bool group_fp_needed(const SirtProblem &q, int s0, int it, double tol2) {
    if (tol2 <= 0.0) return true;
    for (int s = s0; s < min(s0 + V, q.nslices); ++s)
        if (stop_of(q, s) >= it) return true;
    return false;
}

// Adds the block's e^2 to the slices' residual sums: warp i sums slice i.
template <int V>
__device__ __forceinline__ void group_flush_e2(const SirtProblem &q, int s0, int it, const double (&e2)[V],
                                               double (*sh)[256]) {
#pragma unroll
    for (int i = 0; i < V; ++i) sh[i][threadIdx.x] = e2[i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s = s0 + warp;
    if (warp < V && s < q.nslices) {
        double t = 0.0;
        for (int i = lane; i < 256; i += 32) t += sh[warp][i];
        t = warp_sum_d(t);
        if (lane == 0 && t != 0.0) atomicAdd(q.res2 + (size_t)s * (q.iterations + 1) + it, t);
    }
}

// Forward phase: the projector's grid (8/S detectors x S row parts of 32
// angles per block; with S = 1 a warp holds 4 angles x 8 detectors), one slice
// group per blockIdx.z, the residual as its epilogue.
template <int S, int V>
__global__ void __launch_bounds__(256, 4) sirt_fp_slices_kernel(SirtProblem q, int slice_base, int it, double tol2,
                                                                int record_final, int want_e2) {
    __shared__ Vec<V> red[S > 1 ? 8 : 1][32];
    __shared__ double she[V][256];
    const int s0 = slice_base + blockIdx.z * V;
    if (it > q.iterations || (it == q.iterations && !record_final)) return;       // block-uniform
    if (!group_fp_needed<V>(q, s0, it, tol2)) return;
    const int grp = blockIdx.y;
    const int nsteep = __ldg(q.L.counts), nflat = __ldg(q.L.counts + 1);
    if (grp >= nsteep + nflat) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int part = warp % S;
    // S = 1: a warp's 4 angles x 8 detectors with 2 angles x 4 detectors in each
    // quarter, whose eight 16-byte entries of a row then cross fewer lines than
    // those of 8 detectors (N=512, 360 angles, 16 slices: 11.1 -> 10.4 ms; 4 x 2: 10.5)
    const int dl = (lane & 3) + ((lane >> 3) & 1) * 4, al = ((lane >> 2) & 1) + (lane >> 4) * 2;
    const int r = S == 1 ? blockIdx.x * 8 + dl : blockIdx.x * (8 / S) + warp / S;
    const int k = r < q.P.D ? __ldg(q.L.order + grp * 32 + (S == 1 ? warp * 4 + al : lane)) : -1;
    const int jb = (int)((long long)part * q.P.N / S), je = (int)((long long)(part + 1) * q.P.N / S);
    const size_t np = (size_t)q.P.N * (q.P.N + 2);
    const Vec<V> *img = group_ptr<V>(grp < nsteep ? q.xpad : q.xTpad, s0, np);
    const WarpRay R = warp_ray(q.P, k, r, jb, je);
    float v[V];
    group_walk<V>(q.P, R, reinterpret_cast<const char *>(img), v);
    if (S > 1) {
        red[warp][lane] = to_vec(v);
        __syncthreads();
    }
    double e2[V];
#pragma unroll
    for (int i = 0; i < V; ++i) e2[i] = 0.0;
    if (part == 0 && k >= 0) {
        if (S > 1)
            for (int t = 1; t < S; ++t) {
                float o[V];
                to_array(red[warp + t][lane], o);
#pragma unroll
                for (int i = 0; i < V; ++i) v[i] += o[i];
            }
        group_residual<V>(q, s0, k, r, v, want_e2 != 0, e2);
    }
    if (want_e2) group_flush_e2<V>(q, s0, it, e2, she);
}

// fp_exact_ray_warp for V slices: the row's two lengths once, applied to
// every slice in the reference's expressions; the sums in every lane.
template <int V>
__device__ __forceinline__ void exact_ray_group(const ProbGeom &P, int k, int r, const Vec<V> *__restrict__ xs,
                                                const Vec<V> *__restrict__ xTs, int jb, int je, float (&acc)[V]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = 0.0f;
    const AngleGeom g = load_geom(P.geom, k);
    const float rho = __fadd_rn(P.rhozero, __fmul_rn((float)r, P.deltarho));
    if (fabsf(rho) > 0.75f * (float)P.N + 2.0f) return;
    const float intercept = __fdiv_rn(rho, g.cost);
    const Vec<V> *img = g.flat ? xTs : xs;
    const int iend = min(P.half, -P.half + je);
    for (int i = -P.half + jb + lane; i < iend; i += 32) {
        const ExactRow e = fp_row_exact_terms(P.half, g.slope, intercept, g.lbase, i);
        const Vec<V> *row = img + (size_t)(i + P.half) * (P.N + 2) + P.half + 1;
        float b[V], t[V];
#pragma unroll
        for (int j = 0; j < V; ++j) b[j] = t[j] = 0.0f;
        if (e.botin) {
            to_array(__ldg(row + e.xpb), b);
#pragma unroll
            for (int j = 0; j < V; ++j) b[j] = __fmul_rn(e.lbot, b[j]);
        }
        if (e.topin) {
            to_array(__ldg(row + e.xpt), t);
#pragma unroll
            for (int j = 0; j < V; ++j) t[j] = __fmul_rn(e.ltop, t[j]);
        }
#pragma unroll
        for (int j = 0; j < V; ++j) acc[j] = __fadd_rn(acc[j], __fadd_rn(b[j], t[j]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] = __fadd_rn(acc[i], __shfl_xor_sync(0xffffffffu, acc[i], o));
}

// Near-axis rays of the forward phase (a warp per ray, 8 detectors per block,
// kSlotsExact angle slots) and, in slot row 0, the listed corner rays.
template <int V>
__global__ void __launch_bounds__(256) sirt_fp_slices_exact_kernel(SirtProblem q, int slice_base, int it, double tol2,
                                                                   int record_final, int want_e2) {
    __shared__ double she[V][256];
    const int s0 = slice_base + blockIdx.z * V;
    if (it > q.iterations || (it == q.iterations && !record_final)) return;
    const int nexact = __ldg(q.L.counts + 2);
    const int ngraze = graze_count(q);
    if ((int)blockIdx.y >= nexact && (blockIdx.y != 0 || ngraze == 0)) return;
    if (!group_fp_needed<V>(q, s0, it, tol2)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * 8 + warp;
    const size_t np = (size_t)q.P.N * (q.P.N + 2);
    const Vec<V> *xs = group_ptr<V>(q.xpad, s0, np), *xTs = group_ptr<V>(q.xTpad, s0, np);
    double e2[V];
#pragma unroll
    for (int i = 0; i < V; ++i) e2[i] = 0.0;
    float acc[V];
    for (int e = blockIdx.y; e < nexact; e += gridDim.y) {
        const int k = __ldg(q.L.exact + e);
        if (r < q.P.D) {                                   // warp-uniform
            exact_ray_group<V>(q.P, k, r, xs, xTs, 0, q.P.N, acc);
            if (lane == 0) group_residual<V>(q, s0, k, r, acc, want_e2 != 0, e2);
        }
    }
    if (blockIdx.y == 0)
        for (int gidx = blockIdx.x * 8 + warp; gidx < ngraze; gidx += gridDim.x * 8) {
            // graze_ray of sirt.cu for every slice of the group
            int c = 0;
            while (c < 3 && gidx >= __ldg(q.goff + c + 1)) ++c;
            const int slot = c * q.graze_capc + (gidx - __ldg(q.goff + c));
            const int2 ent = __ldg(q.graze + slot);
            const AngleGeom g = load_geom(q.P.geom, ent.x);
            const float rho = __fadd_rn(q.P.rhozero, __fmul_rn((float)ent.y, q.P.deltarho));
            int j0 = 0, j1 = q.P.N;
            lane_rows(q.P, g, ray_x0(g, __fdiv_rn(rho, g.cost)), j0, j1);
            exact_ray_group<V>(q.P, ent.x, ent.y, xs, xTs, j0, j1, acc);
            const size_t pr = (size_t)q.P.a * q.P.D, ray = (size_t)ent.x * q.P.D + ent.y;
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const int s = s0 + i;
                    if (s >= q.nslices) continue;
                    const float e = __fsub_rn(q.b[(size_t)s * pr + ray], acc[i]);
                    q.gcontrib[(size_t)s * 4 * q.graze_capc + slot] =
                        __fmul_rn(__ldg(q.glen + slot), __fmul_rn(-q.R[ray], e));
                    if (want_e2) e2[i] += (double)e * (double)e;
                }
            }
        }
    if (want_e2) group_flush_e2<V>(q, s0, it, e2, she);
}

// Backward phase: a block = a 32 x 32 pixel tile of one slice group, 2 x 2
// pixels per thread, a quarter-warp's lanes 4 x 2 threads.
//   - The tile's detector segment of each angle (at most kSeg entries, zero
//     outside the sinogram) is staged in shared memory, kSub angles at a time,
//     copied asynchronously one step ahead.  A gather from global memory took
//     5.0 L1 cycles (lines crossed by a quarter-warp's 8 lanes); the 4 x 2
//     lanes' entries lie within 8 of each other, so a shared one takes four.
//   - Two pixels next to each other along the axis on which the detector
//     coordinate moves less (|dq| <= sqrt(1/2)) share one window of three
//     detectors: three gathers for two pixels instead of four.  The second pixel's
//     own two are the first two or the last two, and the third gather is whichever
//     of the outer ones it has: a detector outside a pixel's window must not enter
//     it, not even times zero (it may be infinite or NaN).
// Both together took 16 slices x 10 iterations at N=512 / 360 angles from 10.4
// to 9.2 ms against unshared windows gathered from global memory (8.95 since the
// third gather is chosen; two slices took 213 us per iteration with all three added
// and take 217).
// The update x + C*bp and both padded copies are the epilogue.  More than
// kBpChunk angles keep their compensated totals in shared memory between
// chunks.  `first`: block (0,0,0) applies the stopping rule of iteration it.
constexpr int kSeg = 52, kSub = 4;

// Copies entries [0, kSeg) of kSub angles from k0 on (angle k's entry i is
// detector base[k] + i) into seg; angles past the last and detectors outside the row are zero.
template <int V>
__device__ __forceinline__ void stage_segments(const ProbGeom &P, const Vec<V> *__restrict__ rr, const int *base,
                                               int kc, int i0, Vec<V> *seg) {
    for (int t = threadIdx.x; t < kSub * kSeg; t += 256) {
        const int a = t / kSeg, e = t - a * kSeg;
        const int k = kc + i0 + a;
        const int det = k < P.a ? base[i0 + a] + e : -1;
        const bool ok = (unsigned)det < (unsigned)P.D;
        const Vec<V> *src = rr + (ok ? (size_t)k * P.D + det : 0);
        const unsigned dst = (unsigned)__cvta_generic_to_shared(seg + t);
        if (V == 4)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0)
                         : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(ok ? 8 : 0)
                         : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int V>
__device__ __forceinline__ void lds_pairs(unsigned addr, f32x2 (&v)[V / 2]) {
    if constexpr (V == 4)
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "r"(addr));
    else
        asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v[0]) : "r"(addr));
}

template <int V>
__global__ void __launch_bounds__(256, 4) sirt_bp_slices_kernel(SirtProblem q, int slice_base, int it, double tol2,
                                                                int *active, int first) {
    union Shared {
        float2 total[4 * V][256];         // (sum, comp) of a thread's values
        Vec<V> tile[32][33];              // updated pixels, [column][row]
    };
    __shared__ BpStage st;
    __shared__ int base[kBpChunk];        // first staged detector of an angle, centred index + zi
    __shared__ __align__(16) Vec<V> seg[2][kSub * kSeg];
    __shared__ Shared sh;
    __shared__ int any;
    const int s0 = slice_base + blockIdx.z * V;
    if (first && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
        if (threadIdx.x == 0) any = 0;
        __syncthreads();
        int cnt = 0;
        for (int z = threadIdx.x; z < q.nslices; z += blockDim.x) {
            if (bp_needed(tol2, q, z, it)) ++cnt;
            else if (tol2 > 0.0 && it < q.iterations && stop_of(q, z) > it) q.stop_iter[z] = it;
        }
        if (cnt) atomicAdd(&any, cnt);
        __syncthreads();
        if (threadIdx.x == 0) *active = any;
    }
    bool need[V], some = false;
#pragma unroll
    for (int i = 0; i < V; ++i) {
        need[i] = s0 + i < q.nslices && bp_needed(tol2, q, s0 + i, it);
        some |= need[i];
    }
    if (!some) return;                                    // block-uniform
    const ProbGeom &P = q.P;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lx = (lane & 3) + ((lane >> 3) & 1) * 4, ly = ((lane >> 2) & 1) + (lane >> 4) * 2;
    const int cb = (int)blockIdx.x * 32 + (warp & 1) * 16, rb = (int)blockIdx.y * 32 + (warp >> 1) * 8;   // the warp's corner
    const int col0 = cb + 2 * lx, row0 = rb + 2 * ly;
    const float xc0 = (float)(col0 - P.half) + 0.5f, xc1 = xc0 + 1.0f;
    const float yc0 = (float)(row0 - P.half) + 0.5f, yc1 = yc0 + 1.0f;
    const size_t pr = (size_t)P.a * P.D, np = (size_t)P.N * (P.N + 2);
    const Vec<V> *rrv = group_ptr<V>(q.rr, s0, pr);
    constexpr unsigned EB = 4u * V;
    const float fact = fact_f32();
    const float zoff = -P.rz_c - fact;
    const f32x2 mg2 = pk2(kMagic, kMagic), nmg2 = pk2(-kMagic, -kMagic), m1 = pk2(-1.0f, -1.0f);
    const f32x2 nf2 = pk2(-fact, -fact), one2 = pk2(1.0f, 1.0f);
    const f32x2 xc2 = pk2(xc0, xc1), nyc2 = pk2(-yc0, -yc1), zoff2 = pk2(zoff, zoff);
    f32x2 acc[4][V / 2];                                   // pixel 2*j + i: column col0 + i, row row0 + j
    const bool chunks = P.a > kBpChunk;
    // tile centre, for the segments' bases
    const float xm = (float)((int)blockIdx.x * 32 + 16 - P.half), ym = (float)((int)blockIdx.y * 32 + 16 - P.half);
    for (int kc = 0; kc < P.a; kc += kBpChunk) {
        __syncthreads();
        bp_stage(P, kc, st);
        __syncthreads();
        for (int i = threadIdx.x; i < kBpChunk; i += 256) {
            float4 g = st.cs[i];
            if (!(fabsf(g.x) <= 2.0f)) st.cs[i] = g = make_float4(0.0f, 0.0f, -1.0f, 0.0f);   // no finite line: no weight
            // least q of the tile (15.5 pixels to each side of its centre), one below it
            const float qm = fmaf(xm, g.x, fmaf(-ym, g.y, zoff)) - 15.5f * (fabsf(g.x) + fabsf(g.y));
            base[i] = (int)floorf(qm - 0.0625f) + P.zi;
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int p = 0; p < V / 2; ++p) acc[m][p] = pk2(0.0f, 0.0f);
        const int nk = min(kBpChunk, P.a - kc);
        stage_segments<V>(P, rrv, base, kc, 0, seg[0]);
        for (int i0 = 0, buf = 0; i0 < nk; i0 += kSub, buf ^= 1) {
            if (i0 + kSub < nk) {
                stage_segments<V>(P, rrv, base, kc, i0 + kSub, seg[buf ^ 1]);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            const unsigned segb = (unsigned)__cvta_generic_to_shared(seg[buf]);
            const int na = min(kSub, nk - i0);
            for (int a = 0; a < na; ++a) {
                const float4 g = st.cs[i0 + a];
                const float c1 = st.le[i0 + a].y, c2 = c1 - g.w;
                // shared address of entry s (centred index): s*EB + off
                const unsigned off = segb + (unsigned)(a * kSeg + P.zi - base[i0 + a] - kMagicBits) * EB;
                // F, G: the detector coordinates of the pairs' first and second pixels, F <= G
                auto pairs = [&](f32x2 F, f32x2 G, f32x2 (&f0)[V / 2], f32x2 (&g0)[V / 2], f32x2 (&f1)[V / 2],
                                 f32x2 (&g1)[V / 2]) {
                    const f32x2 r = add2_ru(F, mg2);
                    const f32x2 fl = add2(r, nmg2);
                    const f32x2 eF = fma2(F, m1, fl), eG = fma2(G, m1, fl);
                    const f32x2 dG = add2(eG, nf2);
                    const float2 rv = unpk2(r), eFv = unpk2(eF), eGv = unpk2(eG), dFv = unpk2(add2(eF, nf2)),
                                 dGv = unpk2(dG), hGv = unpk2(add2(dG, one2));
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        f32x2(&fa)[V / 2] = o ? f1 : f0;
                        f32x2(&ga)[V / 2] = o ? g1 : g0;
                        const float wF0 = __saturatef(fmaf(-fabsf(o ? dFv.y : dFv.x), g.w, g.z));
                        const float wF1 = __saturatef(fmaf(-(o ? eFv.y : eFv.x), g.w, c1));
                        const float wG0 = __saturatef(fmaf(-fabsf(o ? dGv.y : dGv.x), g.w, g.z));
                        const float wG1 = __saturatef(fmaf(-fabsf(o ? hGv.y : hGv.x), g.w, g.z));
                        const float wG2 = __saturatef(fmaf(-(o ? eGv.y : eGv.x), g.w, c2));
                        const unsigned ad = (unsigned)__float_as_int(o ? rv.y : rv.x) * EB + off;
                        const bool past = (o ? eGv.y : eGv.x) < 0.0f;
                        f32x2 v0[V / 2], v1[V / 2], x[V / 2];
                        lds_pairs<V>(ad, v0);
                        lds_pairs<V>(ad + EB, v1);
                        if constexpr (V == 4) {
                            lds_pairs<V>(past ? ad + 2 * EB : ad, x);
                        } else {                           // few blocks: the address is needed sooner than the value
                            lds_pairs<V>(ad + 2 * EB, x);
                            x[0] = past ? x[0] : v0[0];
                        }
#pragma unroll
                        for (int p = 0; p < V / 2; ++p) {
                            fa[p] = fma2(pk2(wF0, wF0), v0[p], fa[p]);
                            fa[p] = fma2(pk2(wF1, wF1), v1[p], fa[p]);
                        }
                        const float wx = past ? wG2 : wG0;
#pragma unroll
                        for (int p = 0; p < V / 2; ++p) {
                            ga[p] = fma2(pk2(wG1, wG1), v1[p], ga[p]);
                            ga[p] = fma2(pk2(wx, wx), x[p], ga[p]);
                        }
                    }
                };
                if (fabsf(g.x) <= fabsf(g.y)) {            // block-uniform: pairs along x
                    const f32x2 t = fma2(nyc2, pk2(g.y, g.y), zoff2), c = pk2(g.x, g.x);
                    const f32x2 L = fma2(pk2(xc0, xc0), c, t), R = fma2(pk2(xc1, xc1), c, t);
                    if (g.x >= 0.0f) pairs(L, R, acc[0], acc[1], acc[2], acc[3]);
                    else pairs(R, L, acc[1], acc[0], acc[3], acc[2]);
                } else {                                   // pairs along y
                    const float t0 = fmaf(-yc0, g.y, zoff), t1 = fmaf(-yc1, g.y, zoff);
                    const f32x2 c = pk2(g.x, g.x);
                    const f32x2 U = fma2(xc2, c, pk2(t0, t0)), D = fma2(xc2, c, pk2(t1, t1));
                    if (g.y <= 0.0f) pairs(U, D, acc[0], acc[2], acc[1], acc[3]);
                    else pairs(D, U, acc[2], acc[0], acc[3], acc[1]);
                }
            }
            __syncthreads();                               // the buffer is read: the next step overwrites it
        }
        if (chunks) {
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int p = 0; p < V / 2; ++p) {
                    const float2 v = unpk2(acc[m][p]);
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        float2 &tt = sh.total[m * V + 2 * p + o][threadIdx.x];
                        float2 t = kc ? tt : make_float2(0.0f, 0.0f);
                        comp_add(t.x, t.y, o ? v.y : v.x);
                        tt = t;
                    }
                }
        }
    }
    float bpv[4][V];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int p = 0; p < V / 2; ++p) {
            const float2 v = unpk2(acc[m][p]);
            bpv[m][2 * p] = v.x;
            bpv[m][2 * p + 1] = v.y;
            if (chunks)
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    const float2 t = sh.total[m * V + 2 * p + o][threadIdx.x];
                    bpv[m][2 * p + o] = t.x + t.y;
                }
        }
    // near-axis angles, the reference's own expressions (bp_exact_angles)
    const int nexact = __ldg(q.L.counts + 2);
    if (nexact > 0) {
        float ex[4][V];
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int i = 0; i < V; ++i) ex[m][i] = 0.0f;
        for (int e = 0; e < nexact; ++e) {
            const int k = __ldg(q.L.exact + e);
            const AngleGeom g = load_geom(P.geom, k);
            const Vec<V> *srow = rrv + (size_t)k * P.D;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int row = row0 + (m >> 1), col = col0 + (m & 1);
                if (row >= P.N || col >= P.N) continue;
                float a[V];
#pragma unroll
                for (int i = 0; i < V; ++i) a[i] = 0.0f;
                bp_exact_terms(P, g, row, col, [&](int det, float l) {
                    float v[V];
                    to_array(__ldg(srow + det), v);
#pragma unroll
                    for (int i = 0; i < V; ++i) a[i] = __fadd_rn(a[i], __fmul_rn(l, v[i]));
                });
#pragma unroll
                for (int i = 0; i < V; ++i) ex[m][i] += a[i];
            }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int i = 0; i < V; ++i) bpv[m][i] += ex[m][i];
    }
    __syncthreads();                                       // the totals are read: the tile takes their place
    Vec<V> *xs = group_ptr<V>(q.xpad, s0, np), *xTs = group_ptr<V>(q.xTpad, s0, np);
    // the image corners add the terms of the rays that clip only them
    // (warp-uniform tests: the warp that holds the corner pixel sums them)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int crow = c & 2 ? P.N - 1 : 0, ccol = c & 1 ? P.N - 1 : 0;
        if (crow < rb || crow >= rb + 8 || ccol < cb || ccol >= cb + 16) continue;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            if (s0 + i >= q.nslices) continue;
            const float t = corner_terms_warp(q, s0 + i, c);
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (row0 + (m >> 1) == crow && col0 + (m & 1) == ccol) bpv[m][i] = __fadd_rn(bpv[m][i], t);
        }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int row = row0 + (m >> 1), col = col0 + (m & 1);
        float xi[V];
#pragma unroll
        for (int i = 0; i < V; ++i) xi[i] = 0.0f;
        if (row < P.N && col < P.N) {
            const float C = q.C[(size_t)row * P.N + col];
            Vec<V> *xp = xs + (size_t)row * (P.N + 2) + col + 1;
            to_array(*xp, xi);
#pragma unroll
            for (int i = 0; i < V; ++i)
                if (need[i]) xi[i] = __fadd_rn(xi[i], __fmul_rn(C, bpv[m][i]));            // SIRT.fut:38-39
            *xp = to_vec(xi);
        }
        sh.tile[col - blockIdx.x * 32][row - blockIdx.y * 32] = to_vec(xi);
    }
    __syncthreads();
    // transposed write: xTpad[col][row + 1] for the tile's 32 columns x 32 rows
    for (int i = threadIdx.x; i < 1024; i += 256) {
        const int cl = i >> 5, rl = i & 31;
        const int c = blockIdx.x * 32 + cl, r = blockIdx.y * 32 + rl;
        if (c < P.N && r < P.N) xTs[(size_t)c * (P.N + 2) + r + 1] = sh.tile[cl][rl];
    }
}

// xs/xTs of a start image x [nslices][N][N] (the groups are already zero).
template <int V>
__global__ void __launch_bounds__(256) slices_load_kernel(const float *__restrict__ x, float *__restrict__ xs,
                                                          float *__restrict__ xTs, int N, int nslices, int slice_base) {
    __shared__ Vec<V> tile[32][33];
    const int s0 = slice_base + blockIdx.z * V, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const size_t n = (size_t)N * N, np = (size_t)N * (N + 2);
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int y = ty; y < 32; y += 8) {
        const int r = by + y, c = bx + tx;
        if (r < N && c < N) {
            float v[V];
#pragma unroll
            for (int i = 0; i < V; ++i) v[i] = s0 + i < nslices ? x[(size_t)(s0 + i) * n + (size_t)r * N + c] : 0.0f;
            tile[y][tx] = to_vec(v);
            group_ptr<V>(xs, s0, np)[(size_t)r * (N + 2) + c + 1] = to_vec(v);
        }
    }
    __syncthreads();
    for (int y = ty; y < 32; y += 8) {
        const int c = bx + y, r = by + tx;
        if (c < N && r < N) group_ptr<V>(xTs, s0, np)[(size_t)c * (N + 2) + r + 1] = tile[tx][y];
    }
}

template <int V>
__global__ void __launch_bounds__(256) slices_store_kernel(float *__restrict__ xs, float *__restrict__ x, int N,
                                                           int nslices, int slice_base) {
    const int s0 = slice_base + blockIdx.z * V, r = blockIdx.y;
    const size_t n = (size_t)N * N, np = (size_t)N * (N + 2);
    for (int c = blockIdx.x * 256 + threadIdx.x; c < N; c += gridDim.x * 256) {
        float v[V];
        to_array(group_ptr<V>(xs, s0, np)[(size_t)r * (N + 2) + c + 1], v);
#pragma unroll
        for (int i = 0; i < V; ++i)
            if (s0 + i < nslices) x[(size_t)(s0 + i) * n + (size_t)r * N + c] = v[i];
    }
}

template <int V>
cudaError_t fp_slices(const SirtProblem &q, int slice_base, int groups, int it, double tol2, int record_final,
                      int want_e2, cudaStream_t stream) {
    const int S = q.fp_split;
    const dim3 grid((q.P.D + 8 / S - 1) / (8 / S), (q.P.a + 31) / 32 + 2, groups);
    switch (S) {
        case 1: sirt_fp_slices_kernel<1, V><<<grid, 256, 0, stream>>>(q, slice_base, it, tol2, record_final, want_e2); break;
        case 2: sirt_fp_slices_kernel<2, V><<<grid, 256, 0, stream>>>(q, slice_base, it, tol2, record_final, want_e2); break;
        case 4: sirt_fp_slices_kernel<4, V><<<grid, 256, 0, stream>>>(q, slice_base, it, tol2, record_final, want_e2); break;
        default: sirt_fp_slices_kernel<8, V><<<grid, 256, 0, stream>>>(q, slice_base, it, tol2, record_final, want_e2); break;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const dim3 ge((q.P.D + 7) / 8, kSlotsExact, groups);
    sirt_fp_slices_exact_kernel<V><<<ge, 256, 0, stream>>>(q, slice_base, it, tol2, record_final, want_e2);
    return cudaGetLastError();
}

template <int V>
void bp_slices(const SirtProblem &q, int slice_base, int groups, int it, double tol2, int *active, int first,
               cudaStream_t stream) {
    const dim3 grid((q.P.N + 31) / 32, (q.P.N + 31) / 32, groups);
    sirt_bp_slices_kernel<V><<<grid, 256, 0, stream>>>(q, slice_base, it, tol2, active, first);
}

// The stack as groups of four slices and, for one or two left over, a last
// group of two in launches of its own.  While a group of four more fits beside
// the others in one wave of tiles, the rest is such a group: its launch would take
// as long as theirs again (N=160, 360 angles, 10 slices: 254 -> 156 us per iteration).
struct Groups {
    int quads, tail;        // groups of 4; slices left for a group of 2 (0, or 1 and 2)
};
Groups groups_of(int nslices, int N) {
    const int rem = nslices & 3;
    const long long side = (N + 31) / 32;
    Groups g;
    g.quads = nslices / 4;
    g.tail = rem;
    if (rem == 3 || (rem && g.quads && (g.quads + 1) * side * side <= 4LL * device_sms())) {
        ++g.quads;
        g.tail = 0;
    }
    return g;
}

}  // namespace

size_t slices_floats(size_t per_slice, int nslices, int N) {
    const Groups g = groups_of(nslices, N);
    return (4 * (size_t)g.quads + (g.tail ? 2 : 0)) * per_slice + 2 * kGroupPad;
}

bool slices_fit(const ProbGeom &P) {
    // 32-bit byte offsets within a group
    return (double)P.a * P.D * 16.0 < 4294967296.0 && ((double)P.N * (P.N + 2) + 2.0) * 16.0 < 4294967296.0;
}

cudaError_t launch_slices_load(const float *x, float *xs, float *xTs, int N, int nslices, cudaStream_t stream) {
    const Groups g = groups_of(nslices, N);
    const int t = (N + 31) / 32;
    if (g.quads) slices_load_kernel<4><<<dim3(t, t, g.quads), 256, 0, stream>>>(x, xs, xTs, N, nslices, 0);
    if (g.tail) slices_load_kernel<2><<<dim3(t, t, 1), 256, 0, stream>>>(x, xs, xTs, N, nslices, 4 * g.quads);
    return cudaGetLastError();
}

cudaError_t launch_slices_store(float *xs, float *x, int N, int nslices, cudaStream_t stream) {
    const Groups g = groups_of(nslices, N);
    const int t = (N + 255) / 256;
    if (g.quads) slices_store_kernel<4><<<dim3(t, N, g.quads), 256, 0, stream>>>(xs, x, N, nslices, 0);
    if (g.tail) slices_store_kernel<2><<<dim3(t, N, 1), 256, 0, stream>>>(xs, x, N, nslices, 4 * g.quads);
    return cudaGetLastError();
}

cudaError_t launch_sirt_fp_slices(const SirtProblem &q, int it, double tol2, int record_final, int want_e2,
                                  cudaStream_t stream) {
    const Groups g = groups_of(q.nslices, q.P.N);
    cudaError_t e = cudaSuccess;
    if (g.quads) e = fp_slices<4>(q, 0, g.quads, it, tol2, record_final, want_e2, stream);
    if (e == cudaSuccess && g.tail) e = fp_slices<2>(q, 4 * g.quads, 1, it, tol2, record_final, want_e2, stream);
    return e;
}

cudaError_t launch_sirt_bp_slices(const SirtProblem &q, int it, double tol2, int *active, cudaStream_t stream) {
    const Groups g = groups_of(q.nslices, q.P.N);
    if (g.quads) bp_slices<4>(q, 0, g.quads, it, tol2, active, 1, stream);
    if (g.tail) bp_slices<2>(q, 4 * g.quads, 1, it, tol2, active, g.quads == 0, stream);
    return cudaGetLastError();
}

}  // namespace synk
