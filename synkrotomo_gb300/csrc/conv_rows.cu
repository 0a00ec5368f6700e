// 3x3 convolution over long image rows (W a multiple of 128) with every input
// strip read once: forward (bias, ReLU) and backward-data (ReLU mask) of the
// U-Net's wide levels.  BF16 NHWC, FP32 accumulation in TMEM.
//
// A CTA walks down a run of output rows of one 128-pixel column.  The strip of
// one input row (130 pixels, one halo pixel each side, 64 or 32 channels) feeds
// the three output rows it touches, whose accumulators are open in TMEM at the
// same time (a ring of nb buffers of N columns): input row r adds tap row ky=2
// to output row r-1 (which is then complete), ky=1 to r and ky=0 to r+1.  The
// three are one MMA of 3N columns where the ring does not end between them.  Each
// output element still adds its products in the order ky, channel chunk, kx,
// channel, so the results equal those of the tile-by-tile form bit for bit.  The
// weights of all nine taps stay in shared memory for the CTA's lifetime, read
// by TMA straight from the [Cout][9*Cin] layout.
//
//   warp 0      TMA producer of strips        full[s] / empty[s]
//   warp 1      MMA issuer                    tfull[j] / tempty[j]
//   warps 2-9   two epilogue groups of four warps that take turns at the rows;
//               results leave by TMA from a shared tile, and in backward-data
//               the tile first holds the mask (the layer input), loaded by TMA
//               ahead of time and overwritten in place: iofull[j].  One group's
//               chain of waits (accumulator, barrier, TMEM, shared memory, copy)
//               is longer than a row takes to multiply
//
// What bounds it: HBM for the narrow layers (the 32-channel ones move 128 to
// 450 bytes per pixel; 32 -> 32 reaches 0.55 of it), and shared memory, where the
// MMAs read their operands (M=128: 32 cycles for A plus N/4 for B per 16-wide K
// step, and the pipe's N/2 from N=128 on), which is why A is read once for the
// three tap rows.
// Against the tile-by-tile form (a strip per tile and tap row, each strip read
// three times; epilogue stores and mask loads from registers), 8 / 32 images:
// 32 -> 32 at 256 x 256 42 -> 24 / 154 -> 74 us, 96 -> 32 82 -> 42 / 311 -> 139,
// 64 -> 64 at 128 x 128 19 -> 15 / 57 -> 36; backward-data of 32 images 32 -> 96
// 367 -> 167, 32 -> 32 172 -> 100, 64 -> 192 at 128 x 128 190 -> 106.  Of that,
// one MMA for the three tap rows: 32 -> 32 84 -> 74, 96 -> 32 192 -> 139; two
// epilogue groups instead of one: 32 -> 32 109 -> 84.
#include "synk_internal.cuh"
#include "umma.cuh"
#include "umma_gemm.cuh"

namespace synk {
namespace unet {

using namespace umma;

constexpr uint32_t kTiles = 2;   // shared tiles of an epilogue group

struct RowsParams {
    int N, gy, cchunks, H, tiles_w, last_steps;
    int stages, nb, nio, at_once;
    long long rows;                              // B * tiles_w * H output rows of 128 pixels
    uint32_t stage_bytes, strip_tx, w_tx, w_bytes, tap_bytes, io_bytes;
    const float *bias;
    int *err;
    unsigned long long limit_ns;
};

// The output rows [q0, q1) of a CTA, row index (image, column, h), h fastest.
struct RowRun {
    long long q0, q1;
    int n0;
    __device__ __forceinline__ RowRun(const RowsParams &p) {
        const int j = (int)blockIdx.x % p.gy, i = (int)blockIdx.x / p.gy;
        const int cnt = ((int)gridDim.x - j + p.gy - 1) / p.gy;
        q0 = p.rows * i / cnt;
        q1 = p.rows * (i + 1) / cnt;
        n0 = j * p.N;
    }
};
// One part of a run: rows [ha, hb) of column w0 of image b.
struct RowSeg {
    int b, w0, ha, hb;
    __device__ __forceinline__ RowSeg(const RowsParams &p, long long q, long long q1) {
        const long long col = q / p.H;
        ha = (int)(q - col * p.H);
        hb = q1 - q < (long long)(p.H - ha) ? ha + (int)(q1 - q) : p.H;
        b = (int)(col / p.tiles_w);
        w0 = (int)(col - (long long)b * p.tiles_w) * 128;
    }
};
// One row at a time, for the epilogue and its mask copies.
struct RowCursor {
    int b, wt, h;
    long long left;
    __device__ __forceinline__ RowCursor(const RowsParams &p, const RowRun &run) {
        const long long col = run.q0 / p.H;
        h = (int)(run.q0 - col * p.H);
        b = (int)(col / p.tiles_w);
        wt = (int)(col - (long long)b * p.tiles_w);
        left = run.q1 - run.q0;
    }
    __device__ __forceinline__ void next(const RowsParams &p) {
        --left;
        if (++h == p.H) {
            h = 0;
            if (++wt == p.tiles_w) {
                wt = 0;
                ++b;
            }
        }
    }
};

__device__ __forceinline__ bool epi_and(int id, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, %2, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"(v ? 1u : 0u), "r"(id)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void epi_sync(int id) {
    asm volatile("barrier.cta.sync %0, 128;" ::"r"(id) : "memory");
}

__device__ __forceinline__ uint32_t bf2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// One strip (rows of ROW bytes) times the tap rows of c adjacent accumulators of N
// columns from dt on: per kx and K step one MMA of c*N columns, so that the
// strip is read from shared memory once for all of them.  `fresh`: the last
// accumulator is new and its first product overwrites what it held.
template <int ROW>
__device__ __forceinline__ void mma_rows(bool four, uint32_t dt, uint32_t N, uint32_t al, uint32_t bl, uint32_t tap16,
                                         uint32_t hi, uint32_t c, bool fresh) {
    const uint32_t id1 = idesc_bf16(128, 0) | ((N >> 3) << 17), idc = idesc_bf16(128, 0) | ((c * N >> 3) << 17);
    if (fresh) {
        if (c > 1) mma_bf16(dt, al, hi, bl, hi, idc - ((N >> 3) << 17), 1u);
        mma_bf16(dt + (c - 1u) * N, al, hi, bl + (c - 1u) * tap16, hi, id1, 0u);
    } else {
        mma_bf16(dt, al, hi, bl, hi, idc, 1u);
    }
    if (ROW == 128 && four) {
#pragma unroll
        for (uint32_t k = 1; k < 12u; ++k)
            mma_bf16(dt, al + 8u * (k >> 2) + 2u * (k & 3u), hi, bl + 3u * (k >> 2) * tap16 + 2u * (k & 3u), hi, idc, 1u);
    } else {
#pragma unroll
        for (uint32_t k = 1; k < 6u; ++k)
            mma_bf16(dt, al + (ROW / 16u) * (k >> 1) + 2u * (k & 1u), hi, bl + 3u * (k >> 1) * tap16 + 2u * (k & 1u), hi,
                     idc, 1u);
    }
}

// EPI: EPI_BIAS_RELU, EPI_BIAS or EPI_MASK.  CW: channels per strip (64, or 32
// for 32-channel inputs: 64-byte rows, half the shared memory and copy work).
template <int EPI, int CW>
__global__ void __launch_bounds__(320, 1) conv_rows_kernel(const __grid_constant__ CUtensorMap tmX,
                                                           const __grid_constant__ CUtensorMap tmW,
                                                           const __grid_constant__ CUtensorMap tmY,
                                                           const __grid_constant__ CUtensorMap tmM,
                                                           const RowsParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    const int S = p.stages;
    uint8_t *wres = smem + (size_t)S * p.stage_bytes;
    uint8_t *io = wres + p.w_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(io + (size_t)p.nio * p.io_bytes);
    uint64_t *empty = full + S;
    uint64_t *tfull = empty + S;
    uint64_t *tempty = tfull + p.nb;
    uint64_t *iofull = tempty + p.nb;
    uint64_t *wfull = iofull + p.nio;
    uint64_t *drain = wfull + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
    float *sbias = reinterpret_cast<float *>(tmem_slot + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const RowRun run(p);
    if (warp == 0) {
        tmem_alloc(tmem_slot, 512u);
        tmem_relinquish();
    }
    if (warp == 1 && lane == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int j = 0; j < p.nb; ++j) {
            mbar_init(&tfull[j], 1);
            mbar_init(&tempty[j], 4);
        }
        for (int j = 0; j < p.nio; ++j) mbar_init(&iofull[j], 1);
        mbar_init(wfull, 1);
        mbar_init(drain, 1);
        fence_mbar_init();
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmX);
        tma_prefetch_desc(&tmW);
        tma_prefetch_desc(&tmY);
        if (EPI == EPI_MASK) tma_prefetch_desc(&tmM);
    }
    if (EPI != EPI_MASK)
        for (int i = threadIdx.x; i < p.N; i += blockDim.x) sbias[i] = p.bias[run.n0 + i];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---- producer ----
        if (elect_one()) {
            mbar_arrive_expect_tx(wfull, p.w_tx);
            // [chunk][kx][ky = 2, 1, 0][n tile]: for one kx the tap rows stand in the order
            // of the accumulators that one strip adds to
            for (int cc = 0; cc < p.cchunks; ++cc)
                for (int tap = 0; tap < 9; ++tap)
                    tma_load_3d(wres + (size_t)(cc * 9 + (tap % 3) * 3 + 2 - tap / 3) * p.tap_bytes, &tmW, wfull,
                                cc * CW, run.n0, tap);
        }
        __syncwarp();
        uint32_t s = 0, ph = 1, used = 0;
        bool fail = false;
        for (long long q = run.q0; q < run.q1 && !fail;) {
            const RowSeg g(p, q, run.q1);
            for (int r = g.ha - 1; r <= g.hb && !fail; ++r)
                for (int cc = 0; cc < p.cchunks; ++cc) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ph, p.err, p.limit_ns))) {
                        fail = true;
                        break;
                    }
                    if (elect_one()) {
                        // rows -1 and H and pixels -1 and W are out of bounds and read as 0
                        mbar_arrive_expect_tx(&full[s], p.strip_tx);
                        tma_load_4d(smem + (size_t)s * p.stage_bytes, &tmX, &full[s], cc * CW, g.w0 - 1, r, g.b);
                    }
                    __syncwarp();
                    if (used < (uint32_t)S) ++used;
                    if (++s == (uint32_t)S) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            q += g.hb - g.ha;
        }
        // no copy may still be landing when the CTA exits
        for (uint32_t c = 0; c < used; ++c) mbar_drain(&full[c], c < s ? ph ^ 1u : ph, p.limit_ns);
        mbar_drain(wfull, 0u, p.limit_ns);
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer ----
        const uint32_t hi = smem_desc_hi(2 * CW);
        const uint32_t base = smem_u32(smem), w0 = smem_u32(wres);
        const uint32_t nb = (uint32_t)p.nb;
        uint32_t s = 0, ph = 0;
        uint32_t oslot = 0, ophase = 1;   // the next row to open: its buffer, the parity of the buffer's last release
        uint32_t cslot = 0;               // the next row to complete
        bool fail = !__all_sync(0xffffffffu, mbar_wait(wfull, 0u, p.err, p.limit_ns));
        for (long long q = run.q0; q < run.q1 && !fail;) {
            const RowSeg g(p, q, run.q1);
            for (int r = g.ha - 1; r <= g.hb && !fail; ++r) {
                // output rows r+lo .. r+up (ky = 1-lo .. 1-up) take this strip; the first of
                // them is in cslot, the last, if r+1, is a new one in oslot
                const int lo = r > g.ha ? -1 : g.ha - r, up = r + 1 < g.hb ? 1 : g.hb - 1 - r;
                const bool opens = up == 1, closes = lo == -1;
                if (opens) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&tempty[oslot], ophase, p.err, p.limit_ns))) {
                        fail = true;
                        break;
                    }
                    if (++oslot == nb) {
                        oslot = 0;
                        ophase ^= 1u;
                    }
                }
                for (int cc = 0; cc < p.cchunks; ++cc) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&full[s], ph, p.err, p.limit_ns))) {
                        fail = true;
                        break;
                    }
                    tc_fence_after();
                    if (elect_one()) {
                        const bool four = CW == 64 && (cc + 1 < p.cchunks || p.last_steps == 4);
                        const uint32_t al = smem_desc_lo(base + s * p.stage_bytes);
                        const uint32_t tap16 = p.tap_bytes >> 4;
                        uint32_t bl = smem_desc_lo(w0 + (uint32_t)cc * 9u * p.tap_bytes) + (uint32_t)(lo + 1) * tap16;
                        uint32_t slot = cslot;
                        // as many adjacent accumulators per MMA as N <= 256 and the ring's end allow
                        for (int left = up - lo + 1; left > 0;) {
                            const uint32_t c = min((uint32_t)min(left, p.at_once), nb - slot);
                            left -= (int)c;
                            mma_rows<2 * CW>(four, tmem + slot * (uint32_t)p.N, (uint32_t)p.N, al, bl, tap16, hi, c,
                                             opens && cc == 0 && left == 0);
                            bl += c * tap16;
                            slot += c;
                            if (slot == nb) slot = 0;
                        }
                        mma_commit(&empty[s]);
                        if (closes && cc + 1 == p.cchunks) mma_commit(&tfull[cslot]);
                    }
                    __syncwarp();
                    if (++s == (uint32_t)S) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                if (closes && ++cslot == nb) cslot = 0;
            }
            q += g.hb - g.ha;
        }
        // every issued MMA has completed before TMEM is freed
        if (elect_one()) {
            mma_commit(drain);
            mbar_drain(drain, 0u, p.limit_ns);
        }
        __syncwarp();
    } else {
        // ---- epilogue: TMEM lanes 32*(warp % 4) .. +31 are pixels of the row ----
        const int q4 = warp & 3;
        const int row = q4 * 32 + lane;
        const uint32_t nb = (uint32_t)p.nb;
        const uint32_t rsw = (uint32_t)((row >> 1) & 3);
        const int grp = (warp - 2) >> 2, bar = 1 + grp;          // the group takes rows grp, grp + 2, ...
        const bool mover = ((warp - 2) & 3) == 0 && elect_one();   // issues the group's copies
        uint8_t *gio = io + (size_t)grp * kTiles * p.io_bytes;
        uint64_t *gfull = iofull + grp * kTiles;
        RowCursor cur(p, run);
        if (grp) cur.next(p);
        RowCursor ahead = cur;
        uint32_t loads = 0;                            // mask tiles requested (mover only)
        auto load_mask = [&]() {
            const uint32_t j = loads % kTiles;
            mbar_arrive_expect_tx(&gfull[j], p.io_bytes);
            for (int c = 0; c < p.N / 32; ++c)
                tma_load_4d(gio + (size_t)j * p.io_bytes + (size_t)c * 8192u, &tmM, &gfull[j], run.n0 + 32 * c,
                            ahead.wt * 128, ahead.h, ahead.b);
            ++loads;
            ahead.next(p);
            ahead.next(p);
        };
        if (EPI == EPI_MASK && mover)
            for (uint32_t k = 0; k + 1 < kTiles && ahead.left > 0; ++k) load_mask();
        uint32_t slot = (uint32_t)grp, sph = 0;        // the row's accumulator and its phase
        uint32_t j = 0, jph = 0;                       // its shared tile and that tile's phase
        for (; cur.left > 0; cur.next(p), cur.next(p)) {
            bool ok = mbar_wait(&tfull[slot], sph, p.err, p.limit_ns);
            if (EPI == EPI_MASK) {
                ok = ok && mbar_wait(&gfull[j], jph, p.err, p.limit_ns);
            } else if (mover) {
                bulk_wait_read<kTiles - 1>();          // the store that last read this tile is done
            }
            // one decision for the four warps (an accumulator is only ever signalled whole:
            // the error word needs no look here, a trip to L2 per row)
            if (!epi_and(bar, ok)) break;
            __syncwarp();                              // the lanes leave the waits one by one, TMEM is read together
            tc_fence_after();
            uint8_t *tile = gio + (size_t)j * p.io_bytes;
            const uint32_t tbase = tmem + slot * (uint32_t)p.N + ((uint32_t)(q4 * 32) << 16);
            for (int c0 = 0; c0 < p.N; c0 += 32) {
                float v[32];
                tmem_ld_32x32(tbase + (uint32_t)c0, v);
                uint4 *o = reinterpret_cast<uint4 *>(tile + (size_t)(c0 >> 5) * 8192u + (size_t)row * 64u);
#pragma unroll
                for (uint32_t c = 0; c < 4u; ++c) {
                    uint4 *oc = o + (c ^ rsw);
                    uint32_t w[4];
                    if (EPI == EPI_MASK) {
                        const uint4 m = *oc;
                        w[0] = m.x;
                        w[1] = m.y;
                        w[2] = m.z;
                        w[3] = m.w;
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float x0 = v[8 * c + 2 * e], x1 = v[8 * c + 2 * e + 1];
                        if (EPI == EPI_MASK) {
                            // the bits of a positive BF16 number (or infinity)
                            const uint32_t m0 = w[e] & 0xffffu, m1 = w[e] >> 16;
                            x0 = m0 - 1u < 0x7f80u ? x0 : 0.0f;
                            x1 = m1 - 1u < 0x7f80u ? x1 : 0.0f;
                        } else {
                            x0 += sbias[c0 + 8 * c + 2 * e];
                            x1 += sbias[c0 + 8 * c + 2 * e + 1];
                            if (EPI == EPI_BIAS_RELU) {
                                x0 = fmaxf(x0, 0.0f);
                                x1 = fmaxf(x1, 0.0f);
                            }
                        }
                        w[e] = bf2(x0, x1);
                    }
                    *oc = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            // this warp's reads of the accumulator are complete
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[slot]);
            fence_async_shared();
            epi_sync(bar);
            if (mover) {
                for (int c = 0; c < p.N / 32; ++c)
                    tma_store_4d(&tmY, tile + (size_t)c * 8192u, run.n0 + 32 * c, cur.wt * 128, cur.h, cur.b);
                bulk_commit();
                if (EPI == EPI_MASK && ahead.left > 0) {
                    bulk_wait_read<1>();               // the store before this one has left its tile
                    load_mask();
                }
            }
            __syncwarp();
            slot += 2;
            if (slot >= nb) {
                slot -= nb;
                sph ^= 1u;
            }
            if (++j == kTiles) {
                j = 0;
                jph ^= 1u;
            }
        }
        if (mover) {
            bulk_wait_all();
            if (EPI == EPI_MASK)   // no copy may still be landing (only after a failure is one in flight)
                for (uint32_t k = loads > kTiles ? loads - kTiles : 0u; k < loads; ++k)
                    mbar_drain(&gfull[k % kTiles], (k / kTiles) & 1u, p.limit_ns);
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512u);
    }
}

static uint32_t kb1(size_t b) { return (uint32_t)((b + 1023) / 1024 * 1024); }

// The split of a layer over n tiles, shared memory and TMEM; false where the
// weights of all taps do not fit beside two strips and two tiles.
static bool rows_plan(const ConvArgs &c, int epi, RowsParams &p, size_t *smem) {
    if (c.W % 128 || c.Cin % 32 || c.Cout % 32) return false;
    const int cw = c.Cin == 32 ? 32 : 64;
    p.cchunks = (c.Cin + cw - 1) / cw;
    p.last_steps = (c.Cin - cw * (p.cchunks - 1)) / 16;
    p.stage_bytes = kb1(130u * 2 * cw);
    p.strip_tx = 130u * 2 * cw;
    p.nio = 2 * (int)kTiles;
    // the widest n tile of at most 128 columns (four accumulators open at a time in 512)
    // that divides Cout and leaves room; below 64 the MMAs cost more than the copies save
    for (int n = c.Cout <= 128 ? c.Cout : 128; n >= (c.Cout < 64 ? 32 : 64); n -= 32) {
        if (c.Cout % n) continue;
        p.N = n;
        p.gy = c.Cout / n;
        p.tap_bytes = (uint32_t)(n * 2 * cw);
        p.w_bytes = p.w_tx = p.cchunks * 9u * p.tap_bytes;
        p.io_bytes = (uint32_t)n * 256u;
        const size_t fixed = 1024 + p.w_bytes + (size_t)p.nio * p.io_bytes + 8 * (2 * 8 + 2 * 16 + 2 * kTiles + 2) + 16 + 4 * (size_t)n;
        const size_t room = 227u * 1024u;
        if (fixed + 3 * (size_t)p.stage_bytes > room) continue;
        const size_t s = (room - fixed) / p.stage_bytes;
        p.stages = s > 8 ? 8 : (int)s;
        p.nb = 512 / n;   // 16, 8, 5 or 4 accumulators in all of TMEM
        p.at_once = 256 / n < 3 ? 256 / n : 3;
        *smem = fixed + (size_t)p.stages * p.stage_bytes;
        return true;
    }
    return false;
}

template <int EPI, int CW>
static cudaError_t rows_launch(const CUtensorMap &x, const CUtensorMap &w, const CUtensorMap &y, const CUtensorMap &m,
                               const RowsParams &p, size_t smem, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(conv_rows_kernel<EPI, CW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    const long long most = p.rows * p.gy;
    const int sms = device_sms();
    conv_rows_kernel<EPI, CW><<<(unsigned)(most < sms ? most : sms), 320, smem, st>>>(x, w, y, m, p);
    return cudaGetLastError();
}

bool conv_rows_fits(const ConvArgs &c, int epi) {
    RowsParams p = {};
    size_t smem = 0;
    return rows_plan(c, epi, p, &smem);
}

cudaError_t conv_rows(const ConvArgs &c, int epi, int *err, unsigned long long limit_ns, cudaStream_t st) {
    RowsParams p = {};
    size_t smem = 0;
    if (!rows_plan(c, epi, p, &smem) || device_sms() < p.gy) return cudaErrorInvalidValue;
    p.H = c.H;
    p.tiles_w = c.W / 128;
    p.rows = (long long)c.B * p.tiles_w * c.H;
    if (p.rows == 0) return cudaSuccess;
    p.bias = c.bias;
    p.err = err;
    p.limit_ns = limit_ns;
    const int cw = c.Cin == 32 ? 32 : 64;
    auto image = [&](CUtensorMap *m, const uint16_t *q, int ch, long long ld, uint32_t bc, uint32_t bp) {
        const uint64_t d[4] = {(uint64_t)ch, (uint64_t)c.W, (uint64_t)c.H, (uint64_t)c.B};
        const uint64_t s[3] = {(uint64_t)ld * 2, (uint64_t)ld * 2 * c.W, (uint64_t)ld * 2 * c.W * c.H};
        const uint32_t b[4] = {bc, bp, 1, 1};
        return tensor_map(m, q, 4, d, s, b, (int)(2 * bc));
    };
    // w[o][tap*Cin + i] as (i, o, tap), a box per channel chunk and tap
    const uint64_t dw[3] = {(uint64_t)c.Cin, (uint64_t)c.Cout, 9};
    const uint64_t sw[2] = {(uint64_t)c.Cin * 18, (uint64_t)c.Cin * 2};
    const uint32_t bw[3] = {(uint32_t)cw, (uint32_t)p.N, 1};
    CUtensorMap tx, tw, ty, tm;
    cudaError_t e;
    if ((e = image(&tx, c.x + c.xoff, c.Cin, c.ldx, (uint32_t)cw, 130)) != cudaSuccess) return e;
    if ((e = tensor_map(&tw, c.w, 3, dw, sw, bw, 2 * cw)) != cudaSuccess) return e;
    if ((e = image(&ty, c.y + c.yoff, c.Cout, c.ldy, 32, 128)) != cudaSuccess) return e;
    tm = ty;
    if (epi == EPI_MASK && (e = image(&tm, c.mask + c.moff, c.Cout, c.ldm, 32, 128)) != cudaSuccess) return e;
    switch (epi) {
        case EPI_BIAS_RELU:
            return cw == 32 ? rows_launch<EPI_BIAS_RELU, 32>(tx, tw, ty, tm, p, smem, st)
                            : rows_launch<EPI_BIAS_RELU, 64>(tx, tw, ty, tm, p, smem, st);
        case EPI_BIAS:
            return cw == 32 ? rows_launch<EPI_BIAS, 32>(tx, tw, ty, tm, p, smem, st)
                            : rows_launch<EPI_BIAS, 64>(tx, tw, ty, tm, p, smem, st);
        case EPI_MASK:
            return cw == 32 ? rows_launch<EPI_MASK, 32>(tx, tw, ty, tm, p, smem, st)
                            : rows_launch<EPI_MASK, 64>(tx, tw, ty, tm, p, smem, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace unet
}  // namespace synk
