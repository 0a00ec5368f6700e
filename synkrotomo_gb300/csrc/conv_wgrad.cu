// Weight and bias gradients of the U-Net's 3x3 convolutions, straight from the
// NHWC activations: dw[o][ky*3+kx][i] += sum_p dz[p][o] * x[p + (ky-1, kx-1)][i],
// db[o] += sum_p dz[p][o].
//
// The contraction runs over pixels, so both operands are MN-major: a shared
// memory row is one pixel, its 64 (or 32) channels the contiguous dimension, as
// TMA delivers it.  A CTA keeps all nine taps of a block of CI input by CO output
// channels in TMEM and walks down rows of one column of PX pixels:
//   A (M = 128) one strip of input row r, PX + 2 pixels; the taps kx are atoms of
//               CI channels one pixel row further each (leading dimension offset =
//               one row): 4 atoms of 32 channels (three used) or 2 of 64 (kx 0
//               and 1, then kx 2; the fourth is not used)
//   B (N = 3CO) the strips of gradient rows r-1, r, r+1 (ky = 2, 1, 0), neighbours
//               in a ring of strips: atoms one strip apart
// so a strip of either is read from memory once per block and one MMA does 16
// pixels of up to nine taps.  The bias sums are taken from the same strips in
// shared memory by the warps that later drain the accumulators (FP32 atomics, 32
// consecutive input channels per instruction).  Pixel rows are split over CTAs.
//
// What bounds it: HBM in the 32 -> 32 layer (273 MB in 59 us, 0.68 of the copy rate);
// elsewhere the issuing warp (about 500 cycles per stage for its wait and commit, 35
// to 48 per MMA) next to the MMA rate (M=128, N=192: 96 cycles; N=96: 56), and at one
// image the drain, 10 us of atomics.
// Against copies of both operands in a channel-major layout (x three times, shifted
// by kx), one tap per CTA, and a kernel for the bias, 32 images: 32 -> 32 at
// 256 x 256 448 -> 57 us, 96 -> 32 790 -> 156, 192 -> 64 at 128 x 128 396 -> 98,
// 384 -> 128 at 64 x 64 237 -> 104, 256 -> 256 at 32 x 32 113 -> 46; the training
// step 5.98 -> 3.26 ms.  One row per stage with a barrier per operand and ring:
// 384 -> 128 149, 256 -> 256 83.
#include "synk_internal.cuh"
#include "umma.cuh"
#include "umma_gemm.cuh"

namespace synk {
namespace unet {

using namespace umma;

struct DwParams {
    int Cin, Cout, H, tiles_w, nci, nco, nc, splits, turns, stages;
    long long rows;                    // B * tiles_w * H rows of one strip's width
    uint32_t x_bytes, x_tx, z_tx;      // of one input block's rows in a stage; what a stage's copies bring
    float *dw, *db;
    int *err;
    unsigned long long limit_ns;
};

// Rows [ha, hb) of one column: a part of a CTA's run.
struct DwSeg {
    int b, w0, ha, hb, steps;
    template <int PX, int R>
    static __device__ __forceinline__ DwSeg at(const DwParams &p, long long q, long long q1) {
        DwSeg g;
        const long long col = q / p.H;
        g.ha = (int)(q - col * p.H);
        g.hb = q1 - q < (long long)(p.H - g.ha) ? g.ha + (int)(q1 - q) : p.H;
        g.b = (int)(col / p.tiles_w);
        g.w0 = (int)(col - (long long)g.b * p.tiles_w) * PX;
        g.steps = (g.hb - g.ha + 2 + R - 1) / R;   // input rows ha-1 .. hb, R per step
        return g;
    }
};

__device__ __forceinline__ void tmem_zero32(uint32_t taddr) {
    asm volatile(
        "{\n\t.reg .b32 z;\n\tmov.b32 z, 0;\n\t"
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {z, z, z, z, z, z, z, z, z, z, z, z, z, z, z, z, "
        "z, z, z, z, z, z, z, z, z, z, z, z, z, z, z, z};\n\t}" ::"r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// MN-major descriptor, low half: start address and leading-dimension offset
// (from one atom of 64 or 32 channels to the next).  The stride-dimension offset
// of the high half is that from 8 pixel rows to the next 8.
__device__ __forceinline__ uint32_t desc_lo_mn(uint32_t saddr, uint32_t lead_bytes) {
    return ((saddr & 0x3FFFFu) >> 4) | ((lead_bytes >> 4) << 16);
}

// KS: K steps of 16 pixels per row (strips of 16 KS pixels); R: image rows per stage.
template <int CI, int CO, int KS, int R>
__global__ void __launch_bounds__(192, 1) conv_wgrad_kernel(const __grid_constant__ CUtensorMap tmX,
                                                            const __grid_constant__ CUtensorMap tmZ, const DwParams p) {
    constexpr int PX = 16 * KS;
    constexpr uint32_t kRowX = 2 * CI, kRowZ = 2 * CO;   // bytes of one pixel
    constexpr uint32_t kStripX = (PX + 2) * kRowX, kStripZ = PX * kRowZ;
    constexpr uint32_t kM = CI == 64 ? 2 : 1;            // MMAs of M = 128 that hold the three taps kx
    constexpr int kLate = (2 + R - 1) / R;               // steps for which a gradient row is used again
    extern __shared__ uint8_t smem_raw[];
    __shared__ float sdb[4][CO];                         // the warps' bias sums
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *zs = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    const int S = p.stages;
    uint8_t *xs = zs + (size_t)S * R * kStripZ;
    const uint32_t x_stage = (uint32_t)p.nc * p.x_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(xs + (size_t)S * x_stage);
    uint64_t *done = full + S;
    uint64_t *tfull = done + S;
    uint64_t *tempty = tfull + 1;
    uint64_t *drain = tempty + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // block of channels (fastest: CTAs of one part of the rows run together) and rows
    const int nblk = p.nci * p.nco;
    const int blk = (int)blockIdx.x % nblk, part = (int)blockIdx.x / nblk;
    const int ci0 = (blk % p.nci) * p.nc * CI, co0 = (blk / p.nci) * CO;
    const bool bias = blk % p.nci == 0;
    const long long q0 = p.rows * part / p.splits, len = p.rows * (part + 1) / p.splits - q0;
    if (warp == 0) {
        tmem_alloc(tmem_slot, 512u);
        tmem_relinquish();
    }
    if (warp == 1 && lane == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&done[s], bias ? 5 : 1);   // the step's MMAs, and the four warps of the bias
        }
        mbar_init(tfull, 1);
        mbar_init(tempty, 4);
        mbar_init(drain, 1);
        fence_mbar_init();
        tma_prefetch_desc(&tmX);
        tma_prefetch_desc(&tmZ);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    constexpr uint32_t kCols = kM * 3u * CO;   // of one input block
    if (warp >= 2) {
        for (uint32_t c = 0; c < (uint32_t)p.nc * kCols; c += 32u)
            tmem_zero32(tmem + c + ((uint32_t)((warp & 3) * 32) << 16));
        tmem_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    if (warp == 0) {
        // ---- producer: step i brings input rows r .. r+R-1 and gradient rows r+1 .. r+R,
        // which the next kLate steps use again: its stage is free when step i + kLate is done ----
        uint32_t s = 0, used = 0, ph = 0;   // stage; stages filled at least once; parity of this round's "full"
        uint32_t ws = 0, wph = 0;           // the step to wait for
        bool fail = false;
        for (int t = 0; t < p.turns; ++t)
            for (long long q = q0 + len * t / p.turns, q1 = q0 + len * (t + 1) / p.turns; q < q1 && !fail;) {
                const DwSeg g = DwSeg::at<PX, R>(p, q, q1);
                for (int i = 0; i < g.steps; ++i) {
                    if (used == (uint32_t)S) {   // the stage was filled before
                        // step (this one - S + kLate)
                        if (!__all_sync(0xffffffffu, mbar_wait(&done[ws], wph, p.err, p.limit_ns))) {
                            fail = true;
                            break;
                        }
                        if (++ws == (uint32_t)S) {
                            ws = 0;
                            wph ^= 1u;
                        }
                    }
                    if (elect_one()) {
                        const int r = g.ha - 1 + i * R;
                        const bool z = r + 1 < g.hb;
                        // rows and pixels outside the image read as 0
                        mbar_arrive_expect_tx(&full[s], (uint32_t)p.nc * p.x_tx + (z ? p.z_tx : 0u));
                        if (z) tma_load_4d(zs + (size_t)s * R * kStripZ, &tmZ, &full[s], co0, g.w0, r + 1, g.b);
                        for (int c = 0; c < p.nc; ++c)
                            tma_load_4d(xs + (size_t)s * x_stage + (size_t)c * p.x_bytes, &tmX, &full[s], ci0 + c * CI,
                                        g.w0 - 1, r, g.b);
                    }
                    __syncwarp();
                    if (used < (uint32_t)S && ++used == (uint32_t)S) {
                        ws = (uint32_t)kLate;   // the first wait is for step kLate
                        wph = 0;
                    }
                    if (++s == (uint32_t)S) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                q += g.hb - g.ha;
            }
        // no copy may still be landing when the CTA exits: stages below s were last
        // filled in this round, the others in the one before
        for (uint32_t c = 0; c < used; ++c) mbar_drain(&full[c], c < s ? ph : ph ^ 1u, p.limit_ns);
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer ----
        const uint32_t xhi = smem_desc_hi(kRowX), zhi = smem_desc_hi(kRowZ);
        const uint32_t x0 = smem_u32(xs), z0 = smem_u32(zs);
        const uint32_t id1 = idesc_bf16(128, 0) | (3u << 15);   // both operands MN-major
        const uint32_t zrows = (uint32_t)(S * R);
        uint32_t s = 0, ph = 0;
        bool fail = false;
        for (int t = 0; t < p.turns && !fail; ++t) {
            if (t > 0) {
                if (!__all_sync(0xffffffffu, mbar_wait(tempty, (uint32_t)(t - 1) & 1u, p.err, p.limit_ns))) break;
                tc_fence_after();
            }
            const long long q1 = q0 + len * (t + 1) / p.turns;
            for (long long q = q0 + len * t / p.turns; q < q1 && !fail;) {
                const DwSeg g = DwSeg::at<PX, R>(p, q, q1);
                uint32_t zsl = s * R;   // ring slot of the first gradient row that meets input row r
                for (int i = 0; i < g.steps; ++i) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&full[s], ph, p.err, p.limit_ns))) {
                        fail = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t xa = x0 + s * x_stage;
#pragma unroll
                    for (int j = 0; j < R; ++j) {
                        // gradient rows r+lo .. r+up (ky = 1-lo .. 1-up) meet input row r
                        const int r = g.ha - 1 + i * R + j;
                        const int lo = r > g.ha ? -1 : g.ha - r, up = r + 1 < g.hb ? 1 : g.hb - 1 - r;
                        if (lo > up) continue;   // past the last row
                        if (elect_one()) {
                            for (int c = 0; c < p.nc; ++c) {
                                const uint32_t al = desc_lo_mn(xa + (uint32_t)c * p.x_bytes + (uint32_t)j * kStripX, kRowX);
                                uint32_t slot = zsl, d = tmem + (uint32_t)c * kCols + (uint32_t)(lo + 1) * CO;
                                for (int left = up - lo + 1; left > 0;) {
                                    // neighbours in the ring, up to its end
                                    const uint32_t n = min((uint32_t)left, zrows - slot);
                                    const uint32_t idn = id1 | ((n * CO >> 3) << 17);
                                    const uint32_t bl = desc_lo_mn(z0 + slot * kStripZ, kStripZ);
#pragma unroll
                                    for (uint32_t k = 0; k < (uint32_t)KS; ++k) {
                                        mma_bf16(d, al + k * kRowX, xhi, bl + k * kRowZ, zhi, idn, 1u);
                                        if (CI == 64)
                                            mma_bf16(d + 3u * CO, al + k * kRowX + 2u * (kRowX / 16u), xhi,
                                                     bl + k * kRowZ, zhi, idn, 1u);
                                    }
                                    left -= (int)n;
                                    d += n * CO;
                                    slot += n;
                                    if (slot == zrows) slot = 0;
                                }
                            }
                        }
                        __syncwarp();
                        if (lo == -1 && ++zsl == zrows) zsl = 0;
                    }
                    if (elect_one()) mma_commit(&done[s]);
                    __syncwarp();
                    if (++s == (uint32_t)S) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                q += g.hb - g.ha;
            }
            if (!fail && elect_one()) mma_commit(tfull);   // the sums are signalled only whole
            __syncwarp();
        }
        // every issued MMA has completed before TMEM is freed
        if (elect_one()) {
            mma_commit(drain);
            mbar_drain(drain, 0u, p.limit_ns);
        }
        __syncwarp();
    } else {
        // ---- bias sums while the rows pass, then the accumulators, turn by turn ----
        const int q4 = warp & 3;
        const uint32_t tl = tmem + ((uint32_t)(q4 * 32) << 16);
        // bias: lane = (pixel, 8 channels); a warp takes a quarter of a strip's pixels
        constexpr uint32_t kG = CO / 8, kStep = 32 / kG;
        const uint32_t c = (uint32_t)lane % kG, r0 = (uint32_t)lane / kG;
        constexpr uint32_t kPer = PX / 4u;
        float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        uint32_t s = 0, ph = 0;
        bool ok = true;
        for (int t = 0; t < p.turns && ok; ++t) {
            const long long q1 = q0 + len * (t + 1) / p.turns;
            for (long long q = bias ? q0 + len * t / p.turns : q1; q < q1 && ok;) {
                const DwSeg g = DwSeg::at<PX, R>(p, q, q1);
                for (int i = 0; i < g.steps; ++i) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&full[s], ph, p.err, p.limit_ns));
                    if (!ok) break;
                    const int rows = min(R, g.hb - g.ha - i * R);   // gradient rows of this step
                    for (int j = 0; j < rows; ++j) {
                        const uint8_t *z = zs + (size_t)(s * R + (uint32_t)j) * kStripZ;
                        float u8[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                        for (uint32_t k = 0; k < kPer; k += kStep) {
                            const uint32_t row = (uint32_t)q4 * kPer + k + r0;
                            const uint32_t sw = CO == 64 ? row & 7u : (row >> 1) & 3u;
                            const uint4 u = *reinterpret_cast<const uint4 *>(z + row * kRowZ + ((c ^ sw) << 4));
                            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                u8[2 * e] += __uint_as_float(w[e] << 16);
                                u8[2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u);
                            }
                        }
#pragma unroll
                        for (int e = 0; e < 8; ++e) acc[e] += u8[e];
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&done[s]);
                    if (++s == (uint32_t)S) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                q += g.hb - g.ha;
            }
            ok = __all_sync(0xffffffffu, ok && mbar_wait(tfull, (uint32_t)t & 1u, p.err, p.limit_ns));
            if (!ok) break;
            tc_fence_after();
            for (uint32_t cm = 0; cm < (uint32_t)p.nc * kM; ++cm) {   // input block and its MMA
                const int m = q4 * 32 + lane;
                const int kx = CI == 64 ? (int)(cm % kM) * 2 + m / 64 : m / 32;   // uniform over the warp
                if (kx > 2) continue;
                float *o = p.dw + (long long)co0 * 9 * p.Cin + kx * p.Cin + ci0 + (int)(cm / kM) * CI + m % CI;
                // groups of 8 columns, each CTA from another one on: in step, all CTAs would
                // queue at one address after the other
                constexpr uint32_t kGroups = 3u * CO / 8u;
                uint32_t g = (uint32_t)part % kGroups;
                for (uint32_t k = 0; k < kGroups; ++k) {
                    float v[8];
                    tmem_ld_32x8(tl + cm * 3u * CO + 8u * g, v);
                    const uint32_t ky = 2u - 8u * g / CO, oc = 8u * g % CO;
                    float *on = o + (long long)oc * 9 * p.Cin + (long long)ky * 3 * p.Cin;
#pragma unroll
                    for (int j = 0; j < 8; ++j) atomicAdd(on + (long long)j * 9 * p.Cin, v[j]);
                    if (++g == kGroups) g = 0;
                }
            }
            if (t + 1 < p.turns) {
                for (uint32_t k = 0; k < (uint32_t)p.nc * kCols; k += 32u) tmem_zero32(tl + k);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty);
            }
        }
        if (bias) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float a = ok ? acc[e] : 0.0f;
#pragma unroll
                for (uint32_t o = kG; o < 32u; o <<= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                if (r0 == 0u) sdb[q4][8u * c + e] = a;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    // one atomic per CTA and channel: their rounding is most of the sum's (32 images,
    // positive terms: 6.4e-8 of the sum from 64 bits, 4.8e-7 with one per warp)
    if (bias && threadIdx.x < CO)
        atomicAdd(p.db + co0 + threadIdx.x,
                  (sdb[0][threadIdx.x] + sdb[1][threadIdx.x]) + (sdb[2][threadIdx.x] + sdb[3][threadIdx.x]));
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512u);
    }
}

template <int CI, int CO, int KS, int R>
static cudaError_t dw_launch(const DwArgs &a, DwParams &p, cudaStream_t st) {
    constexpr int PX = 16 * KS;
    static_assert(PX / 4 % (32 / (CO / 8)) == 0, "a warp's share of a strip is whole steps of the bias sums");
    p.tiles_w = a.W / PX;
    p.rows = (long long)a.B * p.tiles_w * a.H;
    if (p.rows == 0) return cudaSuccess;
    const int chunks = a.Cin / CI, cols = (CI == 64 ? 2 : 1) * 3 * CO;
    // All SMs work, and while the rows are few a CTA takes as many input blocks as the
    // 512 TMEM columns hold, so that a gradient strip is read for all of them.  The
    // tensor cores' FP32 sums cut off below their last bit at every step, so a sum is
    // the more exact the shorter it is.  Full-resolution layers of 12 and more images:
    // at most 40 parts of one block each took the training step of 32 images 3.59 ms,
    // and the last layer's weight gradient was 6.3e-5 of its absolute sum from 64
    // bits; as many parts as SMs take 3.26 ms and are 9.7e-6 from it.  (All blocks in
    // one CTA there too: another 25 us less, but the 96 -> 32 layer's shorter sums would
    // move the whole gradient by more than the 2e-5 of its norm that one version may
    // differ from the next.)
    const bool many = CI == 32 && CO == 32 && p.rows > 6144;
    p.nc = 1;
    if (!many)
        for (p.nc = 512 / cols < chunks ? 512 / cols : chunks; chunks % p.nc; --p.nc) {}
    p.nci = chunks / p.nc;
    p.nco = a.Cout / CO;
    const int nblk = p.nci * p.nco, sms = device_sms();
    const long long want = nblk < sms ? sms / nblk : 1;
    p.splits = (int)(want < p.rows ? want : p.rows);
    // no sum covers more than a sixteenth of the pixels
    p.turns = (16 + p.splits - 1) / p.splits;
    p.x_tx = (uint32_t)(R * (PX + 2) * 2 * CI);
    p.z_tx = (uint32_t)(R * PX * 2 * CO);
    // one pixel further than the strips for the atom that is not used
    p.x_bytes = (p.x_tx + 2 * CI + 1023) / 1024 * 1024;
    const size_t stage = p.z_tx + (size_t)p.nc * p.x_bytes;
    p.stages = (int)(220u * 1024u / stage) < 12 ? (int)(220u * 1024u / stage) : 12;
    const size_t smem = 1024 + p.stages * stage + 8 * (2 * p.stages + 3) + 16;
    CUtensorMap tx, tz;
    auto image = [&](CUtensorMap *m, const uint16_t *q, int ch, int ld, int bc, int bp) {
        const uint64_t d[4] = {(uint64_t)ch, (uint64_t)a.W, (uint64_t)a.H, (uint64_t)a.B};
        const uint64_t s[3] = {(uint64_t)ld * 2, (uint64_t)ld * 2 * a.W, (uint64_t)ld * 2 * a.W * a.H};
        const uint32_t b[4] = {(uint32_t)bc, (uint32_t)bp, (uint32_t)R, 1};
        return tensor_map(m, q, 4, d, s, b, 2 * bc);
    };
    cudaError_t e;
    if ((e = image(&tx, a.x + a.xoff, a.Cin, a.ldx, CI, PX + 2)) != cudaSuccess) return e;
    if ((e = image(&tz, a.dz, a.Cout, a.Cout, CO, PX)) != cudaSuccess) return e;
    auto kernel = conv_wgrad_kernel<CI, CO, KS, R>;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
    kernel<<<(unsigned)(nblk * p.splits), 192, smem, st>>>(tx, tz, p);
    return cudaGetLastError();
}

cudaError_t conv_wgrad(const DwArgs &a, int *err, unsigned long long limit_ns, cudaStream_t st) {
    if (a.Cin % 32 || a.Cout % 32 || a.ldx % 8 || a.xoff % 8) return cudaErrorInvalidValue;
    DwParams p = {};
    p.Cin = a.Cin;
    p.Cout = a.Cout;
    p.H = a.H;
    p.dw = a.dw;
    p.db = a.db;
    p.err = err;
    p.limit_ns = limit_ns;
    // Strips of 128 pixels, or the whole of narrower rows, and as many rows per stage as
    // give its hand-off (a wait, a commit: about 500 cycles of the issuing warp) 16
    // MMAs to stand against.
    if (a.Cin % 64 || a.Cout % 64) {
        if (a.W % 128) return cudaErrorInvalidValue;
        return a.Cout % 64 == 0 ? dw_launch<32, 64, 8, 2>(a, p, st) : dw_launch<32, 32, 8, 2>(a, p, st);
    }
    if (a.W % 128 == 0) return dw_launch<64, 64, 8, 1>(a, p, st);
    if (a.W == 64) return dw_launch<64, 64, 4, 2>(a, p, st);
    if (a.W == 32) return dw_launch<64, 64, 2, 4>(a, p, st);
    return cudaErrorInvalidValue;
}

}  // namespace unet
}  // namespace synk
