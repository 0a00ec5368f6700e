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
// Against copies of both operands in a channel-major layout (x three times, shifted
// by kx), one tap per CTA, and a kernel for the bias, 32 images: 32 -> 32 at
// 256 x 256 448 -> 96 us, 96 -> 32 790 -> 252, 192 -> 64 at 128 x 128 396 -> 111,
// 384 -> 128 at 64 x 64 237 -> 153, 256 -> 256 at 32 x 32 113 -> 85; the training
// step 5.98 -> 3.64 ms.
#include "synk_internal.cuh"
#include "umma.cuh"
#include "umma_gemm.cuh"

namespace synk {
namespace unet {

using namespace umma;

struct DwParams {
    int Cin, Cout, H, tiles_w, px, nci, nco, nc, splits, turns, sx, sz;
    long long rows;                    // B * tiles_w * H rows of px pixels
    uint32_t x_bytes, z_bytes, x_tx, z_tx;
    float *dw, *db;
    int *err;
    unsigned long long limit_ns;
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

template <int CI, int CO>
__global__ void __launch_bounds__(192, 1) conv_wgrad_kernel(const __grid_constant__ CUtensorMap tmX,
                                                            const __grid_constant__ CUtensorMap tmZ, const DwParams p) {
    constexpr uint32_t kRowX = 2 * CI, kRowZ = 2 * CO;   // bytes of one pixel
    constexpr uint32_t kM = CI == 64 ? 2 : 1;            // MMAs of M = 128 that hold the three taps kx
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *zs = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    uint8_t *xs = zs + (size_t)p.sz * p.z_bytes;
    uint64_t *xfull = reinterpret_cast<uint64_t *>(xs + (size_t)p.sx * p.x_bytes);
    uint64_t *xempty = xfull + p.sx;
    uint64_t *zfull = xempty + p.sx;
    uint64_t *zempty = zfull + p.sz;
    uint64_t *tfull = zempty + p.sz;
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
        for (int s = 0; s < p.sx; ++s) {
            mbar_init(&xfull[s], 1);
            mbar_init(&xempty[s], 1);
        }
        for (int s = 0; s < p.sz; ++s) {
            mbar_init(&zfull[s], 1);
            mbar_init(&zempty[s], bias ? 5 : 1);
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
        for (uint32_t c = 0; c < (uint32_t)p.nc * kCols; c += 32u) tmem_zero32(tmem + c + ((uint32_t)((warp & 3) * 32) << 16));
        tmem_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    if (warp == 0) {
        // ---- producer: gradient row r + 1, then the strips of input row r ----
        uint32_t s = 0, ph = 1, used = 0, zsl = 0, zph = 1, zused = 0;
        bool fail = false;
        for (int t = 0; t < p.turns; ++t)
            for (long long q = q0 + len * t / p.turns, q1 = q0 + len * (t + 1) / p.turns; q < q1 && !fail;) {
                const long long col = q / p.H;
                const int ha = (int)(q - col * p.H);
                const int hb = q1 - q < (long long)(p.H - ha) ? ha + (int)(q1 - q) : p.H;
                const int b = (int)(col / p.tiles_w), w0 = (int)(col - (long long)b * p.tiles_w) * p.px;
                for (int r = ha - 1; r <= hb && !fail; ++r) {
                    if (r + 1 < hb) {
                        if (!__all_sync(0xffffffffu, mbar_wait(&zempty[zsl], zph, p.err, p.limit_ns))) {
                            fail = true;
                            break;
                        }
                        if (elect_one()) {
                            mbar_arrive_expect_tx(&zfull[zsl], p.z_tx);
                            tma_load_4d(zs + (size_t)zsl * p.z_bytes, &tmZ, &zfull[zsl], co0, w0, r + 1, b);
                        }
                        __syncwarp();
                        if (zused < (uint32_t)p.sz) ++zused;
                        if (++zsl == (uint32_t)p.sz) {
                            zsl = 0;
                            zph ^= 1u;
                        }
                    }
                    for (int c = 0; c < p.nc; ++c) {
                        if (!__all_sync(0xffffffffu, mbar_wait(&xempty[s], ph, p.err, p.limit_ns))) {
                            fail = true;
                            break;
                        }
                        if (elect_one()) {
                            // rows -1 and H and pixels -1 and W are out of bounds and read as 0
                            mbar_arrive_expect_tx(&xfull[s], p.x_tx);
                            tma_load_4d(xs + (size_t)s * p.x_bytes, &tmX, &xfull[s], ci0 + c * CI, w0 - 1, r, b);
                        }
                        __syncwarp();
                        if (used < (uint32_t)p.sx) ++used;
                        if (++s == (uint32_t)p.sx) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                }
                q += hb - ha;
            }
        // no copy may still be landing when the CTA exits
        for (uint32_t c = 0; c < used; ++c) mbar_drain(&xfull[c], c < s ? ph ^ 1u : ph, p.limit_ns);
        for (uint32_t c = 0; c < zused; ++c) mbar_drain(&zfull[c], c < zsl ? zph ^ 1u : zph, p.limit_ns);
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer ----
        const uint32_t xhi = smem_desc_hi(kRowX), zhi = smem_desc_hi(kRowZ);
        const uint32_t x0 = smem_u32(xs), z0 = smem_u32(zs);
        const uint32_t id1 = idesc_bf16(128, 0) | (3u << 15);   // both operands MN-major
        const uint32_t sz = (uint32_t)p.sz;
        const int ksteps = p.px / 16;
        uint32_t s = 0, ph = 0, osl = 0, oph = 0, csl = 0;
        bool fail = false;
        for (int t = 0; t < p.turns && !fail; ++t) {
            if (t > 0) {
                if (!__all_sync(0xffffffffu, mbar_wait(tempty, (uint32_t)(t - 1) & 1u, p.err, p.limit_ns))) break;
                tc_fence_after();
            }
            const long long q1 = q0 + len * (t + 1) / p.turns;
            for (long long q = q0 + len * t / p.turns; q < q1 && !fail;) {
                const long long col = q / p.H;
                const int ha = (int)(q - col * p.H);
                const int hb = q1 - q < (long long)(p.H - ha) ? ha + (int)(q1 - q) : p.H;
                for (int r = ha - 1; r <= hb; ++r) {
                    // gradient rows r+lo .. r+up (ky = 1-lo .. 1-up) meet this input row; the
                    // first is in ring slot csl
                    const int lo = r > ha ? -1 : ha - r, up = r + 1 < hb ? 1 : hb - 1 - r;
                    const bool closes = lo == -1;
                    if (up == 1) {
                        if (!__all_sync(0xffffffffu, mbar_wait(&zfull[osl], oph, p.err, p.limit_ns))) fail = true;
                        if (++osl == sz) {
                            osl = 0;
                            oph ^= 1u;
                        }
                    }
                    for (int c = 0; c < p.nc && !fail; ++c) {
                        if (!__all_sync(0xffffffffu, mbar_wait(&xfull[s], ph, p.err, p.limit_ns))) {
                            fail = true;
                            break;
                        }
                        tc_fence_after();
                        if (elect_one()) {
                            const uint32_t al = desc_lo_mn(x0 + s * p.x_bytes, kRowX);
                            uint32_t slot = csl, d = tmem + (uint32_t)c * kCols + (uint32_t)(lo + 1) * CO;
                            for (int left = up - lo + 1; left > 0;) {
                                // neighbours in the ring, up to its end
                                const uint32_t n = min((uint32_t)left, sz - slot);
                                const uint32_t idn = id1 | ((n * CO >> 3) << 17);
                                const uint32_t bl = desc_lo_mn(z0 + slot * p.z_bytes, p.z_bytes);
#pragma unroll 2
                                for (int k = 0; k < ksteps; ++k) {
                                    const uint32_t ak = al + (uint32_t)k * kRowX, bk = bl + (uint32_t)k * kRowZ;
                                    mma_bf16(d, ak, xhi, bk, zhi, idn, 1u);
                                    if (CI == 64)
                                        mma_bf16(d + 3u * CO, ak + 2u * (kRowX / 16u), xhi, bk, zhi, idn, 1u);
                                }
                                left -= (int)n;
                                d += n * CO;
                                slot += n;
                                if (slot == sz) slot = 0;
                            }
                            mma_commit(&xempty[s]);
                            if (closes && c + 1 == p.nc) mma_commit(&zempty[csl]);
                        }
                        __syncwarp();
                        if (++s == (uint32_t)p.sx) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                    if (fail) break;
                    if (closes && ++csl == sz) csl = 0;
                }
                q += hb - ha;
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
        const uint32_t per = (uint32_t)p.px / 4u;
        float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        uint32_t zsl = 0, zph = 0;
        bool ok = true;
        for (int t = 0; t < p.turns && ok; ++t) {
            const long long q1 = q0 + len * (t + 1) / p.turns;
            for (long long q = bias ? q0 + len * t / p.turns : q1; q < q1; ++q) {
                ok = __all_sync(0xffffffffu, mbar_wait(&zfull[zsl], zph, p.err, p.limit_ns));
                if (!ok) break;
                const uint8_t *z = zs + (size_t)zsl * p.z_bytes;
                float u8[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
                for (uint32_t i = r0; i < per; i += kStep) {
                    const uint32_t row = (uint32_t)q4 * per + i;
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
                __syncwarp();
                if (lane == 0) mbar_arrive(&zempty[zsl]);
                if (++zsl == (uint32_t)p.sz) {
                    zsl = 0;
                    zph ^= 1u;
                }
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
        if (bias && ok) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float a = acc[e];
#pragma unroll
                for (uint32_t o = kG; o < 32u; o <<= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                if (r0 == 0u) atomicAdd(p.db + co0 + 8u * c + e, a);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512u);
    }
}

template <int CI, int CO>
static cudaError_t dw_launch(const CUtensorMap &x, const CUtensorMap &z, const DwParams &p, size_t smem, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(conv_wgrad_kernel<CI, CO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    conv_wgrad_kernel<CI, CO><<<(unsigned)(p.nci * p.nco * p.splits), 192, smem, st>>>(x, z, p);
    return cudaGetLastError();
}

cudaError_t conv_wgrad(const DwArgs &a, int *err, unsigned long long limit_ns, cudaStream_t st) {
    if (a.Cin % 32 || a.Cout % 32 || (a.W > 128 ? a.W % 128 : a.W % 16) || a.ldx % 8 || a.xoff % 8)
        return cudaErrorInvalidValue;
    // blocks of 64 channels where they divide, else 32
    const int ci = a.Cin % 64 == 0 ? 64 : 32, co = a.Cout % 64 == 0 ? 64 : 32;
    DwParams p = {};
    p.Cin = a.Cin;
    p.Cout = a.Cout;
    p.H = a.H;
    p.px = a.W < 128 ? a.W : 128;
    p.tiles_w = a.W / p.px;
    p.rows = (long long)a.B * p.tiles_w * a.H;
    if (p.rows == 0) return cudaSuccess;
    // While the rows are few a CTA takes as many input blocks as the 512 TMEM columns
    // hold, so that a gradient strip is read for all of them.  From 8192 rows on it
    // takes one: three blocks over the 96 input channels of a batch of 32 leave sums
    // of 864 steps instead of 2624, and the cut-off bits (see below) that are missing
    // from them then move the gradient by 2.2e-5 of its norm from what sums of 3970
    // steps, one tap per CTA, gave; with one block it stays within 2e-5.
    const int chunks = a.Cin / ci, cols = (ci == 64 ? 2 : 1) * 3 * co;
    p.nc = 1;
    if (p.rows < 8192)
        for (p.nc = 512 / cols < chunks ? 512 / cols : chunks; chunks % p.nc; --p.nc) {}
    p.nci = chunks / p.nc;
    p.nco = a.Cout / co;
    const int nblk = p.nci * p.nco, sms = device_sms();
    const long long want = nblk < sms ? sms / nblk : 1;
    p.splits = (int)(want < p.rows ? want : p.rows);
    // the tensor cores' FP32 sums cut off below their last bit at every step: none
    // covers more than a sixteenth of the pixels before it joins the rounded totals
    p.turns = (16 + p.splits - 1) / p.splits;
    p.x_tx = (uint32_t)(p.px + 2) * 2 * ci;
    p.z_tx = (uint32_t)p.px * 2 * co;
    // one row further than the strip for the atom that is not used
    p.x_bytes = (p.x_tx + 2 * ci + 1023) / 1024 * 1024;
    p.z_bytes = (p.z_tx + 1023) / 1024 * 1024;
    // A gradient strip stays for three input rows, so its ring is three strips longer
    // for the same distance of prefetch.
    const size_t row = (size_t)p.nc * p.x_bytes + p.z_bytes;
    size_t depth = (220u * 1024u - 3 * (size_t)p.z_bytes) / row;
    if (depth > 16) depth = 16;
    p.sx = (int)depth * p.nc;
    p.sz = (int)depth + 3;
    p.dw = a.dw;
    p.db = a.db;
    p.err = err;
    p.limit_ns = limit_ns;
    const size_t smem = 1024 + (size_t)p.sx * p.x_bytes + (size_t)p.sz * p.z_bytes + 8 * (2 * p.sx + 2 * p.sz + 3) + 16;
    CUtensorMap tx, tz;
    auto image = [&](CUtensorMap *m, const uint16_t *q, int ch, int ld, int bc, int bp) {
        const uint64_t d[4] = {(uint64_t)ch, (uint64_t)a.W, (uint64_t)a.H, (uint64_t)a.B};
        const uint64_t s[3] = {(uint64_t)ld * 2, (uint64_t)ld * 2 * a.W, (uint64_t)ld * 2 * a.W * a.H};
        const uint32_t b[4] = {(uint32_t)bc, (uint32_t)bp, 1, 1};
        return tensor_map(m, q, 4, d, s, b, 2 * bc);
    };
    cudaError_t e;
    if ((e = image(&tx, a.x + a.xoff, a.Cin, a.ldx, ci, p.px + 2)) != cudaSuccess) return e;
    if ((e = image(&tz, a.dz, a.Cout, a.Cout, co, p.px)) != cudaSuccess) return e;
    if (ci == 64) return co == 64 ? dw_launch<64, 64>(tx, tz, p, smem, st) : dw_launch<64, 32>(tx, tz, p, smem, st);
    return co == 64 ? dw_launch<32, 64>(tx, tz, p, smem, st) : dw_launch<32, 32>(tx, tz, p, smem, st);
}

}  // namespace unet
}  // namespace synk
