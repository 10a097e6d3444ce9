// pt_conv.cu -- BF16 3x3 convolutions as implicit GEMMs on tcgen05 tensor
// cores, operands brought into shared memory by TMA (no multicast), FP32
// accumulators in tensor memory.  Interface and GEMM shapes: pt_conv.h.
//
// Tiling.  Accumulator tiles have 128 rows:
//   forward / data gradient: 128 pixels (one 128-wide row segment, or
//     128 / W whole rows of a narrow image) x n_tile output channels.  Persistent
//     CTAs of 10 warps walk the tiles: warp 0 streams operands into a ring of
//     `stages` buffers, warp 1 issues the MMAs into one of two accumulators,
//     warps 2-9 run the epilogue of the other (k_conv_fwd_persistent);
//   weight gradient: 128 (tap, input channel) rows x n_tile output channels,
//     accumulated over a range of pixel tiles and added to the FP32 result, by
//     CTAs of 4 warps: thread 0 loads, warp 1 issues the MMAs, all four warps read
//     the accumulators (warp w owns TMEM lanes 32w..32w+31).  One CTA per (chunk
//     of input channels with all nine taps, channel tile, pixel range)
//     (k_conv_wgrad_halo) or per (row tile, channel tile, pixel range) (k_conv_wgrad).
//
// Shared-memory operand layouts are the canonical swizzled ones for a row of
// R = 2 * KC bytes (R = 32, 64, 128 B, TMA swizzle of the same width):
//   K-major (forward A = pixels x channels, B = out channels x channels):
//     rows R bytes apart, 8-row groups SBO = 8R apart; a 16-element K slice
//     starts 32 B further along the row.
//   MN-major (weight gradient, A = channels x pixels, B = channels x pixels):
//     each TMA box holds 128 pixels (K) x KC channels (MN) as 128 rows of R
//     bytes; 8-pixel groups are SBO = 8R apart, consecutive KC-channel blocks
//     LBO = 128R apart; a 16-pixel K slice starts 16R further on.
// The zero padding of the convolution comes from TMA's out-of-bounds fill:
// the box for tap (dy, dx) starts at (x0 + dx - 1, y0 + dy - 1).
//
// Every wait is bounded (at least 2 s, counted in SM cycles): on expiry the kernel records a
// code in *err, stops issuing work, lets issued copies and MMAs drain (again
// with a bound), frees its tensor memory and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

#include "pt_conv.h"
#include "pt_internal.h"

namespace ptconv {

constexpr int kMaxStages = 8;
// A wait's limit counts ticks of two SM cycles, 9/8 per nanosecond: the clock's
// maximum is 2.07 GHz, so it lasts at least its nanoseconds (at one tick per
// nanosecond 400 ms ran out after 387).
constexpr uint64_t wait_ticks(uint64_t ns) { return ns + ns / 8; }
constexpr uint64_t kWaitTicks = wait_ticks(2000000000ull);

// ---------------------------------------------------------------------------
// device primitives (inline PTX)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for the phase with the given parity to complete: false after
// `ticks`, or as soon as *abort is set (another warp of the CTA gave up), so that a
// failing CTA leaves within one limit.  try_wait itself suspends the thread until
// the phase completes or a short hardware limit passes.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint64_t ticks = kWaitTicks,
                                          const volatile int *abort = nullptr) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    const long long limit = static_cast<long long>(ticks * 2);
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 8; i++)
            if (mbar_try(bar, parity)) return true;
        if (clock64() - t0 > limit) return false;
        if (abort && *abort) return false;
    }
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2,
                                            int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Issued by a whole warp, in the lane with `elected` set: the operands then stay
// in uniform registers.  One lane of a diverged warp, forming its descriptors
// per MMA, took 95 cycles for an MMA of 128 x 32 x 16 that runs in 40.
__device__ __forceinline__ void umma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(elected)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar),
        "r"(elected)
        : "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e;
}
// 32 lanes x 16 consecutive 32-bit columns: thread t of the warp gets lane
// (warp base + t), columns col..col+15.  tmem_ld16 starts the load, tmem_wait
// makes v valid; loads put between the two overlap it.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[16], float (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor (tcgen05): start, leading and stride byte
// offsets in 16-byte units, descriptor version 1 at bit 46, swizzle mode in
// bits 61-63 (2 = 128 B, 4 = 64 B, 6 = 32 B).
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t swz) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16) |
           (static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (static_cast<uint64_t>(swz) << 61);
}
// Instruction descriptor, kind::f16: FP32 D, BF16 A and B, K-major (0) or
// MN-major (1) operands, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
           (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
template <int KC>
__host__ __device__ constexpr uint32_t swz_mode() {
    return KC == 64 ? 2u : KC == 32 ? 4u : 6u;
}

__device__ __forceinline__ void record_error(unsigned *err, unsigned code) {
    if (err) atomicOr(err, code);
}

__device__ __forceinline__ uint16_t f2bf(float f) {
    __nv_bfloat16 h = __float2bfloat16_rn(f);
    return *reinterpret_cast<uint16_t *>(&h);
}

// 32-byte global accesses (256-bit loads and stores, sm_100 and later): the
// 16 BF16 channels a thread handles per step are one full sector.
__device__ __forceinline__ void ld_global_v8(const uint16_t *p, uint4 &a, uint4 &b) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                 : "l"(p));
}
__device__ __forceinline__ void st_global_v8(uint16_t *p, uint4 a, uint4 b) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z),
                 "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// 16 biases from channel ch0 on (of which nvalid exist), or zeros.
__device__ __forceinline__ void load_bias(const FwdArgs &a, int ch0, int nvalid, float (&b)[16]) {
    if (a.bias && nvalid == 16 && a.bias16) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(a.bias + ch0) + i);
            b[4 * i] = q.x;
            b[4 * i + 1] = q.y;
            b[4 * i + 2] = q.z;
            b[4 * i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++) b[i] = (a.bias && i < nvalid) ? __ldg(a.bias + ch0 + i) : 0.f;
    }
}

// Forward epilogue of the columns c0, c0 + cstep, ... (16 channels each):
// accumulator row `tid` = pixel (x0 + tid % tile_w, y0 + tid / tile_w); warp
// quadrant w reads TMEM lanes 32w..32w+31.  Bias and mask are loaded while the
// accumulator is.
__device__ __forceinline__ void fwd_epilogue(const FwdArgs &a, uint32_t tmem, int tid, int quad, int img, int x0, int y0,
                                             int n0, int c0, int cstep) {
    int px = tid, py = 0;
    if (a.tile_w != 128) {
        py = tid / a.tile_w;
        px = tid - py * a.tile_w;
    }
    const int x = x0 + px, y = y0 + py;
    const bool valid = py < a.tile_rows && x < a.W && y < a.H;
    const size_t pix = ((size_t)img * a.H + (valid ? y : 0)) * a.W + (valid ? x : 0);
    const uint32_t trow = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    for (int c = c0; c < a.n_tile; c += cstep) {
        uint32_t raw[16];
        tmem_ld16(trow + c, raw);
        const int ch0 = n0 + c;
        const int nvalid = min(16, a.cout - ch0);
        float v[16];
        if (a.epi == EPI_BF16_MASK) {
            uint4 q0 = make_uint4(0, 0, 0, 0), q1 = q0;
            const uint16_t *m = a.mask + pix * a.mask_ctot + a.mask_coff + ch0;
            if (valid && nvalid == 16) {
                if (a.wide_io) {
                    ld_global_v8(m, q0, q1);
                } else {
                    q0 = *reinterpret_cast<const uint4 *>(m);
                    q1 = *reinterpret_cast<const uint4 *>(m + 8);
                }
            } else if (valid) {
                uint16_t *h0 = reinterpret_cast<uint16_t *>(&q0), *h1 = reinterpret_cast<uint16_t *>(&q1);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    if (i < nvalid) h0[i] = m[i];
                    if (i + 8 < nvalid) h1[i] = m[i + 8];
                }
            }
            tmem_wait(raw, v);
            const uint16_t *h0 = reinterpret_cast<const uint16_t *>(&q0), *h1 = reinterpret_cast<const uint16_t *>(&q1);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (!(h0[i] != 0 && (h0[i] & 0x8000u) == 0)) v[i] = 0.f;
                if (!(h1[i] != 0 && (h1[i] & 0x8000u) == 0)) v[i + 8] = 0.f;
            }
        } else {
            float b[16];
            load_bias(a, ch0, nvalid, b);
            tmem_wait(raw, v);
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] += b[i];
        }
        if (!valid || nvalid <= 0) continue;
        if (a.epi == EPI_F32) {
            float *o = static_cast<float *>(a.out) + pix * a.out_ctot + a.out_coff + ch0;
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (i < nvalid) o[i] = v[i];
            continue;
        }
        if (a.epi == EPI_BF16 && a.relu) {
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = fmaxf(v[i], 0.f);
        }
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; i++) w[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
        const uint4 q0 = make_uint4(w[0], w[1], w[2], w[3]), q1 = make_uint4(w[4], w[5], w[6], w[7]);
        uint16_t *o = a.out ? static_cast<uint16_t *>(a.out) + pix * a.out_ctot + a.out_coff + ch0 : nullptr;
        // the four up-sampled copies (pixel (2y + i, 2x + j) of the 2H x 2W tensor)
        uint16_t *u = a.up ? a.up + (((size_t)img * 2 * a.H + 2 * y) * 2 * a.W + 2 * x) * a.up_ctot + ch0 : nullptr;
        const size_t urow = static_cast<size_t>(2 * a.W) * a.up_ctot;
        if (nvalid == 16) {
            if (a.wide_io) {
                if (o) st_global_v8(o, q0, q1);
                if (u) {
                    st_global_v8(u, q0, q1);
                    st_global_v8(u + a.up_ctot, q0, q1);
                    st_global_v8(u + urow, q0, q1);
                    st_global_v8(u + urow + a.up_ctot, q0, q1);
                }
            } else {
                if (o) {
                    reinterpret_cast<uint4 *>(o)[0] = q0;
                    reinterpret_cast<uint4 *>(o)[1] = q1;
                }
                for (int k = 0; u && k < 4; k++) {
                    uint16_t *uk = u + (k >> 1) * urow + (k & 1) * a.up_ctot;
                    reinterpret_cast<uint4 *>(uk)[0] = q0;
                    reinterpret_cast<uint4 *>(uk)[1] = q1;
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) {
                if (i >= nvalid) continue;
                const uint16_t h = static_cast<uint16_t>(w[i >> 1] >> (16 * (i & 1)));
                if (o) o[i] = h;
                for (int k = 0; u && k < 4; k++) u[(k >> 1) * urow + (k & 1) * a.up_ctot + i] = h;
            }
        }
    }
}

// Rows y0 and y0 + 1 of a halo tile with the pooled output (EPI_BF16, cout a
// multiple of 16, 32-byte aligned rows): thread `tid` holds pixel x = x0 + tid of
// both rows (accumulators tmem and tmem + n_tile), its neighbour lane x ^ 1.
// Each row is written as fwd_epilogue writes it; the even lane of each pair
// writes the average of the four BF16 outputs, summed in the order
// (y0, x), (y0, x + 1), (y0 + 1, x), (y0 + 1, x + 1).
__device__ __forceinline__ void fwd_epilogue_pool2(const FwdArgs &a, uint32_t tmem, int tid, int quad, int img, int x0,
                                                   int y0, int n0, int c0, int cstep) {
    const int x = x0 + tid;
    const bool valid = x < a.W && y0 < a.H;
    const size_t pix0 = ((size_t)img * a.H + (valid ? y0 : 0)) * a.W + (valid ? x : 0);
    const size_t ppix = ((size_t)img * (a.H / 2) + (valid ? y0 / 2 : 0)) * (a.W / 2) + (valid ? x / 2 : 0);
    const uint32_t trow = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    for (int c = c0; c < a.n_tile; c += cstep) {
        uint32_t raw0[16], raw1[16];
        tmem_ld16(trow + c, raw0);
        tmem_ld16(trow + a.n_tile + c, raw1);
        const int ch0 = n0 + c;
        float b[16];
        load_bias(a, ch0, min(16, a.cout - ch0), b);
        float v[2][16];
        tmem_wait(raw0, v[0]);
        tmem_wait(raw1, v[1]);
        if (ch0 >= a.cout) continue;  // uniform across the warp
        uint32_t w[2][8];
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float f0 = v[r][2 * i] + b[2 * i], f1 = v[r][2 * i + 1] + b[2 * i + 1];
                if (a.relu) {
                    f0 = fmaxf(f0, 0.f);
                    f1 = fmaxf(f1, 0.f);
                }
                w[r][i] = pack_bf16(f0, f1);
            }
        uint32_t pw[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t n0w = __shfl_xor_sync(0xffffffffu, w[0][i], 1), n1w = __shfl_xor_sync(0xffffffffu, w[1][i], 1);
            float acc[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float own0 = __uint_as_float((w[0][i] >> (16 * h)) << 16);
                const float own1 = __uint_as_float((w[1][i] >> (16 * h)) << 16);
                const float nb0 = __uint_as_float((n0w >> (16 * h)) << 16);
                const float nb1 = __uint_as_float((n1w >> (16 * h)) << 16);
                acc[h] = 0.25f * ((((0.f + own0) + nb0) + own1) + nb1);  // k_pool's order, from 0
            }
            pw[i] = pack_bf16(acc[0], acc[1]);
        }
        if (!valid) continue;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            uint16_t *o = static_cast<uint16_t *>(a.out) + (pix0 + (size_t)r * a.W) * a.out_ctot + a.out_coff + ch0;
            st_global_v8(o, make_uint4(w[r][0], w[r][1], w[r][2], w[r][3]), make_uint4(w[r][4], w[r][5], w[r][6], w[r][7]));
        }
        if ((tid & 1) == 0) {
            uint16_t *o = a.pool + ppix * a.pool_ctot + a.pool_coff + ch0;
            st_global_v8(o, make_uint4(pw[0], pw[1], pw[2], pw[3]), make_uint4(pw[4], pw[5], pw[6], pw[7]));
        }
    }
}

// ---------------------------------------------------------------------------
// halo operand layout (forward / data gradient, images at least 128 pixels wide)
// ---------------------------------------------------------------------------
// The pixel tile is a 128-pixel row segment of R output rows.  Per 16-channel
// chunk one TMA box brings its (R + 2) x 130-pixel neighbourhood (the segment
// and a one-pixel border, zero outside the image) as 32-byte pixel rows in the
// 32-byte-swizzled K-major layout, pixels in row-major order.  The A operand of
// input row i shifted by dx is the same box read from pixel row i * 130 + dx on
// (stride byte offset = 256 B between 8-row groups): the tensor cores apply the
// swizzle to the absolute shared-memory address, as the TMA wrote it, so a start
// at any 32-byte row reads the right data.
// Input row i adds to the output rows i - 2 .. i (taps dy = 2, 1, 0), whose
// accumulators are neighbours in tensor memory: one MMA of N = (up to three) x
// n_tile covers them, its B operand the chunk's weights for dx with dy falling.
// An MMA of 128 x N x 16 takes 32 + N / 4 cycles for N < 128 (measured; the A
// operand's 4 KiB is read either way), so three row taps cost 57 cycles instead
// of three times 40 at N = 32.  Each output row still gets its taps in the order
// dy, dx and is the same sum for every R.
// B holds the chunk's weights for all nine taps ([dx][2 - dy] blocks of n_tile
// rows, 32-byte swizzle, one TMA box per tap).  When one channel tile covers
// every output channel and all weights fit beside the ring, they are loaded once
// per CTA (on their own barrier) and the stages carry only the A box.
constexpr int kHaloW = 130;
__host__ __device__ constexpr int halo_box_bytes(int rows) { return kHaloW * (rows + 2) * 32; }
__host__ __device__ constexpr int halo_b_bytes(int n_tile) { return (9 * n_tile * 32 + 1023) / 1024 * 1024; }

// ---------------------------------------------------------------------------
// persistent forward / data-gradient kernel
// ---------------------------------------------------------------------------
// One CTA per SM slot walks the output tiles (pixel tile x output-channel
// tile) with a stride of gridDim.x.  Warp 0 streams operands into a ring of
// `stages` buffers across tile boundaries, warp 1 issues the MMAs into one of
// two accumulators in tensor memory (2 x rows x n_tile columns), and warps 2-9
// run the epilogue of tile i from one accumulator while the MMAs of tile i + 1
// fill the other.  Epilogue warp w reads TMEM lanes 32 * (w % 4) + 0..31; the
// two warps of a quadrant share a tile's rows or column groups.
// R > 0: the A operand comes from one (R + 2) x 130-pixel halo box per
// 16-channel chunk (width >= 128, see above); R = 0: one box per (tap, chunk).
// At 1920 x 1088 the layers were bound by the MMA issue (80 -> 32 channels 263
// us, of which 242 without loads and epilogue) and by the epilogue (16 -> 32: 84
// of 119 us).
constexpr int kFwdThreads = 320;
template <int KC, int R>
__global__ void __launch_bounds__(kFwdThreads, 2)
    k_conv_fwd_persistent(const __grid_constant__ CUtensorMap act, const __grid_constant__ CUtensorMap wgt,
                          const __grid_constant__ FwdArgs a) {
    constexpr bool HALO = R > 0;
    constexpr int ROWB = KC * 2;
    constexpr int kRows = HALO ? R : 1;  // output rows (accumulators) per tile
    constexpr uint32_t SWZ = swz_mode<KC>();
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 7];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool wres = HALO && a.wres_bytes > 0;  // weights resident ahead of the ring
    const uint32_t wbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t base = wbase + (wres ? static_cast<uint32_t>(a.wres_bytes) : 0u);
    const int S = a.stages;
    const int tiles_img = a.tiles_x * a.tiles_y;
    const int n_n = a.n_tiles_n;
    const int total = a.n_img * tiles_img * n_n;
    const int nk = HALO ? a.nchunks : 9 * a.nchunks;  // stages per tile
    const int a_bytes = HALO ? a.halo_a_bytes : 128 * ROWB;
    const uint32_t chunk_b = HALO ? static_cast<uint32_t>(halo_b_bytes(a.n_tile)) : 0u;
    const uint32_t tap_b = static_cast<uint32_t>(a.n_tile) * 32u;  // one tap's weights of a chunk (halo)
    const uint32_t tx_bytes = HALO ? static_cast<uint32_t>(halo_box_bytes(R) + (wres ? 0 : 9 * a.n_tile * ROWB))
                                   : static_cast<uint32_t>(a.tile_w * a.tile_rows * ROWB + a.n_tile * ROWB);
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (kMaxStages + s); };
    auto acc_full = [&](int b) { return bar0 + 8u * (2 * kMaxStages + b); };
    auto acc_empty = [&](int b) { return bar0 + 8u * (2 * kMaxStages + 2 + b); };
    const uint32_t wbar = bar0 + 8u * (2 * kMaxStages + 4);  // resident weights landed
    const uint32_t sbar = bar0 + 8u * (2 * kMaxStages + 5);  // never arrived at: the stall test waits on it
    const uint32_t mdone = bar0 + 8u * (2 * kMaxStages + 6);  // MMAs of a failing CTA completed
    const uint64_t lim = a.wait_ticks;
    auto tile_of = [&](int t, int &img, int &x0, int &y0, int &n0) {
        const int pt = t / n_n;
        n0 = (t - pt * n_n) * a.n_tile;
        img = pt / tiles_img;
        const int r = pt - img * tiles_img;
        const int ty = r / a.tiles_x;
        x0 = (r - ty * a.tiles_x) * a.tile_w;
        y0 = ty * a.tile_rows;
    };

    if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), a.tmem_cols);
    if (tid == 32) {
        for (int s = 0; s < S; s++) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(acc_full(b), 1);
            mbar_init(acc_empty(b), 256);
        }
        mbar_init(wbar, 1);
        mbar_init(sbar, 1);
        mbar_init(mdone, 1);
        mbar_fence_init();
        s_fail = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    volatile int *fail = &s_fail;

    if (warp == 0) {
        // producer: lane 0 waits for nobody but the ring; the nine weight boxes of a
        // chunk ([dx][2 - dy] blocks, tap = 3 dy + dx) are issued by nine lanes
        const int wdy = lane / 3, wdx = lane - 3 * wdy;
        const auto load_weights = [&](uint32_t dst, uint32_t bar, int k, int n0) {
            if (lane < 9)
                tma_load_2d(dst + static_cast<uint32_t>(wdx * 3 + 2 - wdy) * tap_b, &wgt, bar, lane * a.cin + k * 16, n0);
        };
        const auto wait = [&](uint32_t bar, uint32_t parity) {  // every lane, one answer
            return __all_sync(0xffffffffu, mbar_wait(bar, parity, lim, fail)) != 0;
        };
        if (wres) {
            if (lane == 0) mbar_expect_tx(wbar, static_cast<uint32_t>(a.nchunks * 9 * a.n_tile * ROWB));
            __syncwarp();
            for (int k = 0; k < a.nchunks; k++) load_weights(wbase + static_cast<uint32_t>(k) * chunk_b, wbar, k, 0);
        }
        int kg = 0;  // stages issued so far (ring position and phase)
        int s = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
            int img, x0, y0, n0;
            tile_of(t, img, x0, y0, n0);
            for (int k = 0; k < nk; k++, kg++) {
                if (kg >= S && !(ok = wait(empty(s), phase ^ 1u))) {
                    if (lane == 0) {
                        record_error(a.err, 1u);
                        *fail = 1;
                    }
                    break;
                }
                const uint32_t sa = base + s * a.stage_bytes, sb = sa + a_bytes;
                if ((sa | sb) & 1023u) {  // never with a layout fwd_prepare accepted: give up, bounded
                    if (lane == 0) {
                        record_error(a.err, 8u);
                        *fail = 1;
                    }
                    ok = false;
                    break;
                }
                if (lane == 0) {
                    mbar_expect_tx(full(s), tx_bytes);
                    if (HALO) {
                        tma_load_4d(sa, &act, full(s), k * 16, x0 - 1, y0 - 1, img);
                    } else {
                        const int tap = k / a.nchunks, ch = k - tap * a.nchunks;
                        const int dy = tap / 3, dx = tap - dy * 3;
                        tma_load_4d(sa, &act, full(s), ch * KC, x0 + dx - 1, y0 + dy - 1, img);
                        tma_load_2d(sb, &wgt, full(s), tap * a.cin + ch * KC, n0);
                    }
                }
                if (HALO && !wres) {
                    __syncwarp();
                    load_weights(sb, full(s), k, n0);
                }
                if (++s == S) {
                    s = 0;
                    phase ^= 1u;
                }
            }
            if (*fail) ok = false;
            ok = __all_sync(0xffffffffu, ok);
        }
        __syncwarp();
        // drain: every copy this warp issued has landed before the CTA leaves (the
        // last issue on each ring slot, and the resident weights), also when another
        // warp gave up; within the normal limit
        if (lane == 0) {
            for (int k = kg - S; k < kg; k++)
                if (k >= 0) (void)mbar_wait(full(k % S), (k / S) & 1);
            if (wres) (void)mbar_wait(wbar, 0);
        }
    } else if (warp == 1) {  // MMA issuer: the whole warp, so that descriptors stay uniform
        const uint32_t elected = elect_one();
        const auto wait = [&](uint32_t bar, uint32_t parity) {  // every lane, one answer
            if (__all_sync(0xffffffffu, mbar_wait(bar, parity, lim, fail))) return true;
            if (lane == 0) {
                record_error(a.err, 2u);
                *fail = 1;
            }
            return false;
        };
        const uint32_t idesc0 = idesc_bf16(128, 0, false, false);
        const uint32_t n_desc = static_cast<uint32_t>(a.n_tile >> 3) << 17;  // N = n_tile
        bool ok = true;
        if (a.stall) ok = wait(sbar, 0);  // the stall test: this wait always runs out
        if (ok && wres) ok = wait(wbar, 0);
        int kg = 0, j = 0, s = 0;
        uint32_t phase = 0;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x, j++) {
            const int buf = j & 1;
            if (!(ok = wait(acc_empty(buf), ((j >> 1) & 1) ^ 1))) break;  // epilogue of tile j - 2 done
            tc_fence_after();
            const uint32_t d = tmem + static_cast<uint32_t>(buf * kRows * a.n_tile);
            for (int k = 0; k < nk; k++, kg++) {
                if (!(ok = wait(full(s), phase))) break;
                tc_fence_after();
                const uint32_t sa = base + s * a.stage_bytes;
                const uint32_t sb = wres ? wbase + static_cast<uint32_t>(k) * chunk_b : sa + a_bytes;
                if constexpr (HALO) {
                    const uint64_t da0 = sdesc(sa, 16u, 256u, SWZ), db0 = sdesc(sb, 16u, 256u, SWZ);
                    const uint64_t tap_d = tap_b >> 4;
                    // rows r0..r1 of the tile from input row i shifted by dx
                    const auto mma = [&](int i, int dx, int r0, int r1, uint32_t accumulate) {
                        umma_bf16(d + static_cast<uint32_t>(r0 * a.n_tile), da0 + 2u * (i * kHaloW + dx),
                                  db0 + tap_d * (dx * 3 + 2 - (i - r0)), idesc0 + n_desc * (r1 - r0 + 1), accumulate,
                                  elected);
                    };
#pragma unroll
                    for (int i = 0; i < R + 2; i++) {
                        const int r0 = i >= 2 ? i - 2 : 0, r1 = i < R ? i : R - 1;
#pragma unroll
                        for (int dx = 0; dx < 3; dx++) {
                            if (dx == 0 && i < R && k == 0) {  // row i of the tile starts here
                                if (r0 < i) mma(i, dx, r0, i - 1, 1u);
                                mma(i, dx, i, i, 0u);
                            } else {
                                mma(i, dx, r0, r1, 1u);
                            }
                        }
                    }
                } else {
                    const uint64_t da0 = sdesc(sa, 16u, 8u * ROWB, SWZ), db0 = sdesc(sb, 16u, 8u * ROWB, SWZ);
#pragma unroll
                    for (int q = 0; q < KC / 16; q++)
                        umma_bf16(d, da0 + 2u * q, db0 + 2u * q, idesc0 + n_desc, (k | q) != 0 ? 1u : 0u, elected);
                }
                umma_commit(empty(s), elected);
                if (++s == S) {
                    s = 0;
                    phase ^= 1u;
                }
            }
            if (!ok) break;
            umma_commit(acc_full(buf), elected);
        }
        if (!ok && kg > 0) {  // let the MMAs already issued finish before tensor memory is freed
            umma_commit(mdone, elected);
            (void)mbar_wait(mdone, 0);
        }
    } else {  // epilogue warps 2-9
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const int row = quad * 32 + lane;
        int j = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, j++) {
            const int buf = j & 1;
            int img, x0, y0, n0;
            tile_of(t, img, x0, y0, n0);
            const bool ok = mbar_wait(acc_full(buf), (j >> 1) & 1, lim, fail);
            if (!ok) {
                if (row == 0 && half == 0) record_error(a.err, 4u);
                break;
            }
            tc_fence_after();
            const uint32_t acc = tmem + static_cast<uint32_t>(buf * kRows * a.n_tile);
            if (HALO && R % 2 == 0 && a.pool) {  // row pairs; one pair: its column groups in turn
#pragma unroll
                for (int r = 0; r < R; r += 2)
                    if (R < 4 || (r >> 1) == half)
                        fwd_epilogue_pool2(a, acc + static_cast<uint32_t>(r * a.n_tile), row, quad, img, x0, y0 + r, n0,
                                           R < 4 ? 16 * half : 0, R < 4 ? 32 : 16);
            } else {  // rows in turn, or one row's column groups
                for (int r = kRows > 1 ? half : 0; r < kRows; r += kRows > 1 ? 2 : 1)
                    fwd_epilogue(a, acc + static_cast<uint32_t>(r * a.n_tile), row, quad, img, x0, y0 + r, n0,
                                 kRows > 1 ? 0 : 16 * half, kRows > 1 ? 16 : 32);
            }
            tc_fence_before();
            mbar_arrive(acc_empty(buf));
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, a.tmem_cols);
}

// ---------------------------------------------------------------------------
// weight-gradient kernel
// ---------------------------------------------------------------------------
template <int KCA, int KCB>
__global__ void __launch_bounds__(128, 1)
    k_conv_wgrad(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap gmap, const WgradArgs a) {
    constexpr int RA = KCA * 2, RB = KCB * 2;
    constexpr uint32_t SWZA = swz_mode<KCA>(), SWZB = swz_mode<KCB>();
    constexpr int A_BLOCKS = 128 / KCA;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_issued, s_consumed, s_fail;

    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int S = a.stages;
    const int blk0 = blockIdx.x * A_BLOCKS;
    const int nblk = min(A_BLOCKS, 9 * a.nchunks_a - blk0);
    const int n0 = blockIdx.y * a.n_tile;
    const int nbb = a.n_tile / KCB;
    const int t_begin = blockIdx.z * a.tiles_per_split;
    const int nk = max(0, min(a.total_tiles, t_begin + a.tiles_per_split) - t_begin);
    const int a_bytes = 128 * 128 * 2;
    const int tile_px = a.tile_w * a.tile_rows;  // pixels one box delivers
    const uint32_t tx_bytes = static_cast<uint32_t>(nblk * tile_px * RA + nbb * tile_px * RB);
    const int tiles_img = a.tiles_x * a.tiles_y;
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (kMaxStages + s); };
    const uint32_t done = bar0 + 8u * (2 * kMaxStages);

    // The last M tile's spare A chunk holds BF16 ones in every stage (no box
    // writes it), so its D rows are the sums of gy over the pixels: the bias
    // gradient from the same MMAs.
    const bool ones = a.db != nullptr && a.ones_row >= 0 && blockIdx.x == gridDim.x - 1;
    if (a.zero_fill || ones) {  // zero fill: rows that no box covers must read as zero pixels
        const int ob = ones ? (a.ones_row / KCA) * 128 * RA : a.stage_bytes;  // ones chunk offset in a stage
        uint8_t *p = smem_raw + (base - smem_u32(smem_raw));
        for (int i = tid; i < S * a.stage_bytes / 16; i += blockDim.x) {
            const int off = (i * 16) % a.stage_bytes;
            if (off >= ob && off < ob + 128 * RA)
                reinterpret_cast<uint4 *>(p)[i] = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
            else if (a.zero_fill)
                reinterpret_cast<uint4 *>(p)[i] = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), a.tmem_cols);
    if (tid == 32) {
        for (int s = 0; s < S; s++) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        mbar_init(done, 1);
        mbar_fence_init();
        s_issued = 0;
        s_consumed = 0;
        s_fail = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (tid == 0) {
        int k = 0;
        for (; k < nk; k++) {
            const int s = k % S;
            if (k >= S && !mbar_wait(empty(s), ((k / S) - 1) & 1, a.wait_ticks)) {
                record_error(a.err, 1u);
                s_fail = 1;
                break;
            }
            if (*reinterpret_cast<volatile int *>(&s_fail)) break;
            const int tile = t_begin + k;
            const int img = tile / tiles_img, t = tile - img * tiles_img;
            const int x0 = (t % a.tiles_x) * a.tile_w, y0 = (t / a.tiles_x) * a.tile_rows;
            const uint32_t sa = base + s * a.stage_bytes, sb = sa + a_bytes;
            mbar_expect_tx(full(s), tx_bytes);
            for (int q = 0; q < nblk; q++) {
                const int b = blk0 + q;
                const int tap = b / a.nchunks_a, ch = b - tap * a.nchunks_a;
                const int dy = tap / 3, dx = tap - dy * 3;
                tma_load_4d(sa + q * 128 * RA, &xmap, full(s), ch * KCA, x0 + dx - 1, y0 + dy - 1, img);
            }
            for (int q = 0; q < nbb; q++) tma_load_4d(sb + q * 128 * RB, &gmap, full(s), n0 + q * KCB, x0, y0, img);
        }
        s_issued = k;
    } else if (warp == 1) {  // the whole warp: descriptors stay uniform
        const uint32_t elected = elect_one();
        const uint32_t idesc = idesc_bf16(128, a.n_tile, true, true);
        int k = 0, s = 0;
        uint32_t phase = 0;
        for (; k < nk; k++) {
            if (!__all_sync(0xffffffffu, mbar_wait(full(s), phase, a.wait_ticks))) {
                if (elected) {
                    record_error(a.err, 2u);
                    s_fail = 1;
                }
                break;
            }
            tc_fence_after();
            const uint32_t sa = base + s * a.stage_bytes, sb = sa + a_bytes;
            const uint64_t da0 = sdesc(sa, 128u * RA, 8u * RA, SWZA), db0 = sdesc(sb, 128u * RB, 8u * RB, SWZB);
#pragma unroll
            for (int j = 0; j < 8; j++)  // 16 pixels per MMA
                umma_bf16(tmem, da0 + static_cast<uint64_t>(RA * j), db0 + static_cast<uint64_t>(RB * j), idesc,
                          (k | j) != 0 ? 1u : 0u, elected);
            umma_commit(empty(s), elected);
            if (++s == S) {
                s = 0;
                phase ^= 1u;
            }
        }
        if (elected) s_consumed = k;
        umma_commit(done, elected);
    }
    __syncwarp();
    const bool ok = nk > 0 && mbar_wait(done, 0, a.wait_ticks);
    if (!ok && nk > 0 && tid == 0) record_error(a.err, 4u);
    tc_fence_after();

    // epilogue: row tid = A row (tap, ci) index g; dw[co][g] += D[tid][co - n0]
    const int g = blk0 * KCA + tid;
    const bool valid = ok && tid < nblk * KCA;
    const bool bias_row = ok && ones && tid == a.ones_row;  // db[co] += D[ones_row][co - n0]
    const uint32_t trow = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    const size_t kdim = 9 * static_cast<size_t>(a.cin);
    for (int c = 0; c < a.n_tile; c += 16) {
        uint32_t raw[16];
        float v[16];
        tmem_ld16(trow + c, raw);
        tmem_wait(raw, v);
        if (!valid && !bias_row) continue;
        float *dst = valid ? a.dw + g : a.db;
        const size_t stride = valid ? kdim : 1;
        for (int i = 0; i < 16; i++) {
            const int co = n0 + c + i;
            if (co < a.cout) atomicAdd(dst + co * stride, v[i]);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_fail) {
        for (int k = s_consumed; k < s_issued; k++) (void)mbar_wait(full(k % S), (k / S) & 1);
    }
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, a.tmem_cols);
}

// ---------------------------------------------------------------------------
// weight gradient from halo boxes (width >= 128, or a multiple of 16)
// ---------------------------------------------------------------------------
// The per-tap kernel above brings every 128-pixel tile of x nine times, in rows
// as narrow as 32 bytes, and is bound by those copies (16 x 256^2: 80 -> 32
// channels 222 us, here 121; 32 -> 32 85 us, here 47; 112 -> 48 at half the size 87
// us, here 59; without the MMAs 87, 34 and 30 us, the copies).  Here a CTA takes one chunk of KCA input channels and all
// nine taps: one TMA box per tile holds the chunk's (rows + 2) x (tile_w + 2)
// pixels, and the A operand of a tap is that box read from the tap's pixel on
// (MN-major: 8-pixel groups SBO = 8 RA bytes apart; any start row works, as in
// the forward kernel).  M = 128 holds 128 / KCA channel blocks, LBO bytes apart:
//   KCA = 64: two taps, LBO = their distance; five accumulators
//             (taps 0 1 | 2 3 | 4 5 | 6 7 | 7 8, the second 7 unused)
//   KCA = 32, 16: LBO = one pixel, so the blocks are dx = 0, 1, 2 and unused ones;
//             three accumulators (dy)
// A K slice is 16 pixels of one row.  Unused blocks read up to five pixels past
// the box (inside the stage) and only reach unused accumulator rows.  The last
// chunk may reach past cin: its channels arrive as zeros and are not written.
// Warps 2 and 3 sum dy over the pixels meanwhile: the bias gradient (CTAs of
// chunk 0).
template <int KCA, int KCB, int TW>
__global__ void __launch_bounds__(128, 1)
    k_conv_wgrad_halo(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap gmap,
                      const __grid_constant__ WgradArgs a) {
    constexpr int RA = KCA * 2, RB = KCB * 2;
    constexpr uint32_t SWZA = swz_mode<KCA>(), SWZB = swz_mode<KCB>();
    constexpr int kSets = KCA == 64 ? 5 : 3;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    __shared__ float s_db[128];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int S = a.stages;
    const int chunk = blockIdx.x;
    s_db[tid] = 0.f;
    const int n0 = blockIdx.y * a.n_tile;
    const int nbb = a.n_tile / KCB;
    const int t_begin = blockIdx.z * a.tiles_per_split;
    const int nk = max(0, min(a.total_tiles, t_begin + a.tiles_per_split) - t_begin);
    constexpr int kPitch = TW + 2;  // pixels per row of the box
    const int tile_px = TW * a.tile_rows;
    const uint32_t tx_bytes = static_cast<uint32_t>((a.tile_rows + 2) * kPitch * RA + nbb * tile_px * RB);
    const int tiles_img = a.tiles_x * a.tiles_y;
    const bool bias = a.db != nullptr && chunk == 0;
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (kMaxStages + s); };
    const uint32_t done = bar0 + 8u * (2 * kMaxStages);

    if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), a.tmem_cols);
    if (tid == 32) {
        for (int s = 0; s < S; s++) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), bias ? 3 : 1);  // the MMAs, and the two summing warps
        }
        mbar_init(done, 1);
        mbar_fence_init();
        s_fail = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    volatile int *fail = &s_fail;

    if (warp == 0) {
        if (lane == 0) {  // producer
            int k = 0, s = 0;
            uint32_t phase = 0;
            int img = t_begin / tiles_img, ty = (t_begin - img * tiles_img) / a.tiles_x;
            int tx = t_begin - img * tiles_img - ty * a.tiles_x;
            for (; k < nk && !*fail; k++) {
                if (k >= S && !mbar_wait(empty(s), phase ^ 1u, a.wait_ticks, fail)) {
                    record_error(a.err, 1u);
                    *fail = 1;
                    break;
                }
                const int x0 = tx * TW, y0 = ty * a.tile_rows;
                const uint32_t sa = base + s * a.stage_bytes, sb = sa + a.a_bytes;
                mbar_expect_tx(full(s), tx_bytes);
                tma_load_4d(sa, &xmap, full(s), chunk * KCA, x0 - 1, y0 - 1, img);
                for (int q = 0; q < nbb; q++) tma_load_4d(sb + q * 128 * RB, &gmap, full(s), n0 + q * KCB, x0, y0, img);
                if (++s == S) {
                    s = 0;
                    phase ^= 1u;
                }
                if (++tx == a.tiles_x) {
                    tx = 0;
                    if (++ty == a.tiles_y) {
                        ty = 0;
                        img++;
                    }
                }
            }
            // every copy issued has landed before the CTA leaves, also on failure
            for (int q = k - S; q < k; q++)
                if (q >= 0) (void)mbar_wait(full(q % S), (q / S) & 1);
        }
    } else if (warp == 1) {  // MMA issuer (whole warp: descriptors stay uniform)
        const uint32_t elected = elect_one();
        const uint32_t idesc = idesc_bf16(128, a.n_tile, true, true);
        const int slices = tile_px / 16;
        // per accumulator set: the A descriptor relative to the stage and the slice's pixel
        uint64_t dq[kSets];
#pragma unroll
        for (int q = 0; q < kSets; q++) {
            const int t0 = KCA == 64 ? (q < 4 ? 2 * q : 7) : 3 * q, t1 = t0 + 1;  // taps of the first two blocks
            const uint32_t off = static_cast<uint32_t>((t0 / 3) * kPitch + t0 % 3);
            const uint32_t lbo = static_cast<uint32_t>((t1 / 3 - t0 / 3) * kPitch + t1 % 3 - t0 % 3);
            dq[q] = sdesc(off * RA, (KCA == 64 ? lbo : 1u) * RA, 8u * RA, SWZA);
        }
        int s = 0;
        uint32_t phase = 0;
        for (int k = 0; k < nk; k++) {
            if (!__all_sync(0xffffffffu, mbar_wait(full(s), phase, a.wait_ticks, fail))) {
                if (elected) {
                    record_error(a.err, 2u);
                    *fail = 1;
                }
                break;
            }
            tc_fence_after();
            const uint32_t sa = base + s * a.stage_bytes, sb = sa + a.a_bytes;
            const uint64_t db0 = sdesc(sb, 128u * RB, 8u * RB, SWZB);
#pragma unroll
            for (int j = 0; j < 8; j++) {  // 16 pixels of row j / (TW / 16)
                if (j >= slices) continue;
                const uint32_t at = (sa >> 4) + static_cast<uint32_t>(j / (TW / 16) * kPitch + j % (TW / 16) * 16) * (RA >> 4);
#pragma unroll
                for (int q = 0; q < kSets; q++)
                    umma_bf16(tmem + static_cast<uint32_t>(q * a.n_tile), dq[q] + at,
                              db0 + static_cast<uint64_t>(16 * j * (RB >> 4)), idesc, (k | j) != 0 ? 1u : 0u, elected);
            }
            umma_commit(empty(s), elected);
            if (++s == S) {
                s = 0;
                phase ^= 1u;
            }
        }
        umma_commit(done, elected);
    } else if (bias) {  // warps 2, 3: 8 channels of the pixels lane_p, lane_p + step, ... each
        const int units = a.n_tile / 8, t2 = tid - 64;
        const int unit = t2 % units, lane_p = t2 / units, step = 64 / units;
        const bool active = lane_p < step;
        const int ch = 8 * unit;
        const uint32_t col = static_cast<uint32_t>((ch / KCB) * 128 * RB + (ch % KCB) * 2);
        const uint8_t *smem0 = smem_raw - smem_u32(smem_raw);  // + a shared address
        float sum[8];
#pragma unroll
        for (int i = 0; i < 8; i++) sum[i] = 0.f;
        int s = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int k = 0; k < nk && ok; k++) {
            ok = __all_sync(0xffffffffu, mbar_wait(full(s), phase, a.wait_ticks, fail));
            if (!ok) break;
            const uint32_t sb = base + s * a.stage_bytes + a.a_bytes + col;
#pragma unroll 4
            for (int p = active ? lane_p : tile_px; p < tile_px; p += step) {
                uint32_t addr = sb + static_cast<uint32_t>(p) * RB;
                // the TMA's swizzle: 16-byte unit bits XOR the row bits above 128 bytes
                addr ^= (addr >> 3) & (KCB == 64 ? 0x70u : KCB == 32 ? 0x30u : 0x10u);
                const uint4 v = *reinterpret_cast<const uint4 *>(smem0 + addr);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    sum[2 * i] += __uint_as_float(w[i] << 16);
                    sum[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty(s));
            if (++s == S) {
                s = 0;
                phase ^= 1u;
            }
        }
        if (ok && active)
#pragma unroll
            for (int i = 0; i < 8; i++) atomicAdd(&s_db[ch + i], sum[i]);
    }
    __syncwarp();
    const bool ok = nk > 0 && mbar_wait(done, 0, a.wait_ticks);
    if (!ok && nk > 0 && tid == 0) record_error(a.err, 4u);
    tc_fence_after();

    // epilogue: accumulator row tid = (block, channel) of each set
    const int blk = tid / KCA, ci = chunk * KCA + tid % KCA;
    const uint32_t trow = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    const bool good = __all_sync(0xffffffffu, ok && !*fail);
    for (int q = 0; q < kSets && good; q++) {
        const int tap = KCA == 64 ? (q < 4 ? 2 * q + blk : 8) : 3 * q + blk;
        const bool used = ci < a.cin && (KCA == 64 ? (q < 4 || blk == 1) : blk < 3);
        float *dst = a.dw + static_cast<size_t>(tap) * a.cin + ci;
        for (int c = 0; c < a.n_tile; c += 16) {
            uint32_t raw[16];
            float v[16];
            tmem_ld16(trow + static_cast<uint32_t>(q * a.n_tile + c), raw);
            tmem_wait(raw, v);
            if (!used) continue;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int co = n0 + c + i;
                if (co < a.cout) atomicAdd(dst + static_cast<size_t>(co) * 9 * a.cin, v[i]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (bias && !*fail && tid < a.n_tile && n0 + tid < a.cout) atomicAdd(a.db + n0 + tid, s_db[tid]);
    if (warp == 0) tmem_dealloc(tmem, a.tmem_cols);
}

// ---------------------------------------------------------------------------
// small kernels
// ---------------------------------------------------------------------------
__global__ void k_bias_grad(const uint16_t *g, int ctot, int coff, int c, long long npix, float *db) {
    extern __shared__ float sacc[];
    const int per = blockDim.x / c;  // pixels per pass
    const int lane_c = threadIdx.x % c, lane_p = threadIdx.x / c;
    float acc = 0.f;
    if (lane_p < per) {
        for (long long p = (long long)blockIdx.x * per + lane_p; p < npix; p += (long long)gridDim.x * per) {
            uint32_t bits = static_cast<uint32_t>(g[p * ctot + coff + lane_c]) << 16;
            acc += __uint_as_float(bits);
        }
    }
    sacc[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x < c) {
        float s = 0.f;
        for (int i = 0; i < per; i++) s += sacc[i * c + threadIdx.x];
        atomicAdd(db + threadIdx.x, s);
    }
}

__global__ void k_flip_transpose(const uint16_t *w, int cout, int cin, uint16_t *wt) {
    const long long n = 9ll * cout * cin;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int ci = static_cast<int>(i % cin);
        const int tap = static_cast<int>((i / cin) % 9);
        const int co = static_cast<int>(i / (9ll * cin));
        wt[(static_cast<long long>(ci) * 9 + (8 - tap)) * cout + co] = w[i];
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

CUtensorMapSwizzle swizzle_for(int kc) {
    return kc == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : kc == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
}

struct Tiling {
    int tile_w, tile_rows, tiles_x, tiles_y;
};
Tiling tiling_for(int h, int w) {
    Tiling t;
    if (w >= 128) {
        t.tile_w = 128;
        t.tile_rows = 1;
    } else {
        t.tile_w = w;
        t.tile_rows = std::min(128 / w, h);
    }
    t.tiles_x = (w + t.tile_w - 1) / t.tile_w;
    t.tiles_y = (h + t.tile_rows - 1) / t.tile_rows;
    return t;
}

int act_map_box(CUtensorMap *m, const Act &a, int box_c, int box_w, int box_h, CUtensorMapSwizzle swz, int kc) {
    auto fn = encode_fn();
    if (!fn) {
        pt_set_error("cuTensorMapEncodeTiled is not available from the driver");
        return PT_ERR_CUDA;
    }
    char *p = static_cast<char *>(a.ptr) + 2ull * a.coff;
    if ((reinterpret_cast<uintptr_t>(p) & 15) || (a.ctot % 8) || (a.c % kc)) {
        pt_set_error("activation tensor: base, channel stride or channel count misaligned (ctot %d coff %d c %d)", a.ctot,
                     a.coff, a.c);
        return PT_ERR_INVALID;
    }
    cuuint64_t dims[4] = {(cuuint64_t)a.c, (cuuint64_t)a.w, (cuuint64_t)a.h, (cuuint64_t)a.n};
    cuuint64_t strides[3] = {2ull * a.ctot, 2ull * a.ctot * a.w, 2ull * a.ctot * a.w * a.h};
    cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)box_w, (cuuint32_t)box_h, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, p, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        pt_set_error("cuTensorMapEncodeTiled (activation %dx%dx%dx%d, box %dx%dx%d) failed: %d", a.n, a.h, a.w, a.c,
                     box_c, box_w, box_h, static_cast<int>(r));
        return PT_ERR_CUDA;
    }
    return PT_OK;
}

// Tile boxes: kc channels x the pixel tile, swizzled to the row width.
int act_map(CUtensorMap *m, const Act &a, int kc, const Tiling &t) {
    return act_map_box(m, a, kc, t.tile_w, t.tile_rows, swizzle_for(kc), kc);
}

int wgt_map(CUtensorMap *m, const void *w, int kdim, int rows, int kc, int n_tile) {
    auto fn = encode_fn();
    if (!fn) {
        pt_set_error("cuTensorMapEncodeTiled is not available from the driver");
        return PT_ERR_CUDA;
    }
    if ((reinterpret_cast<uintptr_t>(w) & 15) || (kdim % 8)) {
        pt_set_error("weight tensor misaligned");
        return PT_ERR_INVALID;
    }
    cuuint64_t dims[2] = {(cuuint64_t)kdim, (cuuint64_t)rows};
    cuuint64_t strides[1] = {2ull * kdim};
    cuuint32_t box[2] = {(cuuint32_t)kc, (cuuint32_t)n_tile};
    cuuint32_t es[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(w), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(kc), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        pt_set_error("cuTensorMapEncodeTiled (weights %dx%d, box %dx%d) failed: %d", rows, kdim, kc, n_tile,
                     static_cast<int>(r));
        return PT_ERR_CUDA;
    }
    return PT_OK;
}

int sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
            n = 1;
    }
    return n;
}

bool getenv_flag(const char *name) {
    const char *v = getenv(name);
    return v && *v && *v != '0';
}

int pow2_cols(int n) {
    int c = 32;
    while (c < n) c <<= 1;
    return c;
}

// Dynamic shared memory for `stages` buffers, raised where needed so that no
// more CTAs share an SM than its 512 tensor-memory columns can hold.
int smem_request(int stages, int stage_bytes, int tmem_cols) {
    const int by_stages = stages * stage_bytes + 1024;
    const int max_ctas = 512 / tmem_cols;
    const int floor_bytes = (228 * 1024) / (max_ctas + 1) + 1024;
    return std::max(by_stages, max_ctas >= 32 ? 0 : floor_bytes);
}

// Raises a kernel instantiation's dynamic shared-memory limit to `bytes`
// when a launch needs more than it was given so far (per process).
template <class K>
int set_smem_attr(K kernel, int bytes) {
    static std::mutex mu;
    static std::map<const void *, int> raised;  // kernel -> limit set so far
    std::lock_guard<std::mutex> lock(mu);
    const void *key = reinterpret_cast<const void *>(kernel);
    auto it = raised.find(key);
    const int have = it == raised.end() ? 48 * 1024 : it->second;
    if (bytes <= have) return PT_OK;
    PT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    raised[key] = bytes;
    return PT_OK;
}

}  // namespace

int pick_kc(int c) {
    if (c % 64 == 0) return 64;
    if (c % 32 == 0) return 32;
    return 16;
}

// Limit of the kernels' bounded waits (pt_conv_set_wait_limit; 0 = kWaitTicks)
// and the one-shot request to stall the next forward convolution.
static std::atomic<unsigned long long> g_wait_ns{0};
static std::atomic<int> g_stall_next{0};
unsigned long long wait_limit() {
    const unsigned long long v = g_wait_ns.load();
    return v ? wait_ticks(v) : kWaitTicks;
}
bool take_stall_request() { return g_stall_next.exchange(0) != 0; }
void set_wait_limit(unsigned long long ns, bool stall_next) {
    g_wait_ns.store(ns);
    g_stall_next.store(stall_next ? 1 : 0);
}

int fwd_prepare(FwdOp *op, const Act &in, const void *w, int w_rows, int cout, const float *bias, int epi, int relu,
                void *out, int out_ctot, int out_coff, const Act *mask, unsigned *err, void *up, int up_ctot,
                void *pool, int pool_ctot, int pool_coff) {
    if (in.c <= 0 || in.c % 16 || cout <= 0 || in.n <= 0 || in.h <= 0 || in.w <= 0) {
        pt_set_error("conv forward: channel counts must be positive multiples of 16 (cin %d, cout %d)", in.c, cout);
        return PT_ERR_INVALID;
    }
    if (epi == EPI_BF16_MASK && (!mask || mask->n != in.n || mask->h != in.h || mask->w != in.w)) {
        pt_set_error("conv forward: mask tensor missing or of the wrong shape");
        return PT_ERR_INVALID;
    }
    if (!out && !(up && epi == EPI_BF16)) {
        pt_set_error("conv forward: no output");
        return PT_ERR_INVALID;
    }
    if (epi != EPI_F32 && ((out_ctot % 8) || (out_coff % 8))) {
        pt_set_error("conv forward: bf16 output channel stride/offset must be multiples of 8");
        return PT_ERR_INVALID;
    }
    const bool halo = in.w >= 128 && !getenv_flag("PT_CONV_NO_HALO");
    const int kc = halo ? 16 : pick_kc(in.c);
    const Tiling t = tiling_for(in.h, in.w);
    const int cout_pad = (cout + 15) / 16 * 16;
    int ntiles = (cout_pad + 255) / 256;
    // Narrow images with few pixel tiles (an eighth of the SMs or less): the output
    // channels are split, down to 32 a tile, until the SMs have a tile each.  Such a
    // CTA is bound by what one SM takes in for a chunk, so fewer columns of weights
    // beside the 16 KB of pixels shorten its chain.  Training step 2 x 256^2 658 ->
    // 620 us, 320 x 180 frame 278 -> 264, 960 x 540 mirror ensemble 672 -> 656.  With
    // more tiles than that the pixels read again cost as much as the split gives
    // (16 x 256^2: 1470 us without, 1475 with it).
    if (!halo) {
        const long long tiles = (long long)in.n * t.tiles_x * t.tiles_y;
        if (8 * tiles <= sm_count())
            ntiles = std::max(ntiles, (int)std::min<long long>(sm_count() / tiles, (cout_pad + 31) / 32));
    }
    int n_tile = ((cout_pad / ntiles) + 15) / 16 * 16;
    ntiles = (cout_pad + n_tile - 1) / n_tile;
    // Output rows per halo tile: four while both accumulators of every row fit the
    // 512 tensor-memory columns and three rows' outputs one MMA (N <= 256), else
    // two or one; fewer where the tiles would not give every SM two.
    // PT_CONV_HALO_ROWS=1..4 overrides (as far as tensor memory allows).
    const auto rows_fit = [&](int r) {
        return pow2_cols(2 * r * n_tile) <= 512 && std::min(r, 3) * n_tile <= 256;
    };
    const auto tiles_at = [&](int r) {
        return (long long)in.n * ((in.w + 127) / 128) * ((in.h + r - 1) / r) * ntiles;
    };
    const auto box_bytes = [](int r) { return (halo_box_bytes(r) + 1023) / 1024 * 1024; };
    const int wres_bytes = in.c / 16 * halo_b_bytes(n_tile);
    const auto resident = [&](int r, int budget) { return ntiles == 1 && wres_bytes + 3 * box_bytes(r) <= budget; };
    const auto budget_of = [](int ctas) { return (225 * 1024) / ctas - 4096; };
    int halo_rows = 4;
    // (weights that do not stay cross L2 once per tile: then one tile for most SMs is enough)
    while (halo_rows > 1 && (!rows_fit(halo_rows) ||
                             tiles_at(halo_rows) < (resident(halo_rows, budget_of(1)) ? 2ll * sm_count() : 3ll * sm_count() / 4)))
        halo_rows /= 2;
    if (const char *e = getenv("PT_CONV_HALO_ROWS")) {
        halo_rows = std::min(std::max(atoi(e), 1), 4);
        while (halo_rows > 1 && !rows_fit(halo_rows)) halo_rows--;
    }
    int st;
    if (halo) {
        if ((st = act_map_box(&op->act, in, 16, kHaloW, halo_rows + 2, CU_TENSOR_MAP_SWIZZLE_32B, 16)) != PT_OK)
            return st;
    } else if ((st = act_map(&op->act, in, kc, t)) != PT_OK) {
        return st;
    }
    if ((st = wgt_map(&op->wgt, w, 9 * in.c, w_rows, kc, n_tile)) != PT_OK) return st;
    FwdArgs &a = op->args;
    memset(&a, 0, sizeof(a));
    a.n_img = in.n;
    a.H = in.h;
    a.W = in.w;
    a.tile_w = t.tile_w;
    a.tile_rows = t.tile_rows;
    a.tiles_x = t.tiles_x;
    a.tiles_y = t.tiles_y;
    a.cin = in.c;
    a.nchunks = in.c / kc;
    a.n_tile = n_tile;
    a.cout = cout;
    a.n_tiles_n = ntiles;
    a.tmem_cols = pow2_cols(2 * (halo ? halo_rows : 1) * n_tile);  // double-buffered accumulators
    a.halo_a_bytes = box_bytes(halo_rows);
    // CTAs per SM (two at most: 640 threads; PT_CONV_FWD_CTAS=1 or 2 overrides) and
    // the ring: resident weights where a ring of three stages fits beside them,
    // at one CTA per SM if need be
    int ctas = std::min(512 / a.tmem_cols, 2);
    if (const char *e = getenv("PT_CONV_FWD_CTAS")) ctas = std::min(ctas, std::max(atoi(e), 1));
    a.wres_bytes = 0;
    if (halo && !getenv_flag("PT_CONV_NO_RESIDENT"))
        for (int c = ctas; c >= 1 && !a.wres_bytes; c--)
            if (resident(halo_rows, budget_of(c))) {
                a.wres_bytes = wres_bytes;
                ctas = c;
            }
    a.stage_bytes = halo ? a.halo_a_bytes + (a.wres_bytes ? 0 : halo_b_bytes(n_tile))
                         : (128 * 2 * kc + n_tile * 2 * kc + 1023) / 1024 * 1024;
    if (ctas > 1 && 2 * a.stage_bytes + a.wres_bytes > budget_of(ctas)) ctas = 1;
    a.stages = std::max(2, std::min(kMaxStages, (budget_of(ctas) - a.wres_bytes) / a.stage_bytes));
    // every stage, A box and chunk of weights on a 1 KiB boundary of the
    // 1 KiB-aligned ring (the producer checks it again), a tap's weights on 512 B
    if (a.stage_bytes % 1024 || a.wres_bytes % 1024 || (halo && (a.halo_a_bytes % 1024 || n_tile % 16))) {
        pt_set_error("conv forward: shared-memory layout off 1 KiB boundaries");
        return PT_ERR_INVALID;
    }
    if (halo) {
        a.tile_w = 128;
        a.tile_rows = halo_rows;
        a.tiles_x = (in.w + 127) / 128;
        a.tiles_y = (in.h + halo_rows - 1) / halo_rows;
    }
    a.epi = epi;
    a.relu = relu;
    a.bias = bias;
    a.out = out;
    a.out_ctot = out_ctot;
    a.out_coff = out_coff;
    if (mask) {
        a.mask = static_cast<const uint16_t *>(mask->ptr);
        a.mask_ctot = mask->ctot;
        a.mask_coff = mask->coff;
    }
    // 32-byte accesses when every 16-channel group of the output (and mask)
    // starts on a 32-byte boundary
    auto al32 = [](const void *ptr, int ctot, int coff) {
        return (reinterpret_cast<uintptr_t>(ptr) % 32) == 0 && ctot % 16 == 0 && coff % 16 == 0;
    };
    a.bias16 = bias && (reinterpret_cast<uintptr_t>(bias) % 16) == 0 ? 1 : 0;
    if (up && epi == EPI_BF16) {
        if (up_ctot < cout || up_ctot % 8) {
            pt_set_error("conv forward: up-sampled output needs at least cout channels, a multiple of 8");
            return PT_ERR_INVALID;
        }
        a.up = static_cast<uint16_t *>(up);
        a.up_ctot = up_ctot;
    }
    // the 2x2 average pooling of the output, in the epilogue of halo tiles of two
    // or four rows (both rows of a pixel pair are in one thread, the pair in
    // neighbouring lanes); otherwise the caller pools
    if (pool && halo && halo_rows % 2 == 0 && epi == EPI_BF16 && cout % 16 == 0 && in.w % 2 == 0 && in.h % 2 == 0 &&
        ntiles == 1 && al32(pool, pool_ctot, pool_coff) && al32(out, out_ctot, out_coff) &&
        !getenv_flag("PT_CONV_NO_FUSED_POOL")) {  // (the pooled epilogue writes both outputs with 32-byte stores)
        a.pool = static_cast<uint16_t *>(pool);
        a.pool_ctot = pool_ctot;
        a.pool_coff = pool_coff;
    }
    a.wide_io = epi != EPI_F32 && al32(out, out_ctot, out_coff) &&
                (!mask || al32(mask->ptr, mask->ctot, mask->coff)) && (!a.up || al32(a.up, a.up_ctot, 0)) &&
                !getenv_flag("PT_CONV_NO_WIDE_IO");
    a.err = err;
    a.wait_ticks = wait_limit();
    a.stall = take_stall_request() ? 1 : 0;
    op->kc = kc;
    // no more CTAs on an SM than tensor memory holds accumulators for
    const auto smem_of = [&] {
        const int by_stages = a.stages * a.stage_bytes + a.wres_bytes + 1024;
        return std::max(by_stages, (228 * 1024) / (ctas + 1) + 1024);
    };
    while (a.stages > 2 && smem_of() > 220 * 1024) a.stages--;
    op->smem = smem_of();
    op->rows = halo ? halo_rows : 0;
    const long long total = (long long)in.n * a.tiles_x * a.tiles_y * ntiles;
    op->grid = dim3(static_cast<unsigned>(std::min<long long>(total, (long long)ctas * sm_count())), 1, 1);
    if (op->smem > 220 * 1024) {
        pt_set_error("conv forward: shared memory request %d too large", op->smem);
        return PT_ERR_INVALID;
    }
    return PT_OK;
}

template <int KC, int R>
static int fwd_persistent_go(const FwdOp &op, cudaStream_t stream) {
    int st = set_smem_attr(k_conv_fwd_persistent<KC, R>, op.smem);
    if (st != PT_OK) return st;
    k_conv_fwd_persistent<KC, R><<<op.grid, kFwdThreads, op.smem, stream>>>(op.act, op.wgt, op.args);
    PT_CUDA_TRY(cudaGetLastError());
    return PT_OK;
}

int fwd_launch(const FwdOp &op, cudaStream_t stream) {
    switch (op.rows) {
        case 1: return fwd_persistent_go<16, 1>(op, stream);
        case 2: return fwd_persistent_go<16, 2>(op, stream);
        case 3: return fwd_persistent_go<16, 3>(op, stream);
        case 4: return fwd_persistent_go<16, 4>(op, stream);
        default: break;
    }
    if (op.kc == 64) return fwd_persistent_go<64, 0>(op, stream);
    if (op.kc == 32) return fwd_persistent_go<32, 0>(op, stream);
    return fwd_persistent_go<16, 0>(op, stream);
}

// Halo kernel: chunk width by the MMAs a tile takes (accumulator sets x chunks;
// 48, 64, 112 and wider inputs: 64 channels, 80: 32), equal ones wider.
static int wgrad_prepare_halo(WgradOp *op, const Act &x, const Act &gy, float *dw, float *db, int num_sms,
                              unsigned *err) {
    int kca = 64, cost = 5 * ((x.c + 63) / 64);
    for (int kc : {32, 16}) {
        const int c = 3 * ((x.c + kc - 1) / kc);
        if (c < cost) {
            cost = c;
            kca = kc;
        }
    }
    const int sets = kca == 64 ? 5 : 3;
    // output channels per CTA: a multiple of the dy chunk whose accumulators fit
    // the 512 tensor-memory columns
    const int kcb = pick_kc(gy.c);
    int n_tile = gy.c;
    while (sets * n_tile > 512 || n_tile > 128 || gy.c % n_tile || n_tile % kcb) n_tile -= 16;
    Tiling t;
    // 32 x 4 pixels (16 x 8 where 32 would leave part of every row): 204 pixels of
    // x per tile instead of the 390 of a 128-pixel row segment
    t.tile_w = x.w >= 128 || x.w % 32 == 0 ? 32 : 16;
    t.tile_rows = std::min(128 / t.tile_w, x.h);
    t.tiles_x = (x.w + t.tile_w - 1) / t.tile_w;
    t.tiles_y = (x.h + t.tile_rows - 1) / t.tile_rows;
    int st;
    if ((st = act_map_box(&op->act, x, kca, t.tile_w + 2, t.tile_rows + 2, swizzle_for(kca), 16)) != PT_OK) return st;
    if ((st = act_map(&op->grad, gy, kcb, t)) != PT_OK) return st;
    WgradArgs &a = op->args;
    memset(&a, 0, sizeof(a));
    a.n_img = x.n;
    a.H = x.h;
    a.W = x.w;
    a.tile_w = t.tile_w;
    a.tile_rows = t.tile_rows;
    a.tiles_x = t.tiles_x;
    a.tiles_y = t.tiles_y;
    a.cin = x.c;
    a.nchunks_a = (x.c + kca - 1) / kca;
    a.cout = gy.c;
    a.n_tile = n_tile;
    a.tmem_cols = pow2_cols(sets * n_tile);
    a.a_bytes = ((t.tile_rows + 2) * (t.tile_w + 2) * 2 * kca + 1023) / 1024 * 1024;
    a.stage_bytes = a.a_bytes + 256 * n_tile;
    // about half an SM's shared memory, so that a data-gradient CTA of the other
    // stream fits beside it; two stages at least
    a.stages = std::min(4, std::max(2, (100 * 1024) / a.stage_bytes));
    a.total_tiles = x.n * t.tiles_x * t.tiles_y;
    a.db = db;
    a.ones_row = -1;
    a.dw = dw;
    a.err = err;
    a.wait_ticks = wait_limit();
    op->bias_fused = db != nullptr;
    op->smem = std::max(a.stages * a.stage_bytes + 1024, (228 * 1024) / (512 / a.tmem_cols + 1) + 1024);
    const int base_ctas = a.nchunks_a * (gy.c / n_tile);
    // Pixel ranges: one CTA per SM.  (Fewer, so that fewer CTAs add to the gradient,
    // measured no faster: 64 -> 64 channels on 16 x 64^2 28 against 25 us.)
    int splits = std::max(1, std::max(num_sms, 1) / base_ctas);
    splits = std::min(splits, a.total_tiles);
    a.tiles_per_split = (a.total_tiles + splits - 1) / splits;
    splits = (a.total_tiles + a.tiles_per_split - 1) / a.tiles_per_split;
    op->kca = kca;
    op->kcb = kcb;
    op->halo = true;
    op->grid = dim3(static_cast<unsigned>(a.nchunks_a), static_cast<unsigned>(gy.c / n_tile),
                    static_cast<unsigned>(splits));
    if (op->smem > 220 * 1024) {
        pt_set_error("conv weight gradient: shared memory request %d too large", op->smem);
        return PT_ERR_INVALID;
    }
    return PT_OK;
}

int wgrad_prepare(WgradOp *op, const Act &x, const Act &gy, float *dw, float *db, int num_sms, unsigned *err) {
    if (x.n != gy.n || x.h != gy.h || x.w != gy.w || x.c % 16 || gy.c % 16 || x.c <= 0 || gy.c <= 0) {
        pt_set_error("conv weight gradient: shapes differ or channels not multiples of 16");
        return PT_ERR_INVALID;
    }
    if (x.w >= 128 || x.w % 16 == 0) return wgrad_prepare_halo(op, x, gy, dw, db, num_sms, err);
    const int kca = pick_kc(x.c);
    const Tiling t = tiling_for(x.h, x.w);
    // output channels per CTA: a multiple of the dy chunk, at most 256
    int kcb = pick_kc(gy.c);
    int ntiles = (gy.c + 255) / 256;
    while (gy.c % (ntiles * kcb) != 0 && kcb > 16) kcb /= 2;
    while (gy.c % (ntiles * kcb) != 0) ntiles++;
    const int n_tile = gy.c / ntiles;
    int st;
    if ((st = act_map(&op->act, x, kca, t)) != PT_OK) return st;
    if ((st = act_map(&op->grad, gy, kcb, t)) != PT_OK) return st;
    WgradArgs &a = op->args;
    memset(&a, 0, sizeof(a));
    a.n_img = x.n;
    a.H = x.h;
    a.W = x.w;
    a.tile_w = t.tile_w;
    a.tile_rows = t.tile_rows;
    a.tiles_x = t.tiles_x;
    a.tiles_y = t.tiles_y;
    a.cin = x.c;
    a.nchunks_a = x.c / kca;
    a.cout = gy.c;
    a.n_tile = n_tile;
    a.tmem_cols = pow2_cols(n_tile);
    a.stage_bytes = 128 * 128 * 2 + 256 * n_tile;
    // two stages per CTA, so that two CTAs (two producer / MMA thread pairs)
    // share an SM: 2.66 ms per training step at batch 16 x 256^2 instead of
    // 3.21 ms with up to four stages and one CTA per SM
    a.stages = 2;
    a.total_tiles = x.n * t.tiles_x * t.tiles_y;
    a.zero_fill = t.tile_w * t.tile_rows < 128 ? 1 : 0;
    const int m_tiles = (9 * a.nchunks_a * kca + 127) / 128;
    const int base_ctas = m_tiles * ntiles;
    const int last_blocks = 9 * a.nchunks_a - (m_tiles - 1) * (128 / kca);  // chunks in the last M tile
    a.ones_row = last_blocks < 128 / kca ? last_blocks * kca : -1;
    a.db = a.ones_row >= 0 && !getenv_flag("PT_CONV_NO_FUSED_BIAS") ? db : nullptr;
    op->bias_fused = a.db != nullptr;
    op->smem = smem_request(a.stages, a.stage_bytes, a.tmem_cols);
    // split the pixel tiles so that the grid is one full wave of resident CTAs
    const int per_sm = std::max(1, std::min((228 * 1024) / (op->smem + 1024), 512 / a.tmem_cols));
    int splits = std::max(1, (per_sm * std::max(num_sms, 1)) / base_ctas);
    splits = std::min(splits, std::max(1, a.total_tiles / 4));
    a.tiles_per_split = (a.total_tiles + splits - 1) / splits;
    splits = (a.total_tiles + a.tiles_per_split - 1) / a.tiles_per_split;
    a.dw = dw;
    a.err = err;
    a.wait_ticks = wait_limit();
    op->kca = kca;
    op->kcb = kcb;
    op->halo = false;
    op->grid = dim3(static_cast<unsigned>(m_tiles), static_cast<unsigned>(ntiles), static_cast<unsigned>(splits));
    if (op->smem > 220 * 1024) {
        pt_set_error("conv weight gradient: shared memory request %d too large", op->smem);
        return PT_ERR_INVALID;
    }
    return PT_OK;
}

template <int KCA, int KCB>
static int wgrad_go(const WgradOp &op, cudaStream_t stream) {
    if (op.halo) {
        const auto kernel = op.args.tile_w == 32 ? k_conv_wgrad_halo<KCA, KCB, 32> : k_conv_wgrad_halo<KCA, KCB, 16>;
        const int e = set_smem_attr(kernel, op.smem);
        if (e != PT_OK) return e;
        kernel<<<op.grid, 128, op.smem, stream>>>(op.act, op.grad, op.args);
        PT_CUDA_TRY(cudaGetLastError());
        return PT_OK;
    }
    int st = set_smem_attr(k_conv_wgrad<KCA, KCB>, op.smem);
    if (st != PT_OK) return st;
    k_conv_wgrad<KCA, KCB><<<op.grid, 128, op.smem, stream>>>(op.act, op.grad, op.args);
    PT_CUDA_TRY(cudaGetLastError());
    return PT_OK;
}

int wgrad_launch(const WgradOp &op, cudaStream_t stream) {
#define PT_WG(A, B) \
    if (op.kca == A && op.kcb == B) return wgrad_go<A, B>(op, stream);
    PT_WG(64, 64) PT_WG(64, 32) PT_WG(64, 16) PT_WG(32, 64) PT_WG(32, 32) PT_WG(32, 16) PT_WG(16, 64) PT_WG(16, 32)
    PT_WG(16, 16)
#undef PT_WG
    pt_set_error("conv weight gradient: unsupported chunk pair %d/%d", op.kca, op.kcb);
    return PT_ERR_INVALID;
}

int bias_grad_launch(const Act &g, float *db, cudaStream_t stream) {
    if (g.c <= 0 || g.c > 512) {
        pt_set_error("bias gradient: %d channels", g.c);
        return PT_ERR_INVALID;
    }
    const int threads = std::max(g.c, (256 / g.c) * g.c);
    const long long npix = (long long)g.n * g.h * g.w;
    const int blocks = static_cast<int>(std::min<long long>(1024, (npix + 63) / 64));
    k_bias_grad<<<blocks, threads, threads * sizeof(float), stream>>>(static_cast<const uint16_t *>(g.ptr), g.ctot,
                                                                       g.coff, g.c, npix, db);
    PT_CUDA_TRY(cudaGetLastError());
    return PT_OK;
}

int flip_transpose_launch(const uint16_t *w, int cout, int cin, uint16_t *wt, cudaStream_t stream) {
    const long long n = 9ll * cout * cin;
    const int blocks = static_cast<int>(std::min<long long>(4096, (n + 255) / 256));
    k_flip_transpose<<<blocks, 256, 0, stream>>>(w, cout, cin, wt);
    PT_CUDA_TRY(cudaGetLastError());
    return PT_OK;
}

}  // namespace ptconv
