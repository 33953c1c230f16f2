// fp16 convolution (group 1; any kernel, stride up to 8, dilation, padding) as an implicit GEMM on tcgen05:
//     Y[n, m, h, w] = act(B[m] + sum_{c, i, j} W[m, c, i, j] * X[n, c, sh h - pad_top + dh i, sw w - pad_left + dw j] * gate[n, c]) + R[n, m, h, w]
// (the reference's routes: daceml/onnx/op_implementations/img_op_implementations.py:217-288, cudnn_implementations.py:123-410).
//
// X is read channels-last ([N][H][W][Cp], Cp = C rounded up to 8): a box of {64 channels, wb x hb pixels, nb images} at the
// window position of one kernel tap is then a K-major operand tile that the TMA unit lays out by itself - the padding is
// its zero fill, a stride its element stride - so there is no im2col buffer and no shifting by warps.  An NCHW X is turned
// by a small kernel first (nchw_to_nhwc_kernel, which also applies a squeeze-excite gate); between two convolutions of a
// graph the epilogue writes channels-last directly (B200ML_CONV_X_NHWC / Y_NHWC) and the turn is not needed.
// The reduction runs over (tap, channel chunk of 16, 32 or 64); the weights of a step come as one bulk copy from a copy
// laid out beforehand in the operand tile's swizzled order (once per constant weight, else once per call).
//
// One 128-pixel x BN-channel tile per CTA, two to four CTAs per SM so that one's epilogue runs under the others' main loops; few
// tiles split the reduction over a cluster (partial tiles through distributed shared memory, summed in rank order).
// The box wb x hb x nb <= 128 is chosen to cover the output with the fewest tiles (56 x 56: 28 x 4).
// Bound: L2 -> shared memory traffic (every tap re-reads its window) and, on small layers, latency.
//
// Measured (us, direct FMA kernel before -> turn + convolution): two 3x3, 64 -> 64 at 56 x 56, 8 images 535 -> 16.5 (one turn);
// 3x3 32 -> 36 at 117 x 117, 24 images 17.5 + 46; 1x1 24 -> 144 at 56 x 56, 32 images 8.8 + 42.
#include "gemm_common.cuh"

namespace b200ml {

namespace {

constexpr int H_BM = 128;
constexpr int H_THREADS = 64 + 128;         // TMA warp, MMA warp, four epilogue warps
constexpr int H_PIPE_BYTES = 96 * 1024;     // operand stages of a CTA: two CTAs fit on an SM ...
constexpr int H_MIN_PIPE_BYTES = 48 * 1024; // ... up to four where the reduction is short; never more, for the tensor memory's sake
constexpr int H_MAX_STAGES = 8;
constexpr int H_PART_LD = H_BM + 4;         // floats between columns of a parked partial tile
constexpr int H_PACK_ROWS = 32;

struct ConvHArgs {
    const __half* w;         // packed weights: [step][rows (padded)][kc], swizzled
    const __half* bias;
    const __half* residual;
    __half* y;
    int32_t n, m, oh, ow;
    int32_t wb, hb, nb;                       // pixels of a tile
    int32_t tiles_w, tiles_h, tiles_n, tiles_m;
    int32_t kc, chunks, steps, kw;            // channels per step, chunks of channels per tap, steps in all
    int32_t packed_rows, stages, pipe_bytes, split;
    int32_t sh, sw, dh, dw, pad_top, pad_left;
    int32_t act, y_nhwc;
    int32_t* status;
};

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(ptx::smem_u32(bar))
                 : "memory");
}

// K-major operand tile with rows of 2 * kc bytes in the matching swizzle (128, 64 or 32 bytes): 8-row groups are
// 16 * kc bytes apart.
__device__ __forceinline__ uint64_t conv_desc(uint32_t addr, int kc) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr & 0x3ffffu) >> 4);
    d |= 1ull << 16;
    d |= static_cast<uint64_t>(kc & 0x3fff) << 32;  // (16 * kc) >> 4
    d |= 1ull << 46;
    d |= static_cast<uint64_t>(kc == 64 ? 2 : (kc == 32 ? 4 : 6)) << 61;
    return d;
}

// Sixteen channels from m0 on of one output pixel.
__device__ __forceinline__ void finish16(const ConvHArgs& g, const float (&acc)[16], int m0, int64_t pix_nchw, int64_t pix_nhwc) {
    const int64_t plane = static_cast<int64_t>(g.oh) * g.ow;
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = acc[j];
    if (g.bias) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (m0 + j < g.m) v[j] += __half2float(__ldg(g.bias + m0 + j));
    }
    if (g.act) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = conv_act(v[j], g.act);
    }
    if (g.y_nhwc) {  // m is a multiple of 8 here
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (m0 + 8 * u < g.m) {
                float o[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = v[8 * u + j];
                if (g.residual) {
                    float q[8];
                    unpack8(__ldg(reinterpret_cast<const uint4*>(g.residual + pix_nhwc + m0 + 8 * u)), q);
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[j] += q[j];
                }
                *reinterpret_cast<uint4*>(g.y + pix_nhwc + m0 + 8 * u) = pack8(o);
            }
        }
        return;
    }
    __half r[16];
    if (g.residual) {
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = m0 + j < g.m ? g.residual[pix_nchw + (m0 + j) * plane] : __float2half_rn(0.0f);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += __half2float(r[j]);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (m0 + j < g.m) g.y[pix_nchw + (m0 + j) * plane] = __float2half_rn(v[j]);
}

template <int BN>
__global__ void __launch_bounds__(H_THREADS, 4) conv_f16_kernel(const __grid_constant__ CUtensorMap tmap_x, const ConvHArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + g.pipe_bytes);
    uint64_t* empty_bar = full_bar + H_MAX_STAGES;
    uint64_t* acc_bar = empty_bar + H_MAX_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = g.split > 1 ? static_cast<int>(ptx::cluster_ctarank()) : 0;
    int t = blockIdx.x / g.split;
    const int mt = t % g.tiles_m;  // the channel blocks of one window run at the same time: its second read hits L2
    t /= g.tiles_m;
    const int w0 = (t % g.tiles_w) * g.wb;
    t /= g.tiles_w;
    const int h0 = (t % g.tiles_h) * g.hb;
    const int n0 = (t / g.tiles_h) * g.nb;
    const int per = (g.steps + g.split - 1) / g.split;
    const int begin = rank * per < g.steps ? rank * per : g.steps;
    const int nk = (begin + per < g.steps ? begin + per : g.steps) - begin;
    const int a_bytes = H_BM * g.kc * 2, stage_bytes = a_bytes + BN * g.kc * 2;

    if (warp == 0 && lane == 0) ptx::prefetch_tensormap(&tmap_x);
    if (warp == 1) {
        if (lane == 0) {
            for (int s = 0; s < g.stages; ++s) {
                ptx::mbar_init(&full_bar[s], 1);
                ptx::mbar_init(&empty_bar[s], 1);
            }
            ptx::mbar_init(acc_bar, 1);
            ptx::fence_mbar_init();
        }
        __syncwarp();
        ptx::tmem_alloc(tmem_slot, BN);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    pdl_launch_dependents();  // after the allocation: an early CTA of the next kernel cannot take this CTA's tensor memory
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------ producer: one box of X and one block of weights per step ------------------------------
        if (ptx::elect_one()) {
            pdl_wait();
            const int rows = g.packed_rows - mt * BN < BN ? g.packed_rows - mt * BN : BN;
            const uint32_t w_bytes = rows * g.kc * 2, x_bytes = g.wb * g.hb * g.nb * g.kc * 2;
            int stage = 0;
            uint32_t phase = 0;
            int chunk = begin % g.chunks, tap = begin / g.chunks;
            int ti = tap / g.kw, tj = tap - ti * g.kw;
            for (int i = 0; i < nk; ++i) {
                if (!ptx::mbar_wait(&empty_bar[stage], phase ^ 1)) {
                    atomicExch(g.status, DEV_TIMEOUT_PRODUCER);
                    break;
                }
                uint8_t* dst = smem + stage * stage_bytes;
                ptx::mbar_expect_tx(&full_bar[stage], w_bytes + x_bytes);
                bulk_copy(ptx::smem_u32(dst + a_bytes), g.w + (static_cast<int64_t>(begin + i) * g.packed_rows + mt * BN) * g.kc, w_bytes, &full_bar[stage]);
                ptx::tma_load_4d(dst, &tmap_x, &full_bar[stage], chunk * g.kc, w0 * g.sw - g.pad_left + tj * g.dw, h0 * g.sh - g.pad_top + ti * g.dh, n0);
                if (++chunk == g.chunks) {
                    chunk = 0;
                    if (++tj == g.kw) tj = 0, ++ti;
                }
                if (++stage == g.stages) stage = 0, phase ^= 1;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        if (ptx::elect_one()) {
            constexpr uint32_t idesc = ptx::make_idesc_f16(H_BM, BN, 0, 0);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int i = 0; i < nk; ++i) {
                if (!ptx::mbar_wait(&full_bar[stage], phase)) {
                    atomicExch(g.status, DEV_TIMEOUT_MMA);
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                const uint32_t a = ptx::smem_u32(smem + stage * stage_bytes);
                const uint64_t da = conv_desc(a, g.kc), db = conv_desc(a + a_bytes, g.kc);
                for (int kk = 0; kk < g.kc / 16; ++kk)  // 32 bytes along the line per step
                    ptx::mma_f16_ss(tmem_base, da + 2 * kk, db + 2 * kk, idesc, (i | kk) != 0 ? 1u : 0u);
                ptx::mma_commit(&empty_bar[stage]);
                if (++stage == g.stages) stage = 0, phase ^= 1;
            }
            if (ok && nk > 0) ptx::mma_commit(acc_bar);
        }
        __syncwarp();
    }
    // ------------------------------ epilogue: a lane = a pixel, a warp = 32 pixels ------------------------------
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int pw = w0 + row % g.wb, ph = h0 + (row / g.wb) % g.hb, pn = n0 + row / (g.wb * g.hb);
    const bool pix_ok = row < g.wb * g.hb * g.nb && pw < g.ow && ph < g.oh && pn < g.n;
    const int64_t pix_nchw = (static_cast<int64_t>(pn) * g.m * g.oh + ph) * g.ow + pw;
    const int64_t pix_nhwc = ((static_cast<int64_t>(pn) * g.oh + ph) * g.ow + pw) * g.m;
    float* partial = reinterpret_cast<float*>(smem);
    if (warp >= 2) {
        bool ok = true;
        pdl_wait();  // the residual, and Y itself, may be a predecessor's
        if (nk > 0 && !ptx::mbar_wait(acc_bar, 0)) {
            if (lane == 0) atomicExch(g.status, DEV_TIMEOUT_EPILOGUE);
            ok = false;
        }
        __syncwarp();
        ptx::tc_fence_after();
#pragma unroll 1
        for (int c = 0; ok && c < BN; c += 16) {
            if (mt * BN + c >= g.m) break;  // warp-uniform
            uint32_t r[16];
            if (nk > 0) {
                ptx::tmem_ld_32x32b_x16(tmem_base + c + (static_cast<uint32_t>(quarter * 32) << 16), r);
                ptx::tmem_ld_wait();
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) r[j] = 0u;
            }
            if (g.split == 1) {
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
                if (pix_ok) finish16(g, v, mt * BN + c, pix_nchw, pix_nhwc);
                __syncwarp();
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) partial[(c + j) * H_PART_LD + row] = __uint_as_float(r[j]);
            }
        }
        ptx::tc_fence_before();
    }
    if (g.split > 1) {
        ptx::cluster_sync_acq_rel();
        if (warp >= 2) {
            // this CTA's share of the channels, in pieces of sixteen
            const int share = BN / g.split;  // 16 or more
            for (int c = rank * share; c < (rank + 1) * share; c += 16) {
                if (mt * BN + c >= g.m) break;
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = 0.0f;
                for (int q = 0; q < g.split; ++q) {  // rank order: the same sum on every run
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] += ptx::ld_shared_cluster_f32(partial + (c + j) * H_PART_LD + row, q);
                }
                if (pix_ok) finish16(g, v, mt * BN + c, pix_nchw, pix_nhwc);
            }
        }
        ptx::cluster_sync_acq_rel();  // no CTA leaves while a peer may still read its partial tile
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        if (*reinterpret_cast<volatile int32_t*>(g.status) != DEV_OK) {
            for (int i = 0; i < 200; ++i) __nanosleep(1000);  // a wait gave up: let copies and MMAs in flight land
        }
        ptx::tmem_dealloc(tmem_base, BN);
    }
}

// [N][C][HW] -> [N][HW][Cp] (zeros in the channels past C), optionally times gate[n][c].  A block turns 64 channels x 64
// pixels through shared memory: 128-byte rows in, 16-byte units of eight channels out.  Bound: memory (one read, one write).
__global__ void __launch_bounds__(256) nchw_to_nhwc_kernel(const __half* __restrict__ x, const __half* __restrict__ gate, __half* __restrict__ y,
                                                           int c, int cp, int hw, int vec) {
    __shared__ __half tile[64][66];
    pdl_launch_dependents();
    pdl_wait();
    const int p0 = blockIdx.x * 64, c0 = blockIdx.y * 64;
    const int64_t img = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = p0 + lane * 2;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int ch = c0 + warp + 8 * i;
        __half2 v = __float2half2_rn(0.0f);
        if (ch < c) {
            const __half* src = x + (img * c + ch) * hw + p;
            if (vec && p + 1 < hw) v = *reinterpret_cast<const __half2*>(src);
            else {
                if (p < hw) v.x = src[0];
                if (p + 1 < hw) v.y = src[1];
            }
            if (gate) {
                const float gv = __half2float(gate[img * c + ch]);
                v = __floats2half2_rn(__low2float(v) * gv, __high2float(v) * gv);
            }
        }
        *reinterpret_cast<__half2*>(&tile[warp + 8 * i][lane * 2]) = v;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int unit = threadIdx.x + 256 * i, cg = unit & 7, px = unit >> 3;
        if (c0 + cg * 8 < cp && p0 + px < hw) {
            __align__(16) __half o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = tile[cg * 8 + j][px];
            *reinterpret_cast<uint4*>(y + (img * hw + p0 + px) * cp + c0 + cg * 8) = *reinterpret_cast<const uint4*>(o);
        }
    }
}

// Weights [M][C][kh][kw] -> [tap][chunk][row (padded)][kc] in the operand tile's swizzle; a thread makes eight channels.
__global__ void __launch_bounds__(256) conv_f16_pack_kernel(const __half* __restrict__ w, __half* __restrict__ out, int m, int c, int taps, int kc,
                                                            int chunks, int rows, int64_t units) {
    pdl_launch_dependents();
    pdl_wait();
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < units; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int per_row = kc / 8;
        const int u = static_cast<int>(i % per_row);
        int64_t rest = i / per_row;
        const int row = static_cast<int>(rest % rows);
        rest /= rows;
        const int chunk = static_cast<int>(rest % chunks), tap = static_cast<int>(rest / chunks);
        __align__(16) __half o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int ch = chunk * kc + u * 8 + j;
            o[j] = row < m && ch < c ? w[(static_cast<int64_t>(row) * c + ch) * taps + tap] : __float2half_rn(0.0f);
        }
        const int sw = kc == 64 ? (u ^ (row & 7)) : (kc == 32 ? (u ^ ((row >> 1) & 3)) : (u ^ ((row >> 2) & 1)));
        *reinterpret_cast<uint4*>(out + ((static_cast<int64_t>(tap) * chunks + chunk) * rows + row) * kc + sw * 8) = *reinterpret_cast<const uint4*>(o);
    }
}

int channels_per_step(int64_t cp) { return cp > 32 ? 64 : (cp > 16 ? 32 : 16); }

int pack_weights(const b200ml_ctx* ctx, const b200ml_conv_params* p, __half* out, cudaStream_t s) {
    const int64_t cp = ceil_div(p->c, 8) * 8;
    const int kc = channels_per_step(cp), chunks = (int)ceil_div(cp, kc);
    const int64_t rows = ceil_div(p->m, H_PACK_ROWS) * H_PACK_ROWS, taps = p->kh * p->kw;
    const int64_t units = taps * chunks * rows * (kc / 8), blocks = ceil_div(units, 256), cap = (int64_t)ctx->sm_count * 8;
    B200ML_CUDA(launch_pdl(conv_f16_pack_kernel, dim3((unsigned)(blocks < cap ? blocks : cap)), dim3(256), 0, s,
                           static_cast<const __half*>(p->weight), out, (int)p->m, (int)p->c, (int)taps, kc, chunks, (int)rows, units));
    return check_launch("conv_f16_pack");
}

template <int BN>
int launch_conv(const b200ml_ctx* ctx, const CUtensorMap& tx, ConvHArgs& g, cudaStream_t s) {
    auto kernel = conv_f16_kernel<BN>;
    static bool configured[64] = {};  // per instantiation and device
    if (!configured[ctx->device & 63]) {
        B200ML_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, H_PIPE_BYTES + 1280));
        configured[ctx->device & 63] = true;
    }
    g.tiles_m = (int32_t)ceil_div(g.m, BN);
    const int64_t tiles = (int64_t)g.tiles_w * g.tiles_h * g.tiles_n * g.tiles_m;
    B200ML_REQUIRE(tiles < (1ll << 27), "conv f16: too many tiles");
    const int stage_bytes = (H_BM + BN) * g.kc * 2;
    g.stages = H_PIPE_BYTES / stage_bytes < H_MAX_STAGES ? H_PIPE_BYTES / stage_bytes : H_MAX_STAGES;
    // Few tiles: the reduction is split while that adds CTAs, every CTA keeps four steps and a share of sixteen channels.
    g.split = 1;
    while (g.split < 4 && tiles * g.split * 2 <= ctx->sm_count && g.steps >= g.split * 8 && BN / (g.split * 2) >= 16) g.split *= 2;
    const int per = (int)ceil_div(g.steps, g.split);
    if (g.stages > per) g.stages = per;
    int pipe = g.stages * stage_bytes;
    if (pipe < H_MIN_PIPE_BYTES) pipe = H_MIN_PIPE_BYTES;
    if (g.split > 1 && pipe < BN * H_PART_LD * 4) pipe = (BN * H_PART_LD * 4 + 1023) & ~1023;
    g.pipe_bytes = pipe;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * g.split));
    cfg.blockDim = dim3(H_THREADS);
    cfg.dynamicSmemBytes = pipe + 1280;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = g.split, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    B200ML_CUDA(cudaLaunchKernelEx(&cfg, kernel, tx, g));
    return check_launch("conv_f16");
}

}  // namespace

// fp16, group 1, strides the TMA unit can make, enough work for the launches to pay (a 128 x 32 tile's worth of products).
bool conv_f16_applies(const b200ml_ctx* ctx, const b200ml_conv_params* p, int64_t oh, int64_t ow) {
    if (p->dtype != B200ML_F16 || p->group != 1 || !ctx->encode_tiled) return false;
    if (p->stride_h > 8 || p->stride_w > 8 || p->pad_top > 1024 || p->pad_left > 1024) return false;
    if (p->n * p->m * oh * ow * p->c * p->kh * p->kw < (1ll << 19)) return false;
    if ((p->act & (B200ML_CONV_X_NHWC | B200ML_CONV_Y_NHWC)) && (!aligned16(p->x) || !aligned16(p->y))) return false;
    const int64_t cp = ceil_div(p->c, 8) * 8;
    return cp * p->h * p->w * 2 <= ctx->workspace_bytes / 2;  // at least one image fits beside run-time weights
}

int64_t conv_f16_pack_bytes(const b200ml_conv_params* p) {
    const int64_t cp = ceil_div(p->c, 8) * 8;
    const int kc = channels_per_step(cp);
    return p->kh * p->kw * ceil_div(cp, kc) * ceil_div(p->m, H_PACK_ROWS) * H_PACK_ROWS * kc * 2;
}

int conv_f16_pack(const b200ml_ctx* ctx, const b200ml_conv_params* p, void* packed, cudaStream_t s) {
    return pack_weights(ctx, p, static_cast<__half*>(packed), s);
}

int conv_f16(const b200ml_ctx* ctx, const b200ml_conv_params* p, int64_t oh, int64_t ow, cudaStream_t s) {
    const int64_t cp = ceil_div(p->c, 8) * 8;
    const bool x_nhwc = (p->act & B200ML_CONV_X_NHWC) != 0, y_nhwc = (p->act & B200ML_CONV_Y_NHWC) != 0;
    B200ML_REQUIRE(!(x_nhwc || y_nhwc) || !p->pool_sum, "conv f16: no pooled output of channels-last tensors");
    B200ML_REQUIRE(!x_nhwc || (p->c % 8 == 0 && !p->gate), "conv f16: a channels-last X needs a multiple of 8 channels and no gate");
    B200ML_REQUIRE(!y_nhwc || p->m % 8 == 0, "conv f16: a channels-last Y needs a multiple of 8 channels");
    char* ws = static_cast<char*>(ctx->workspace);
    int64_t room = ctx->workspace_bytes;
    const __half* w = static_cast<const __half*>(p->packed_weight);
    if (!w) {
        const int64_t bytes = ceil_div(conv_f16_pack_bytes(p), 1024) * 1024;
        if (bytes > room / 2) return fail(B200ML_ERR_WORKSPACE, "conv f16: the weights (%lld bytes laid out) exceed the workspace", (long long)bytes);
        const int rc = pack_weights(ctx, p, reinterpret_cast<__half*>(ws), s);
        if (rc) return rc;
        w = reinterpret_cast<const __half*>(ws);
        ws += bytes, room -= bytes;
    }
    // images in pieces whose channels-last copy fits the workspace
    const int64_t image = cp * p->h * p->w;
    int64_t piece = p->n;
    if (!x_nhwc) {
        const int64_t fit = room / (image * 2);
        piece = fit < p->n ? fit : p->n;
        if (piece > 65535) piece = 65535;
        piece = ceil_div(p->n, ceil_div(p->n, piece));
    }
    for (int64_t n0 = 0; n0 < p->n; n0 += piece) {
        const int64_t n = p->n - n0 < piece ? p->n - n0 : piece;
        const __half* x = static_cast<const __half*>(p->x) + n0 * p->c * p->h * p->w;
        if (!x_nhwc) {
            __half* turned = reinterpret_cast<__half*>(ws);
            const int64_t hw = p->h * p->w;
            const int vec = hw % 2 == 0 && (reinterpret_cast<uintptr_t>(x) & 3) == 0 ? 1 : 0;
            B200ML_REQUIRE(ceil_div(cp, 64) <= 65535, "conv f16: too many channels");
            B200ML_CUDA(launch_pdl(nchw_to_nhwc_kernel, dim3((unsigned)ceil_div(hw, 64), (unsigned)ceil_div(cp, 64), (unsigned)n), dim3(256), 0, s, x,
                                   p->gate ? static_cast<const __half*>(p->gate) + n0 * p->c : nullptr, turned, (int)p->c, (int)cp, (int)hw, vec));
            const int rc = check_launch("nchw_to_nhwc");
            if (rc) return rc;
            x = turned;
        }
        ConvHArgs g{};
        g.w = w;
        g.bias = static_cast<const __half*>(p->bias);
        g.residual = p->residual ? static_cast<const __half*>(p->residual) + n0 * p->m * oh * ow : nullptr;
        g.y = static_cast<__half*>(p->y) + n0 * p->m * oh * ow;
        g.n = (int32_t)n, g.m = (int32_t)p->m, g.oh = (int32_t)oh, g.ow = (int32_t)ow;
        g.kc = channels_per_step(cp), g.chunks = (int32_t)ceil_div(cp, g.kc);
        g.steps = (int32_t)(p->kh * p->kw) * g.chunks, g.kw = (int32_t)p->kw;
        g.packed_rows = (int32_t)(ceil_div(p->m, H_PACK_ROWS) * H_PACK_ROWS);
        g.sh = (int32_t)p->stride_h, g.sw = (int32_t)p->stride_w, g.dh = (int32_t)p->dil_h, g.dw = (int32_t)p->dil_w;
        g.pad_top = (int32_t)p->pad_top, g.pad_left = (int32_t)p->pad_left;
        g.act = p->act & (B200ML_EPI_RELU | B200ML_EPI_GELU | B200ML_EPI_SWISH);
        g.y_nhwc = y_nhwc ? 1 : 0;
        g.status = ctx->status_dev;
        // the pixel box that covers the output with the fewest tiles; an element stride limits its extent (256 source elements)
        int64_t best = INT64_MAX;
        const int64_t max_w = ow < 128 ? ow : 128;
        for (int64_t wb = max_w; wb >= 1; --wb) {
            if ((wb - 1) * p->stride_w + 1 > 256) continue;
            int64_t hb = oh < 128 / wb ? oh : 128 / wb;
            while ((hb - 1) * p->stride_h + 1 > 256) --hb;
            int64_t nb = wb == ow && hb == oh ? 128 / (wb * hb) : 1;
            if (nb > n) nb = n;
            const int64_t tiles = ceil_div(ow, wb) * ceil_div(oh, hb) * ceil_div(n, nb);
            if (tiles < best) best = tiles, g.wb = (int32_t)wb, g.hb = (int32_t)hb, g.nb = (int32_t)nb;
        }
        g.tiles_w = (int32_t)ceil_div(ow, g.wb), g.tiles_h = (int32_t)ceil_div(oh, g.hb), g.tiles_n = (int32_t)ceil_div(n, g.nb);
        const cuuint64_t dims[4] = {(cuuint64_t)cp, (cuuint64_t)p->w, (cuuint64_t)p->h, (cuuint64_t)n};
        const cuuint64_t strides[3] = {(cuuint64_t)cp * 2, (cuuint64_t)(cp * p->w) * 2, (cuuint64_t)image * 2};
        const cuuint32_t box[4] = {(cuuint32_t)g.kc, (cuuint32_t)((g.wb - 1) * p->stride_w + 1), (cuuint32_t)((g.hb - 1) * p->stride_h + 1), (cuuint32_t)g.nb};
        const cuuint32_t step[4] = {1, (cuuint32_t)p->stride_w, (cuuint32_t)p->stride_h, 1};
        CUtensorMap tx;
        CUresult r = encode_tiled_cached(ctx, &tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, dims, strides, box,
                                         g.kc == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : (g.kc == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B), step);
        if (r != CUDA_SUCCESS) return fail(B200ML_ERR_CUDA, "cuTensorMapEncodeTiled(X channels-last, fp16) failed with CUresult %d", (int)r);
        // Narrower channel blocks where the wide ones would leave half of the CTA slots idle.
        const int64_t pixel_tiles = (int64_t)g.tiles_w * g.tiles_h * g.tiles_n;
        int rc;
        if (p->m <= 32) rc = launch_conv<32>(ctx, tx, g, s);
        else if (p->m <= 64 || pixel_tiles * ceil_div(p->m, 128) < ctx->sm_count) rc = launch_conv<64>(ctx, tx, g, s);
        else rc = launch_conv<128>(ctx, tx, g, s);
        if (rc) return rc;
    }
    return B200ML_OK;
}

}  // namespace b200ml
