// k_wgrad.cu -- weight gradient of a 3x3 convolution (stride 1, zero padding 1)
// of NHWC BF16 tensors on the 5th-generation tensor cores.
//
// dW[co][tap][ci] = sum over pixels of dZ[p][co] * X[p + shift(tap)][ci]: for a
// row of three taps one GEMM with M = output channels, N = 3 x input channels and
// K = pixels.  Both operands lie in memory with their channels contiguous, i.e.
// MN-major, and are taken as TMA brings them: boxes of {16, 32 or 64 channels,
// 64 pixels} with the 32, 64 or 128-byte swizzle, three X boxes at the taps' pixel
// offsets (rows and columns outside the image are zero-filled, which is the
// padding).  M is always 128: where a layer has fewer output channels the
// descriptor repeats them (leading offset 0) and the repeated rows are dropped.
//
// CTA (split, tap row, channel chunk) walks its 64-pixel tiles.  The tensor core
// adds into its accumulator by truncation, so a long sum there drifts towards
// zero (128 steps: 1.6e-6 of the result, a CUDA-core FP32 sum 6e-7).  A tile's
// four steps are therefore all that is summed in TMEM: eight epilogue warps add
// each tile's accumulator to FP32 registers (round to nearest) while the next
// tile runs, and the CTA writes one partial; k_reduce_parts adds the splits.
// Against a 64-bit sum the result is as close as the CUDA-core kernel's or
// closer.  A ring of stages overlaps the copies with the MMAs; every wait is
// bounded, past the bound the kernel sets the network's failure flag and skips
// its remaining work.
//
// What bounds it: the CUDA-core kernel it replaced spent one FP32 multiply-add
// per product; here it is the L2 traffic of the nine shifted copies of X and
// three of dZ.
#include "nn_conv.cuh"
#include "tc_nn.h"

namespace nn {

constexpr int kWgTile = 64;  // pixels of a stage
constexpr int kWgMax = 2048; // pixels of a split

struct WgradArgs {
    int nb, H, W, bx, by;       // bx * by = 64 pixels
    int cout, cin;              // channels of dZ and of dW
    int x_off, cc;              // first channel of X in its tensor, channels of a chunk (N)
    int za, zn;                 // channels and number of the dZ boxes
    int tiles, per_split;       // 64-pixel tiles in all and of a split
    int stages;
    float* part;                // [split][cout][9][cin]
    int* fail;
    const int* test_flag;       // timeout-path test, as ConvArgs
};

// 16 accumulator columns of this warp's lanes (the caller waits for the loads)
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(saddr(b)) : "memory");
}

// CC channels of X; two accumulators where they fit the 512 TMEM columns
template <int CC>
__global__ void __launch_bounds__(320, 1) k_wgrad(const __grid_constant__ CUtensorMap zmap,
                                                  const __grid_constant__ CUtensorMap xmap, WgradArgs a) {
    constexpr int NCOL = 3 * CC, NB = 2 * NCOL <= 512 ? 2 : 1;
    constexpr uint32_t kCols = NB * NCOL <= 128 ? 128 : (NB * NCOL <= 256 ? 256 : 512);
    constexpr int HALF = NCOL / 2;  // columns of an epilogue warp
    constexpr int XA = CC % 64 == 0 ? 64 : (CC % 32 == 0 ? 32 : 16), XN = CC / XA;
    constexpr int xrow = XA * 2, xbox = kWgTile * xrow, xtile = XN * xbox;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[8], empty[8], accf[2], acce[2];
    __shared__ uint32_t tmem_base;
    __shared__ int bad;
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dy = (int)blockIdx.y - 1, c0 = (int)blockIdx.z * CC;
    const int t0 = (int)blockIdx.x * a.per_split, nt = min(a.per_split, a.tiles - t0);
    const int zrow = a.za * 2, zbox = kWgTile * zrow;  // bytes
    const int st_bytes = a.zn * zbox + 3 * xtile;
    if (tid == 0) {
        bad = 0;
        for (int s = 0; s < a.stages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&accf[b], 1);
            mbar_init(&acce[b], 8);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tmem_base)),
                     "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    if (a.test_flag != nullptr) {
        if (tid == 0) {
            long it = 0;
            while (*(volatile const int*)a.test_flag == 0 && ++it <= (1l << 14)) {
            }
            bad = 1;
        }
        __syncthreads();
    }
    bool fail = false;
    if (bad) {
        // (timeout-path test: no copy issued, nothing to wait for)
    } else if (warp == 0) {
        if (lane == 0) {
            const int tiles_x = a.W / a.bx, tiles_y = a.H / a.by;
            for (int i = 0; i < nt; i++) {
                const int s = i % a.stages;
                if (i >= a.stages && !mbar_wait(&empty[s], ((i / a.stages) - 1) & 1)) { fail = true; break; }
                int t = t0 + i;
                const int x0 = (t % tiles_x) * a.bx;
                t /= tiles_x;
                const int y0 = (t % tiles_y) * a.by, n = t / tiles_y;
                unsigned char* zs = smem + (size_t)s * st_bytes;
                unsigned char* xs = zs + a.zn * zbox;
                mbar_expect_tx(&full[s], (uint32_t)st_bytes);
                for (int q = 0; q < a.zn; q++) tma_load4(zs + q * zbox, &zmap, q * a.za, x0, y0, n, &full[s]);
                for (int d = 0; d < 3; d++)
                    for (int q = 0; q < XN; q++)
                        tma_load4(xs + d * xtile + q * xbox, &xmap, a.x_off + c0 + q * XA, x0 + d - 1, y0 + dy, n,
                                  &full[s]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // both operands MN-major (bits 15, 16)
            constexpr uint32_t idesc = idesc_bf16(128, CC) | 1u << 15 | 1u << 16;
            for (int i = 0; i < nt; i++) {
                const int s = i % a.stages, b = i % NB, use = i / NB;
                // the epilogue has read the buffer's previous tile
                if (use > 0 && !mbar_wait(&acce[b], (use - 1) & 1)) { fail = true; break; }
                if (!mbar_wait(&full[s], (i / a.stages) & 1)) { fail = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t zs = saddr(smem + (size_t)s * st_bytes), xs = zs + a.zn * zbox;
#pragma unroll 1
                for (int d = 0; d < 3; d++)
                    for (int k = 0; k < kWgTile / 16; k++) {
                        // 128 output channels: the boxes in turn, or one box again and again
                        const uint64_t ad = smem_desc_swizzled(zs + k * 16 * zrow, a.cout == 128 ? zbox : 0, 8 * zrow, zrow);
                        const uint64_t bd = smem_desc_swizzled(xs + d * xtile + k * 16 * xrow, xbox, 8 * xrow, xrow);
                        umma_bf16(tmem + (uint32_t)(b * NCOL + d * CC), ad, bd, idesc, k > 0 ? 1u : 0u);
                    }
                umma_commit(&empty[s]);
                umma_commit(&accf[b]);
            }
        }
    } else {
        // epilogue, warps 2..9: TMEM lanes 32 (warp % 4) .. + 31 are output
        // channels; each warp of a pair takes half of the columns
        const int q = warp & 3, half = (warp - 2) / 4, co = q * 32 + lane;
        const bool mine = q * 32 < a.cout;
        float acc[HALF];
#pragma unroll
        for (int c = 0; c < HALF; c++) acc[c] = 0.f;
        for (int i = 0; i < nt; i++) {
            const int b = i % NB;
            const bool ok = __all_sync(0xffffffffu, mbar_wait(&accf[b], (i / NB) & 1) ? 1 : 0) != 0;
            if (!ok) { fail = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (mine) {
                const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * NCOL + half * HALF);
                if constexpr (HALF % 16 == 0) {
#pragma unroll
                    for (int c = 0; c < HALF; c += 16) {
                        uint32_t r[16];
                        tmem_ld16(at + c, r);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; j++) acc[c + j] += __uint_as_float(r[j]);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < HALF; c += 8) {
                        float v[8];
                        tmem_ld8(at + c, v);
#pragma unroll
                        for (int j = 0; j < 8; j++) acc[c + j] += v[j];
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&acce[b]);
        }
        if (mine && !fail) {
#pragma unroll
            for (int c = 0; c < HALF; c += 4) {
                const int col = half * HALF + c, d = col / CC, ci = c0 + col % CC;
                float* out = a.part + (((size_t)blockIdx.x * a.cout + co) * 9 + blockIdx.y * 3 + d) * a.cin + ci;
                if (a.cin >= 16) *reinterpret_cast<float4*>(out) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
                else
                    for (int j = 0; j < 4; j++)
                        if (ci + j < a.cin) out[j] = acc[c + j];
            }
        }
    }
    if (fail) atomicExch(&bad, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (bad && tid == 0) atomicExch(a.fail, 1);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
}

template <int CC>
static int launch_cc(cudaStream_t s, const CUtensorMap& zmap, const CUtensorMap& xmap, const WgradArgs& a, dim3 grid,
                     int smem) {
    static PerDevice set;
    if (set.get([] {
            return cudaFuncSetAttribute(k_wgrad<CC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 202 * 1024) ==
                           cudaSuccess
                       ? 0
                       : -1;
        }) != 0)
        return 4;
    k_wgrad<CC><<<grid, 320, smem, s>>>(zmap, xmap, a);
    tc_note_launch();
    return cudaGetLastError() == cudaSuccess ? 0 : 5;
}

// 64-pixel tiles of a split and the number of splits: at most kWgMax pixels
// each, and enough splits to fill the GPU
static void split_of(int tiles, int ctas, int nsm, int* per, int* splits) {
    int s = (tiles * kWgTile + kWgMax - 1) / kWgMax;
    const int want = (nsm + ctas - 1) / ctas;
    if (s < want) s = want < tiles ? want : tiles;
    *per = (tiles + s - 1) / s;
    *splits = (tiles + *per - 1) / *per;
}

// channels of a chunk: a CTA's accumulators and their register copies fit
static int chunk_of(int cin_p) { return cin_p <= 32 || cin_p == 96 ? cin_p : 64; }

}  // namespace nn

using namespace nn;

// number of splits of a layer's weight gradient on nb images (partials of
// cout * 9 * cin floats each)
int wgrad_splits(int nb, int H, int W, int cin) {
    const int cin_p = (cin + 15) / 16 * 16, chunks = cin_p / chunk_of(cin_p);
    int per, s;
    split_of(nb * H * W / kWgTile, 3 * chunks, tc_sm_count(), &per, &s);
    return s;
}

int wgrad_launch(cudaStream_t s, const __nv_bfloat16* x, int x_tot, int x_off, int cin, const __nv_bfloat16* dz,
                 int cout, int nb, int H, int W, float* part, int* fail, const int* test_flag) {
    const int cin_p = (cin + 15) / 16 * 16;
    if (!(cout == 32 || cout == 64 || cout == 128) || (cin % 16 && cin >= 16) || x_off % 8) return 1;
    WgradArgs a;
    a.nb = nb; a.H = H; a.W = W;
    a.bx = W < kWgTile ? W : kWgTile;
    if (kWgTile % a.bx || W % a.bx) return 1;
    a.by = kWgTile / a.bx;
    if (H % a.by) return 1;
    a.cout = cout; a.cin = cin; a.x_off = x_off;
    a.cc = chunk_of(cin_p);
    if (cin_p % a.cc || !(a.cc == 16 || a.cc == 32 || a.cc == 64 || a.cc == 96)) return 1;
    const int xa = a.cc % 64 == 0 ? 64 : (a.cc % 32 == 0 ? 32 : 16);
    a.za = cout < 64 ? cout : 64;
    a.zn = cout / a.za;
    a.tiles = nb * H * W / kWgTile;
    int splits;
    split_of(a.tiles, 3 * (cin_p / a.cc), tc_sm_count(), &a.per_split, &splits);
    const int st_bytes = kWgTile * 2 * (cout + 3 * a.cc);
    a.stages = (200 * 1024) / st_bytes;
    if (a.stages > 8) a.stages = 8;
    if (a.stages > a.per_split) a.stages = a.per_split;
    a.part = part; a.fail = fail; a.test_flag = test_flag;
    CUtensorMap zmap, xmap;
    if (!nn_tensor_map(&zmap, dz, nb, H, W, cout, a.za, a.bx, a.by, a.za * 2) ||
        !nn_tensor_map(&xmap, x, nb, H, W, x_tot, xa, a.bx, a.by, xa * 2))
        return 3;
    const int smem = a.stages * st_bytes + 1024;
    const dim3 grid((unsigned)splits, 3, (unsigned)(cin_p / a.cc));
    switch (a.cc) {
        case 16: return launch_cc<16>(s, zmap, xmap, a, grid, smem);
        case 32: return launch_cc<32>(s, zmap, xmap, a, grid, smem);
        case 64: return launch_cc<64>(s, zmap, xmap, a, grid, smem);
        default: return launch_cc<96>(s, zmap, xmap, a, grid, smem);
    }
}
