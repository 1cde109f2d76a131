// A small convolutional U-Net that predicts a correction to the multigrid's
// initial guess, with its training on the GPU.
//
// The network sees the residual r = b - A z0 of the time-extrapolated guess z0
// (normalised by its RMS, on a grid coarsened by an integer factor) and
// predicts delta ~ A^-1 r, the error of z0; z0 + delta starts the V-cycles,
// which still iterate to tolerance. Layers (all 3x3, zero padding, NHWC BF16
// activations, FP32 accumulation, ReLU except the last):
//   L1 16->16, L2 16->16 = e1 | pool | L3 16->32, L4 32->32 = e2 | pool |
//   L5 32->64, L6 64->64 = e3 | pool | L7 64->64, L8 64->64 | up |
//   L9 64->64 (+e3), L10 64->32 | up | L11 32->32 (+e2), L12 32->16 | up |
//   L13 16->16 (+e1), L14 16->16 (linear; channel 0 is the output)
// The input has one channel, padded to 16. Skips are added after the
// convolution of the upsampled tensor, before the ReLU.
//
// Convolutions are implicit GEMMs on the tensor cores (mma.sync m16n8k16,
// BF16 operands, FP32 accumulators): M = pixels (a warp owns 16 pixels of one
// image row), N = output channels, K = 9 taps x input channels. The input
// gradient is the same convolution with flipped, transposed weights; the
// weight gradient is a second GEMM (output channels x input channels over
// pixels) accumulated per CTA and added atomically.
#include "vdi_internal.hh"

#include <cuda_bf16.h>
#include <cstdint>
#include <type_traits>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace vdi {
namespace unet {

typedef __nv_bfloat16 bf16;

// ------------------------------------------------------------ tensor cores
__device__ __forceinline__ void mma_bf16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack2(bf16 lo, bf16 hi) {
    return uint32_t(__bfloat16_as_ushort(lo)) | (uint32_t(__bfloat16_as_ushort(hi)) << 16);
}

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<bf16>(bf16 v) { return __bfloat162float(v); }

template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ bf16 from_f<bf16>(float v) { return __float2bfloat16(v); }

enum { SRC_DIRECT = 0, SRC_UP2 = 1, SRC_POOL2 = 2 };

/** Value of the convolution input at (y,x) of the operating grid (H x W):
 * the source read directly, upsampled x2 (nearest) or pooled 2x2 (mean);
 * zero outside. mask (same shape as the source) zeroes entries whose mask is
 * not positive (the ReLU derivative in the backward pass). */
template <typename TIN>
__device__ __forceinline__ float src_at(const TIN* src, const bf16* mask, int mode, int H, int W, int C, int b, int y,
                                        int x, int c) {
    if (y < 0 || y >= H || x < 0 || x >= W) return 0.f;
    if (mode == SRC_DIRECT) {
        size_t k = ((size_t(b) * H + y) * W + x) * C + c;
        float v = to_f(src[k]);
        return (mask && !(to_f(mask[k]) > 0.f)) ? 0.f : v;
    }
    if (mode == SRC_UP2) {
        int Hs = H >> 1, Ws = W >> 1;
        size_t k = ((size_t(b) * Hs + (y >> 1)) * Ws + (x >> 1)) * C + c;
        return to_f(src[k]);
    }
    int Hs = H * 2, Ws = W * 2;
    float s = 0.f;
    for (int dy = 0; dy < 2; dy++)
        for (int dx = 0; dx < 2; dx++) s += to_f(src[((size_t(b) * Hs + 2 * y + dy) * Ws + 2 * x + dx) * C + c]);
    return 0.25f * s;
}

template <typename TIN, typename TOUT>
struct ConvArgs {
    const TIN* src;        // input source (layout depends on mode)
    const bf16* mask;      // optional ReLU mask for the source (same shape)
    int mode;
    const bf16* w;         // [9][COUT][CIN]
    const float* bias;     // optional [COUT]
    const bf16* resid;     // optional [B][H][W][COUT] added before the activation
    int relu;
    TOUT* out;             // [B][H][W][COUT]
    int B, H, W;
};

constexpr int TPX = 16, TPY = 8;   // pixel tile: 8 rows of 16 pixels, one warp per row

/** 3x3 convolution on the tensor cores. */
template <int CIN, int COUT, typename TIN, typename TOUT>
__global__ void __launch_bounds__(256) conv3x3_k(ConvArgs<TIN, TOUT> a) {
    constexpr int CS = CIN + 8;             // padded pixel stride (bf16) of the input patch
    constexpr int WS = CIN + 8;             // padded stride of a weight row
    constexpr int PW = TPX + 2, PH = TPY + 2;
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* patch = reinterpret_cast<bf16*>(smem);              // [PH][PW][CS]
    bf16* wsm = patch + PH * PW * CS;                         // [9][COUT][WS]
    const int tilesx = (a.W + TPX - 1) / TPX;
    const int bx = blockIdx.x % tilesx, by = blockIdx.x / tilesx;
    const int b = blockIdx.y;
    const int x0 = bx * TPX, y0 = by * TPY;
    for (int t = threadIdx.x; t < PH * PW * CIN; t += blockDim.x) {
        int c = t % CIN, p = t / CIN;
        int px = p % PW, py = p / PW;
        float v = src_at(a.src, a.mask, a.mode, a.H, a.W, CIN, b, y0 + py - 1, x0 + px - 1, c);
        patch[(py * PW + px) * CS + c] = __float2bfloat16(v);
    }
    for (int t = threadIdx.x; t < 9 * COUT * CIN; t += blockDim.x) {
        int c = t % CIN, r = t / CIN;
        wsm[r * WS + c] = a.w[t];
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    float acc[COUT / 8][4];
#pragma unroll
    for (int n = 0; n < COUT / 8; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll
    for (int tap = 0; tap < 9; tap++) {
        const int ky = tap / 3, kx = tap % 3;
        const bf16* prow = patch + ((warp + ky) * PW + kx) * CS;   // pixel 0 of this warp's row, shifted by the tap
        const bf16* wt = wsm + tap * COUT * WS;
#pragma unroll
        for (int kc = 0; kc < CIN / 16; kc++) {
            const int k0 = kc * 16 + 2 * tq;
            uint32_t a0 = *reinterpret_cast<const uint32_t*>(prow + g * CS + k0);
            uint32_t a1 = *reinterpret_cast<const uint32_t*>(prow + (g + 8) * CS + k0);
            uint32_t a2 = *reinterpret_cast<const uint32_t*>(prow + g * CS + k0 + 8);
            uint32_t a3 = *reinterpret_cast<const uint32_t*>(prow + (g + 8) * CS + k0 + 8);
#pragma unroll
            for (int n = 0; n < COUT / 8; n++) {
                const bf16* wr = wt + (n * 8 + g) * WS + k0;
                uint32_t b0 = *reinterpret_cast<const uint32_t*>(wr);
                uint32_t b1 = *reinterpret_cast<const uint32_t*>(wr + 8);
                mma_bf16(acc[n], a0, a1, a2, a3, b0, b1);
            }
        }
    }
    const int y = y0 + warp;
    if (y >= a.H) return;
#pragma unroll
    for (int n = 0; n < COUT / 8; n++) {
        const int co = n * 8 + 2 * tq;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int x = x0 + g + 8 * h;
            if (x >= a.W) continue;
            size_t k = ((size_t(b) * a.H + y) * a.W + x) * COUT + co;
            float v0 = acc[n][2 * h], v1 = acc[n][2 * h + 1];
            if (a.bias) {
                v0 += a.bias[co];
                v1 += a.bias[co + 1];
            }
            if (a.resid) {
                v0 += __bfloat162float(a.resid[k]);
                v1 += __bfloat162float(a.resid[k + 1]);
            }
            if (a.relu) {
                v0 = fmaxf(v0, 0.f);
                v1 = fmaxf(v1, 0.f);
            }
            a.out[k] = from_f<TOUT>(v0);
            a.out[k + 1] = from_f<TOUT>(v1);
        }
    }
}

/** Eight channels (from c, a multiple of 8) of the convolution input at
 * (y, x) of the operating grid, as src_at gives them; zero outside. */
__device__ __forceinline__ uint4 src8_at(const bf16* src, int mode, int H, int W, int C, int b, int y, int x, int c) {
    if (y < 0 || y >= H || x < 0 || x >= W) return make_uint4(0, 0, 0, 0);
    if (mode == SRC_DIRECT) return *reinterpret_cast<const uint4*>(src + ((size_t(b) * H + y) * W + x) * C + c);
    if (mode == SRC_UP2)
        return *reinterpret_cast<const uint4*>(src + ((size_t(b) * (H >> 1) + (y >> 1)) * (W >> 1) + (x >> 1)) * C + c);
    float s[8];
#pragma unroll
    for (int k = 0; k < 8; k++) s[k] = 0.f;
#pragma unroll
    for (int d = 0; d < 4; d++) {
        const uint4 v = *reinterpret_cast<const uint4*>(
            src + ((size_t(b) * H * 2 + 2 * y + (d >> 1)) * W * 2 + 2 * x + (d & 1)) * C + c);
        const bf16* e = reinterpret_cast<const bf16*>(&v);
#pragma unroll
        for (int k = 0; k < 8; k++) s[k] += __bfloat162float(e[k]);
    }
    uint4 r;
    bf16* e = reinterpret_cast<bf16*>(&r);
#pragma unroll
    for (int k = 0; k < 8; k++) e[k] = __float2bfloat16(0.25f * s[k]);
    return r;
}

// ------------------------------------------- Blackwell tensor-core path
// The same convolution on the fifth-generation tensor cores (the default
// path; VDI_UNET_TC=0 keeps the mma.sync kernel above): tcgen05.mma with
// both operands in shared memory and the FP32 accumulator in tensor memory.
// One CTA of four warps takes a row segment of TC_M = 128 output pixels
// (the MMA's M), so the A operand of tap (dy, dx) is a window of the staged
// input rows shifted by whole pixels: a pixel's 8-channel chunk is one
// 16-byte core-matrix row, 8 consecutive pixels one 8 x 16-byte core
// matrix, and the operand needs no copy per tap. The weights, already stored
// [tap][cout][cin], are K-major B operands. A CTA stages the weights once and
// then walks a contiguous run of segments, consecutive rows of one segment
// where it can, keeping the input rows in a ring of four: a new segment
// stages one row (BF16 sources read as they are by asynchronous 16-byte
// copies), while the tensor cores work on the previous one. Several CTAs
// share an SM (tc_blocks), so one's staging and epilogue overlap another's
// MMAs. Each segment is 9 * CIN/16 MMAs (K = 16 each) into one accumulator, read back
// with tcgen05.ld for the bias, skip-add, ReLU epilogue.
// A launch on one image is bound by latency (8 to 14 us each at 256 x 512,
// where the bytes take 1): so the weights and every row that is read as it
// is, upsampled ones too, come by asynchronous copies through L1 (the CTAs of
// an SM share the weights; past L1 the 16-channel layers took 14 us in place
// of 11), the skip's values are fetched while the MMAs run, and a forward
// call's launches set up while the ones before them run. A forward call of 1
// image takes 143 us with these, 240 without; a training step of 8 2.42 and
// 2.57 ms. CTAs of two launches then share an SM: shared memory holds at most
// four, of 64 tensor-memory columns at most, so that no allocation of columns
// waits on a launch that waits itself.
namespace tc {

constexpr int TC_M = 128;            // output pixels per segment (MMA M)
constexpr int TC_PX = TC_M + 2;      // staged pixels per input row (one halo pixel each side)
constexpr int TC_THREADS = 256;     // all stage rows, the first four warps read the accumulator
constexpr int TC_RING = 4;           // staged input rows: three in use, the next being loaded

__device__ int g_timeout;            // set when a bounded wait gave up

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

/** Shared-memory matrix descriptor of a K-major operand without swizzle:
 * core matrices of 8 rows x 16 bytes, lbo the byte distance between the two
 * core matrices of one K = 16 step, sbo between consecutive 8-row groups. */
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = uint64_t((addr >> 4) & 0x3FFFu);
    d |= uint64_t((lbo >> 4) & 0x3FFFu) << 16;
    d |= uint64_t((sbo >> 4) & 0x3FFFu) << 32;
    d |= uint64_t(1) << 46;          // descriptor version of sm_100
    return d;                         // base offset 0, no swizzle
}

/** Instruction descriptor of kind::f16: BF16 A and B, both K-major, FP32 D,
 * M x N. */
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16_ss(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
        :
        : "r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(z), "r"(z), "r"(z), "r"(z));
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

/** Waits for the mbarrier phase with a time limit (about 0.5 s of SM
 * clock); false if it gave up. */
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
    const long long t0 = clock64();
    while (true) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > 1000000000LL) return false;
    }
}

/** Asynchronous 16-byte copy to shared memory of `bytes` bytes (16, or 0 for
 * zeros). */
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

/** 16 consecutive FP32 accumulator columns of this thread's TMEM lane. */
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = __uint_as_float(r[k]);
}

/** Dynamic shared memory of conv3x3_tc: the weights and the ring of staged
 * input rows, plus TC_PAD bytes that no descriptor is meant to reach. The pad
 * keeps every address an operand could span inside the CTA's own
 * allocation even if the K and M core-matrix strides were interpreted the
 * other way round (the A operand would then reach 15 x 2080 + 128 bytes
 * past its start): a misread operand gives wrong numbers, which the tests
 * catch, rather than an access outside the CTA's shared memory. */
constexpr size_t TC_PAD = 32 * 1024;
template <int CIN, int COUT>
constexpr size_t tc_smem() {
    return size_t(9) * (CIN / 8) * COUT * 16 + size_t(TC_RING) * (CIN / 8) * TC_PX * 16 + TC_PAD;
}

/** CTAs of conv3x3_tc that an SM holds: by shared memory, at most four (of 32
 * or 64 tensor-memory columns each). The occupancy query answers one. */
template <int CIN, int COUT>
constexpr int tc_blocks() {
    const int by_smem = int(size_t(227 * 1024) / (tc_smem<CIN, COUT>() + 2048));
    return by_smem < 1 ? 1 : (by_smem > 4 ? 4 : by_smem);
}

template <int CIN, int COUT, typename TIN, typename TOUT>
__global__ void __launch_bounds__(TC_THREADS) conv3x3_tc(ConvArgs<TIN, TOUT> a) {
    constexpr int KC = CIN / 8;                              // 16-byte channel chunks
    constexpr uint32_t CHUNKB = uint32_t(TC_PX) * 16;        // one chunk of one staged row
    constexpr uint32_t ROWB = uint32_t(KC) * CHUNKB;         // one staged row, all chunks
    constexpr uint32_t WTAPB = uint32_t(KC) * COUT * 16;     // one tap of weights
    constexpr int TCOLS = COUT < 32 ? 32 : COUT;             // TMEM columns (a power of two, >= 32)
    static_assert(CIN % 16 == 0 && COUT % 16 == 0 && COUT <= 256, "tcgen05 shape");
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* wsm = smem;                               // [9][KC][COUT][8] bf16
    unsigned char* rows = smem + 9 * WTAPB;                  // ring [TC_RING][KC][TC_PX][8] bf16
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_slot;
    __shared__ float bias_s[COUT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // the next launch may set up beside this one; it waits below for this
    // one's results
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll 4
    for (int q = tid; q < 9 * COUT * KC; q += TC_THREADS) {
        const int kc = q % KC, co = (q / KC) % COUT, t = q / (KC * COUT);
        cp_async16(wsm + (uint32_t(t) * KC + kc) * COUT * 16 + co * 16, a.w + (size_t(t) * COUT + co) * CIN + kc * 8,
                   16);
    }
    if (tid < COUT) bias_s[tid] = a.bias ? a.bias[tid] : 0.f;
    const uint32_t bar_a = smem_u32(&bar);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(TCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    constexpr uint32_t IDESC = idesc_bf16(TC_M, COUT);
    const int segs = (a.W + TC_M - 1) / TC_M;
    // tasks in (segment, image, row) order; each CTA takes a contiguous run,
    // so that consecutive tasks are usually consecutive rows of one segment
    const long tasks = long(a.B) * a.H * segs;
    const long t0 = tasks * blockIdx.x / gridDim.x, t1 = tasks * (blockIdx.x + 1) / gridDim.x;
    // input row yy of image b (pixels x0-1 .. x0+TC_M) into ring slot
    // (yy + 1) % TC_RING, as 16-byte channel chunks
    auto stage = [&](int b, int yy, int x0) {
        unsigned char* dst = rows + uint32_t((yy + 1 + TC_RING) % TC_RING) * ROWB;
        const bool rin = yy >= 0 && yy < a.H;
        if constexpr (std::is_same<TIN, bf16>::value) {
            if (a.mode != SRC_POOL2) {
                const int up = a.mode == SRC_UP2;   // a pixel of the source covers 2 x 2
                const bf16* row = a.src + (size_t(b) * (a.H >> up) + (rin ? yy >> up : 0)) * (a.W >> up) * CIN;
                for (int q = tid; q < KC * TC_PX; q += TC_THREADS) {
                    const int kc = q % KC, px = q / KC, xx = x0 + px - 1;
                    const bool in = rin && xx >= 0 && xx < a.W;
                    // zero-filled outside the image
                    cp_async16(dst + uint32_t(kc) * CHUNKB + uint32_t(px) * 16,
                               row + (in ? size_t(xx >> up) * CIN + kc * 8 : 0), in ? 16 : 0);
                }
            } else {
#pragma unroll 3
                for (int q = tid; q < KC * TC_PX; q += TC_THREADS) {
                    const int kc = q % KC, px = q / KC;
                    *reinterpret_cast<uint4*>(dst + uint32_t(kc) * CHUNKB + uint32_t(px) * 16) =
                        src8_at(a.src, a.mode, a.H, a.W, CIN, b, yy, x0 + px - 1, kc * 8);
                }
            }
        } else {
            // FP32 source (the input gradient's dY, read directly), 8 channels
            // in two 16-byte loads, the ReLU mask as one 16-byte load
#pragma unroll 2
            for (int q = tid; q < KC * TC_PX; q += TC_THREADS) {
                const int kc = q % KC, px = q / KC, xx = x0 + px - 1;
                uint4 v = make_uint4(0, 0, 0, 0);
                if (rin && xx >= 0 && xx < a.W) {
                    const size_t k8 = ((size_t(b) * a.H + yy) * a.W + xx) * CIN + kc * 8;
                    const float4 lo = *reinterpret_cast<const float4*>(a.src + k8);
                    const float4 hi = *reinterpret_cast<const float4*>(a.src + k8 + 4);
                    float f[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                    if (a.mask) {
                        const uint4 mv = *reinterpret_cast<const uint4*>(a.mask + k8);
                        const bf16* mk = reinterpret_cast<const bf16*>(&mv);
#pragma unroll
                        for (int c = 0; c < 8; c++)
                            if (!(__bfloat162float(mk[c]) > 0.f)) f[c] = 0.f;
                    }
                    bf16* e = reinterpret_cast<bf16*>(&v);
#pragma unroll
                    for (int c = 0; c < 8; c++) e[c] = __float2bfloat16(f[c]);
                }
                *reinterpret_cast<uint4*>(dst + uint32_t(kc) * CHUNKB + uint32_t(px) * 16) = v;
            }
        }
    };
    uint32_t phase = 0;
    int ok = 1;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the launches before this one, complete
    int pseg = -1, pb = -1, py = -2;   // the previous task, whose next row is staged
    for (long task = t0; task < t1 && ok; task++) {
        const int y = int(task % a.H);
        const long r = task / a.H;
        const int b = int(r % a.B), seg = int(r / a.B), x0 = seg * TC_M;
        if (!(seg == pseg && b == pb && y == py + 1)) {
            stage(b, y - 1, x0);
            stage(b, y, x0);
            stage(b, y + 1, x0);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        fence_async_smem();   // the staged rows (and weights) become visible to the tensor cores
        fence_before();
        __syncthreads();
        fence_after();
        if (tid == 0) {
            uint32_t acc = 0;
#pragma unroll 1
            for (int t = 0; t < 9; t++) {
                const int dy = t / 3, dx = t % 3;
                unsigned char* src_row = rows + uint32_t((y + dy + TC_RING) % TC_RING) * ROWB;   // row y-1+dy
#pragma unroll
                for (int kb = 0; kb < CIN / 16; kb++) {
                    const uint32_t aa = smem_u32(src_row + uint32_t(2 * kb) * CHUNKB + dx * 16);
                    const uint32_t ba = smem_u32(wsm + uint32_t(t) * WTAPB + uint32_t(2 * kb) * COUT * 16);
                    mma_bf16_ss(tmem, sdesc(aa, CHUNKB, 128), sdesc(ba, uint32_t(COUT) * 16, 128), IDESC, acc);
                    acc = 1;
                }
            }
            mma_commit(bar_a);
        }
        // while the tensor cores run: the next task's new row, if it continues
        // this segment, into the ring slot these MMAs do not read (row y-2's)
        if (task + 1 < t1 && y + 1 < a.H) stage(b, y + 2, x0);
        pseg = seg;
        pb = b;
        py = y;
        const int x = x0 + warp * 32 + lane;
        uint4 skip[COUT / 8];
        if (a.resid && warp < 4 && x < a.W) {
            const uint4* q = reinterpret_cast<const uint4*>(a.resid + ((size_t(b) * a.H + y) * a.W + x) * COUT);
#pragma unroll
            for (int h = 0; h < COUT / 8; h++) skip[h] = q[h];
        }
        ok = mbar_wait(bar_a, phase) ? 1 : 0;
        phase ^= 1;
        ok = __syncthreads_and(ok);
        fence_after();
        if (ok && warp < 4) {
            const uint32_t ta = tmem + (uint32_t(warp * 32) << 16);
#pragma unroll
            for (int c0 = 0; c0 < COUT; c0 += 16) {
                float v[16];
                tmem_ld16(ta + c0, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (x < a.W) {
                    const size_t k = ((size_t(b) * a.H + y) * a.W + x) * COUT + c0;
                    if (a.bias) {
#pragma unroll
                        for (int c = 0; c < 16; c++) v[c] += bias_s[c0 + c];
                    }
                    if (a.resid) {
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const uint4 rv = skip[c0 / 8 + h];
                            const bf16* r = reinterpret_cast<const bf16*>(&rv);
#pragma unroll
                            for (int c = 0; c < 8; c++) v[8 * h + c] += __bfloat162float(r[c]);
                        }
                    }
                    if (a.relu) {
#pragma unroll
                        for (int c = 0; c < 16; c++) v[c] = fmaxf(v[c], 0.f);
                    }
                    // 16 channels of a pixel as 16-byte stores
                    if constexpr (std::is_same<TOUT, float>::value) {
#pragma unroll
                        for (int h = 0; h < 4; h++)
                            *reinterpret_cast<float4*>(a.out + k + 4 * h) =
                                make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
                    } else {
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            uint4 o;
                            bf16* e = reinterpret_cast<bf16*>(&o);
#pragma unroll
                            for (int c = 0; c < 8; c++) e[c] = __float2bfloat16(v[8 * h + c]);
                            *reinterpret_cast<uint4*>(a.out + k + 8 * h) = o;
                        }
                    }
                }
            }
        }
        fence_before();
        __syncthreads();   // accumulator read and staged rows consumed before the next segment
        fence_after();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!ok) {
        // a wait gave up: note it, and give any MMA still in flight a bounded
        // time to finish before the tensor memory is released
        if (tid == 0) {
            atomicExch(&g_timeout, 1);
            (void)mbar_wait(bar_a, phase ^ 1);
        }
        __syncthreads();
    }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS) : "memory");
}

}  // namespace tc

template <int CIN, int COUT>
constexpr size_t conv_smem() {
    return (size_t(TPY + 2) * (TPX + 2) * (CIN + 8) + size_t(9) * COUT * (CIN + 8)) * sizeof(bf16);
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const bf16* p) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a)
                 : "memory");
}

/** Shape of the weight-gradient GEMM of one layer: M = output channels, N =
 * input channels for each of the 9 taps, K = pixels. A warp takes 16 x 8 PN
 * of (M, N) for all taps in registers; NG warps cover (M, N), and the other
 * factor KS of the block's eight splits the pixels. */
template <int CIN, int COUT>
struct WGrad {
    static constexpr int TW = 32, TH = 8, NPX = TW * TH, XW = TW + 2, XPX = XW * (TH + 2);
    static constexpr int GS = COUT + 8, XS = CIN + 8;   // pixel strides: 16 bytes off a multiple of 128
    static constexpr int MT = COUT / 16, NT = CIN / 8, PN = NT < 4 ? NT : 4, NG = MT * (NT / PN), KS = 8 / NG;
    static constexpr size_t TILE = (size_t(NPX) * GS + size_t(XPX) * XS) * sizeof(bf16);
    static constexpr size_t RED = KS > 1 ? size_t(9) * COUT * CIN * sizeof(float) : 0;
    static constexpr size_t SMEM = TILE > RED ? TILE : RED;
    static constexpr int MINB = PN == 4 ? 1 : 2;
};

/** Weight gradient dW[tap][co][ci] += sum_p G[p][co] X_tap[p][ci] and bias
 * gradient, with G = dY masked by the layer's ReLU (mask = layer output) and
 * X the (resampled) layer input, on mma.sync m16n8k16 with both operands
 * read by transposing ldmatrix from pixel-major tiles. A block walks tiles of
 * 8 rows of 32 pixels: a tile (and X's halo) is staged once for all nine taps,
 * whose accumulators stay in registers until the end, when the pixel-splitting
 * warps add up in shared memory and the block adds its sums to dW.
 *
 * Bound: reading dY (FP32), the mask and X once, 8 (bytes) COUT + 2 CIN a
 * pixel. At 8 x 256 x 512 pixels 16 -> 16 takes 76 us (134 MB, 1.8 TB/s), 32 ->
 * 32 at half the side 71 us; with one tap a block (everything read nine
 * times, element by element) they took 975 and 468 us. */
template <int CIN, int COUT>
__global__ void __launch_bounds__(256, WGrad<CIN, COUT>::MINB)
conv_wgrad_k(const bf16* __restrict__ src, int mode, const float* __restrict__ dy, const bf16* __restrict__ ymask,
             float* dw, float* db, int B, int H, int W) {
    using S = WGrad<CIN, COUT>;
    constexpr int GC = COUT / 8, XC = CIN / 8, TW = S::TW, TH = S::TH;
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* gsm = reinterpret_cast<bf16*>(smem);        // [NPX][GS]
    bf16* xsm = gsm + S::NPX * S::GS;                 // [XPX][XS]
    __shared__ float bsm[COUT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gi = warp % S::NG, ki = warp / S::NG;
    const int m0 = (gi % S::MT) * 16, n0 = (gi / S::MT) * (8 * S::PN);
    if (tid < COUT) bsm[tid] = 0.f;
    float acc[9][S::PN][4];
#pragma unroll
    for (int t = 0; t < 9; t++)
#pragma unroll
        for (int j = 0; j < S::PN; j++) acc[t][j][0] = acc[t][j][1] = acc[t][j][2] = acc[t][j][3] = 0.f;
    float bacc[8];
#pragma unroll
    for (int k = 0; k < 8; k++) bacc[k] = 0.f;
    static_assert(256 % GC == 0 && 8 % S::NG == 0, "a thread keeps its channels");
    const int gc = tid % GC, xc = tid % XC;
    // ldmatrix row addresses of this lane (matrix lane / 8, row lane % 8):
    // A's matrices run over output channels first, B's over pixels first
    const int mi = lane >> 3, lr = lane & 7;
    const int ga = ((mi >> 1) * 8 + lr) * S::GS + m0 + (mi & 1) * 8;
    const int xa = ((mi & 1) * 8 + lr) * S::XS + n0 + (mi >> 1) * 8;
    const int tilesx = (W + TW - 1) / TW, tilesy = (H + TH - 1) / TH, ntiles = tilesx * tilesy * B;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int b = tile / (tilesx * tilesy), r = tile - b * tilesx * tilesy;
        const int x0 = (r % tilesx) * TW, y0 = (r / tilesx) * TH;
        __syncthreads();
#pragma unroll 4
        for (int p = tid / GC; p < S::NPX; p += 256 / GC) {
            const int x = x0 + p % TW, y = y0 + p / TW;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (x < W && y < H) {
                const size_t k = ((size_t(b) * H + y) * W + x) * COUT + gc * 8;
                const float4 lo = *reinterpret_cast<const float4*>(dy + k), hi = *reinterpret_cast<const float4*>(dy + k + 4);
                float f[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                if (ymask) {
                    const uint4 mv = *reinterpret_cast<const uint4*>(ymask + k);
                    const bf16* mk = reinterpret_cast<const bf16*>(&mv);
#pragma unroll
                    for (int c = 0; c < 8; c++)
                        if (!(__bfloat162float(mk[c]) > 0.f)) f[c] = 0.f;
                }
                bf16* e = reinterpret_cast<bf16*>(&v);
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    e[c] = __float2bfloat16(f[c]);
                    bacc[c] += __bfloat162float(e[c]);
                }
            }
            *reinterpret_cast<uint4*>(gsm + p * S::GS + gc * 8) = v;
        }
#pragma unroll 4
        for (int p = tid / XC; p < S::XPX; p += 256 / XC)
            *reinterpret_cast<uint4*>(xsm + p * S::XS + xc * 8) =
                src8_at(src, mode, H, W, CIN, b, y0 + p / S::XW - 1, x0 + p % S::XW - 1, xc * 8);
        __syncthreads();
#pragma unroll 1
        for (int ks = ki; ks < S::NPX / 16; ks += S::KS) {
            const int row = ks >> 1, cx = (ks & 1) * 16;
            uint32_t av[4];
            ldsm_x4_t(av, gsm + (row * TW + cx) * S::GS + ga);
#pragma unroll
            for (int t = 0; t < 9; t++) {
                const bf16* xb = xsm + ((row + t / 3) * S::XW + cx + t % 3) * S::XS + xa;
#pragma unroll
                for (int j = 0; j < S::PN; j += 2) {
                    uint32_t bv[4];
                    ldsm_x4_t(bv, xb + j * 8);
                    mma_bf16(acc[t][j], av[0], av[1], av[2], av[3], bv[0], bv[1]);
                    mma_bf16(acc[t][j + 1], av[0], av[1], av[2], av[3], bv[2], bv[3]);
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; k++) atomicAdd(&bsm[gc * 8 + k], bacc[k]);
    const int g = lane >> 2, tq = lane & 3;
    if constexpr (S::KS == 1) {
#pragma unroll
        for (int t = 0; t < 9; t++)
#pragma unroll
            for (int j = 0; j < S::PN; j++) {
                float* d = dw + (size_t(t) * COUT + m0 + g) * CIN + n0 + j * 8 + 2 * tq;
                atomicAdd(d, acc[t][j][0]);
                atomicAdd(d + 1, acc[t][j][1]);
                atomicAdd(d + 8 * CIN, acc[t][j][2]);
                atomicAdd(d + 8 * CIN + 1, acc[t][j][3]);
            }
        __syncthreads();
    } else {
        float* red = reinterpret_cast<float*>(smem);   // [9][COUT][CIN]
        for (int q = 0; q < S::KS; q++) {
            if (ki == q) {
#pragma unroll
                for (int t = 0; t < 9; t++)
#pragma unroll
                    for (int j = 0; j < S::PN; j++) {
                        float* d = red + (t * COUT + m0 + g) * CIN + n0 + j * 8 + 2 * tq;
                        float* e = d + 8 * CIN;
                        d[0] = (q ? d[0] : 0.f) + acc[t][j][0];
                        d[1] = (q ? d[1] : 0.f) + acc[t][j][1];
                        e[0] = (q ? e[0] : 0.f) + acc[t][j][2];
                        e[1] = (q ? e[1] : 0.f) + acc[t][j][3];
                    }
            }
            __syncthreads();
        }
        for (int k = tid; k < 9 * COUT * CIN; k += 256) atomicAdd(dw + k, red[k]);
    }
    if (tid < COUT) atomicAdd(db + tid, bsm[tid]);
}

/** Flipped, transposed weights for the input gradient of every layer
 * (blockIdx.y): wt[8-tap][ci][co] = w[tap][co][ci]. */
struct FlipArgs {
    const bf16* w[14];
    bf16* wt[14];
    int cin[14], cout[14];
};
__global__ void flip_transpose_k(FlipArgs a) {
    const int l = blockIdx.y, cin = a.cin[l], cout = a.cout[l];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 9 * cin * cout) return;
    const int ci = t % cin, r = t / cin, co = r % cout, tap = r / cout;
    a.wt[l][(size_t(8 - tap) * cin + ci) * cout + co] = a.w[l][t];
}

/** dsrc = the adjoint of nearest upsampling by two applied to dx (operating
 * grid H x W, C channels): the sum over each source pixel's 2 x 2 block, four
 * channels a thread. */
__global__ void upsample_adjoint_k(const float* __restrict__ dx, float* __restrict__ dsrc, int B, int H, int W, int C) {
    const int Hs = H >> 1, Ws = W >> 1, C4 = C >> 2;
    const size_t n = size_t(B) * Hs * Ws * C4;
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x) {
        const int c = int(k % C4);
        const size_t p = k / C4;
        const int xs = int(p % Ws), ys = int((p / Ws) % Hs), b = int(p / (size_t(Ws) * Hs));
        const float4* q = reinterpret_cast<const float4*>(dx + ((size_t(b) * H + 2 * ys) * W + 2 * xs) * C) + c;
        const float4 v00 = q[0], v01 = q[C4], v10 = q[size_t(W) * C4], v11 = q[size_t(W) * C4 + C4];
        float4 s;
        s.x = ((v00.x + v01.x) + v10.x) + v11.x;
        s.y = ((v00.y + v01.y) + v10.y) + v11.y;
        s.z = ((v00.z + v01.z) + v10.z) + v11.z;
        s.w = ((v00.w + v01.w) + v10.w) + v11.w;
        reinterpret_cast<float4*>(dsrc)[k] = s;
    }
}

/** dsrc += the adjoint of the 2 x 2 mean applied to dx (operating grid H x W,
 * C channels): a quarter of each value for its four source pixels, four
 * channels a thread. */
__global__ void pool_adjoint_add_k(const float* __restrict__ dx, float* __restrict__ dsrc, int B, int H, int W, int C) {
    const int Ws = 2 * W, C4 = C >> 2;
    const size_t n = size_t(B) * 2 * H * Ws * C4;
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x) {
        const int c = int(k % C4);
        const size_t p = k / C4;
        const int xs = int(p % Ws), ys = int((p / Ws) % (2 * H)), b = int(p / (size_t(Ws) * 2 * H));
        const float4 v = reinterpret_cast<const float4*>(dx + ((size_t(b) * H + (ys >> 1)) * W + (xs >> 1)) * C)[c];
        float4 d = reinterpret_cast<const float4*>(dsrc)[k];
        d.x += 0.25f * v.x;
        d.y += 0.25f * v.y;
        d.z += 0.25f * v.z;
        d.w += 0.25f * v.w;
        reinterpret_cast<float4*>(dsrc)[k] = d;
    }
}

/** One parameter array of the optimiser: FP32 master values, their BF16 copy
 * (or null), gradient and moments. */
struct AdamArray {
    float* w;
    bf16* wb;
    float *g, *m1, *m2;
    int n;
};
struct AdamArgs {
    AdamArray a[28];
    float lr, b1, b2, c1, c2, eps;
};
/** Adam step on every parameter array (blockIdx.y), refreshing the BF16
 * copies and clearing the gradients. */
__global__ void adam_k(const __grid_constant__ AdamArgs p) {
    const AdamArray& q = p.a[blockIdx.y];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < q.n; k += gridDim.x * blockDim.x) {
        float gv = q.g[k];
        float a = p.b1 * q.m1[k] + (1.f - p.b1) * gv;
        float v = p.b2 * q.m2[k] + (1.f - p.b2) * gv * gv;
        q.m1[k] = a;
        q.m2[k] = v;
        float wv = q.w[k] - p.lr * (a / p.c1) / (sqrtf(v / p.c2) + p.eps);
        q.w[k] = wv;
        if (q.wb) q.wb[k] = __float2bfloat16(wv);
        q.g[k] = 0.f;
    }
}

/** Loss and its gradient on output channel 0: L = mean (y0 - t)^2. */
__global__ void mse_k(const float* y, const float* t, float* dy, int npx, int C, float* loss) {
    __shared__ float ws[32];
    float s = 0.f;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npx; p += gridDim.x * blockDim.x) {
        float d = y[size_t(p) * C] - t[p];
        s += d * d;
        // the other channels have no target: C (a multiple of 4) values a pixel
        float4* o = reinterpret_cast<float4*>(dy + size_t(p) * C);
        o[0] = make_float4(2.f * d / npx, 0.f, 0.f, 0.f);
        for (int q = 1; q < C / 4; q++) o[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float q = 0.f;
        for (int w = 0; w < int(blockDim.x >> 5); w++) q += ws[w];
        atomicAdd(loss, q / npx);
    }
}

/** Packs a one-channel FP32 image into the 16-channel BF16 network input. */
__global__ void pack_input_k(const float* x, bf16* in, size_t npx) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (size_t p = blockIdx.x * size_t(blockDim.x) + threadIdx.x; p < npx; p += size_t(gridDim.x) * blockDim.x) {
        uint4* o = reinterpret_cast<uint4*>(in + p * 16);
        o[0] = make_uint4(__bfloat16_as_ushort(__float2bfloat16(x[p])), 0, 0, 0);
        o[1] = make_uint4(0, 0, 0, 0);
    }
}

__global__ void unpack_output_k(const float* y, float* out, size_t npx) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (size_t p = blockIdx.x * size_t(blockDim.x) + threadIdx.x; p < npx; p += size_t(gridDim.x) * blockDim.x)
        out[p] = y[p * 16];
}

// ---------------------------------------------------------------- host
struct Layer {
    int cin, cout, mode, relu, skip;   // skip: index of the layer whose output is added, or -1
    int src;                           // index of the layer whose output is the input, -1 = network input
    float *w = nullptr, *g = nullptr, *m1 = nullptr, *m2 = nullptr;          // [9][cout][cin]
    float *b = nullptr, *gb = nullptr, *bm1 = nullptr, *bm2 = nullptr;       // [cout]
    bf16* wb = nullptr;
    bf16* wt = nullptr;                // flipped, transposed copy for the input gradient
    int H, W;                          // operating grid
};

static const int NL = 14;

struct Net {
    int H, W, Bmax;                    // input grid and batch capacity
    Layer L[NL];
    std::vector<void*> bufs;
    bf16* in = nullptr;                // [B][H][W][16]
    bf16* act[NL];                     // layer outputs (BF16)
    float* outf = nullptr;             // last layer output (FP32)
    float* gact[NL];                   // gradients of layer outputs
    float* tmp = nullptr;              // input-gradient scratch (largest layer input)
    float* loss = nullptr;
    int step = 0;
};

/** Whether the forward and input-gradient convolutions run on tcgen05
 * (default) or on mma.sync (VDI_UNET_TC=0), read once per process. */
static bool use_tc() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("VDI_UNET_TC");
        v = (e && e[0] == '0') ? 0 : 1;
    }
    return v == 1;
}

/** Launches a kernel; with early, it may start before the launch ahead of it
 * in the stream has ended (programmatic dependent launch) and waits itself for
 * that one's results. What it reads before waiting, the weights, has to be
 * complete before the launch ahead starts: that one was launched in the plain
 * way, or behind a plain launch that is behind the weights' last writer. */
template <class... P, class... A>
static cudaError_t launch_early(cudaStream_t s, bool early, void (*kernel)(P...), int grid, int threads, size_t smem,
                                const A&... a) {
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.gridDim = dim3(unsigned(grid));
    c.blockDim = dim3(unsigned(threads));
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, P(a)...);
}

template <int CIN, int COUT, typename TIN, typename TOUT>
static cudaError_t conv_launch(cudaStream_t s, const ConvArgs<TIN, TOUT>& a, bool early) {
    if (use_tc()) {
        // one wave of resident CTAs: each takes a contiguous run of tasks and
        // stages the next rows while its MMAs run
        static int resident = 0;
        if (!resident) {
            cudaError_t e = cudaFuncSetAttribute(tc::conv3x3_tc<CIN, COUT, TIN, TOUT>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 int(tc::tc_smem<CIN, COUT>()));
            if (e != cudaSuccess) return e;
            int dev = 0, sms = 0;
            if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
                (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
                return e;
            resident = sms * tc::tc_blocks<CIN, COUT>();
        }
        const long tasks = long(a.B) * a.H * ((a.W + tc::TC_M - 1) / tc::TC_M);
        const int grid = int(tasks < resident ? tasks : resident);
        return launch_early(s, early, tc::conv3x3_tc<CIN, COUT, TIN, TOUT>, grid, tc::TC_THREADS,
                            tc::tc_smem<CIN, COUT>(), a);
    }
    static bool attr = false;
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(conv3x3_k<CIN, COUT, TIN, TOUT>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, int(conv_smem<CIN, COUT>()));
        if (e != cudaSuccess) return e;
        attr = true;
    }
    int tiles = ((a.W + TPX - 1) / TPX) * ((a.H + TPY - 1) / TPY);
    conv3x3_k<CIN, COUT, TIN, TOUT><<<dim3(tiles, a.B), 256, conv_smem<CIN, COUT>(), s>>>(a);
    return cudaGetLastError();
}

template <typename TIN, typename TOUT>
static cudaError_t conv_dispatch(cudaStream_t s, int cin, int cout, const ConvArgs<TIN, TOUT>& a, bool early) {
#define VDI_CONV(CI, CO) \
    if (cin == CI && cout == CO) return conv_launch<CI, CO, TIN, TOUT>(s, a, early);
    VDI_CONV(16, 16) VDI_CONV(16, 32) VDI_CONV(32, 32) VDI_CONV(32, 64) VDI_CONV(64, 64) VDI_CONV(64, 32)
    VDI_CONV(32, 16)
#undef VDI_CONV
    return cudaErrorInvalidValue;
}

template <int CIN, int COUT>
static cudaError_t wgrad_launch(cudaStream_t s, const Layer& l, const bf16* src, const float* dy, const bf16* ymask,
                                int B) {
    using S = WGrad<CIN, COUT>;
    cudaError_t e = cudaFuncSetAttribute(conv_wgrad_k<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(S::SMEM));
    if (e != cudaSuccess) return e;
    const int tiles = ((l.W + S::TW - 1) / S::TW) * ((l.H + S::TH - 1) / S::TH) * B;
    conv_wgrad_k<CIN, COUT><<<std::min(tiles, 148 * S::MINB), 256, S::SMEM, s>>>(src, l.mode, dy, ymask, l.g, l.gb, B,
                                                                                 l.H, l.W);
    return cudaGetLastError();
}

static cudaError_t wgrad_dispatch(cudaStream_t s, const Layer& l, const bf16* src, const float* dy, const bf16* ymask,
                                  int B) {
#define VDI_WG(CI, CO) \
    if (l.cin == CI && l.cout == CO) return wgrad_launch<CI, CO>(s, l, src, dy, ymask, B);
    VDI_WG(16, 16) VDI_WG(16, 32) VDI_WG(32, 32) VDI_WG(32, 64) VDI_WG(64, 64) VDI_WG(64, 32) VDI_WG(32, 16)
#undef VDI_WG
    return cudaErrorInvalidValue;
}

static int falloc(Net* n, float** p, size_t count) {
    VDI_CUDA(cudaMalloc(p, count * sizeof(float)));
    VDI_CUDA(cudaMemset(*p, 0, count * sizeof(float)));
    n->bufs.push_back(*p);
    return VDI_OK;
}

static int balloc(Net* n, bf16** p, size_t count) {
    VDI_CUDA(cudaMalloc(p, count * sizeof(bf16)));
    VDI_CUDA(cudaMemset(*p, 0, count * sizeof(bf16)));
    n->bufs.push_back(*p);
    return VDI_OK;
}

/** Deterministic initialisation: He-scaled values from a hash of the index. */
static void init_weights(std::vector<float>& w, int fan_in, unsigned seed) {
    double sc = std::sqrt(2.0 / fan_in);
    for (size_t k = 0; k < w.size(); k++) {
        unsigned h = unsigned(k) * 2654435761u ^ (seed * 0x9E3779B9u);
        h ^= h >> 15; h *= 0x2c1b3c6du; h ^= h >> 12; h *= 0x297a2d39u; h ^= h >> 15;
        double u = (h + 0.5) / 4294967296.0;                     // (0,1)
        w[k] = float(sc * std::sqrt(3.0) * (2 * u - 1));         // uniform with the He variance
    }
}

static void net_free(Net* n) {
    for (auto p : n->bufs) cudaFree(p);
    n->bufs.clear();
}

static int net_create(int H, int W, int Bmax, unsigned seed, Net** out) {
    if (H % 8 || W % 16 || H < 8 || W < 16 || Bmax < 1) {
        set_error("unet: grid %dx%d must be a multiple of 8 rows and 16 columns", H, W);
        return VDI_ERR_INVALID_ARGUMENT;
    }
    Net* n = new Net();
    n->H = H; n->W = W; n->Bmax = Bmax;
    // {cin, cout, mode, relu, skip, src}; grid level from the layer position
    const int spec[NL][6] = {{16, 16, 0, 1, -1, -1}, {16, 16, 0, 1, -1, 0},  {16, 32, 2, 1, -1, 1},
                             {32, 32, 0, 1, -1, 2},  {32, 64, 2, 1, -1, 3},  {64, 64, 0, 1, -1, 4},
                             {64, 64, 2, 1, -1, 5},  {64, 64, 0, 1, -1, 6},  {64, 64, 1, 1, 5, 7},
                             {64, 32, 0, 1, -1, 8},  {32, 32, 1, 1, 3, 9},   {32, 16, 0, 1, -1, 10},
                             {16, 16, 1, 1, 1, 11},  {16, 16, 0, 0, -1, 12}};
    const int level[NL] = {0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0};
    int st;
    auto fail = [&](int s) {
        net_free(n);
        delete n;
        return s;
    };
    for (int k = 0; k < NL; k++) {
        Layer& l = n->L[k];
        l.cin = spec[k][0]; l.cout = spec[k][1]; l.mode = spec[k][2]; l.relu = spec[k][3];
        l.skip = spec[k][4]; l.src = spec[k][5];
        l.H = H >> level[k]; l.W = W >> level[k];
        size_t nw = size_t(9) * l.cin * l.cout;
        if ((st = falloc(n, &l.w, nw)) || (st = falloc(n, &l.g, nw)) || (st = falloc(n, &l.m1, nw)) ||
            (st = falloc(n, &l.m2, nw)) || (st = falloc(n, &l.b, l.cout)) || (st = falloc(n, &l.gb, l.cout)) ||
            (st = falloc(n, &l.bm1, l.cout)) || (st = falloc(n, &l.bm2, l.cout)) || (st = balloc(n, &l.wb, nw)) ||
            (st = balloc(n, &l.wt, nw)))
            return fail(st);
        std::vector<float> w(nw);
        init_weights(w, 9 * l.cin, seed + 7919u * k);
        if (k == NL - 1)
            for (auto& v : w) v *= 0.1f;   // start near a zero correction
        std::vector<bf16> wb(nw);
        for (size_t q = 0; q < nw; q++) wb[q] = __float2bfloat16(w[q]);
        if (cudaMemcpy(l.w, w.data(), nw * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemcpy(l.wb, wb.data(), nw * 2, cudaMemcpyHostToDevice) != cudaSuccess)
            return fail(VDI_ERR_CUDA);
        size_t na = size_t(Bmax) * l.H * l.W * l.cout;
        if ((st = balloc(n, &n->act[k], na)) || (st = falloc(n, &n->gact[k], na))) return fail(st);
    }
    size_t npx = size_t(Bmax) * H * W;
    if ((st = balloc(n, &n->in, npx * 16)) || (st = falloc(n, &n->outf, npx * 16)) ||
        (st = falloc(n, &n->tmp, npx * 64)) || (st = falloc(n, &n->loss, 1)))
        return fail(st);
    *out = n;
    return VDI_OK;
}

static const bf16* layer_input(const Net* n, int k) { return n->L[k].src < 0 ? n->in : n->act[n->L[k].src]; }

/** The network on an FP32 image batch, its input packed and (with out) its
 * output unpacked. Each launch behind the first starts beside the one before
 * it (16 launches of 2-3 us of set-up each),
 * but in a stream that is being captured: there the edges stay plain, as a
 * conditional node's body needs them. */
static int net_forward(Net* n, cudaStream_t s, const float* in, float* out, int B) {
    cudaStreamCaptureStatus cap;
    VDI_CUDA(cudaStreamIsCapturing(s, &cap));
    const bool early = use_tc() && cap == cudaStreamCaptureStatusNone;
    const size_t npx = size_t(B) * n->H * n->W;
    pack_input_k<<<592, 256, 0, s>>>(in, n->in, npx);
    VDI_CUDA(cudaGetLastError());
    for (int k = 0; k < NL; k++) {
        const Layer& l = n->L[k];
        if (k == NL - 1) {
            ConvArgs<bf16, float> a{layer_input(n, k), nullptr, l.mode, l.wb, l.b, nullptr, 0, n->outf, B, l.H, l.W};
            VDI_CUDA(conv_dispatch(s, l.cin, l.cout, a, early));
        } else {
            ConvArgs<bf16, bf16> a{layer_input(n, k), nullptr, l.mode, l.wb, l.b,
                                   l.skip >= 0 ? n->act[l.skip] : nullptr, l.relu, n->act[k], B, l.H, l.W};
            VDI_CUDA(conv_dispatch(s, l.cin, l.cout, a, early));
        }
    }
    if (out) VDI_CUDA(launch_early(s, early, unpack_output_k, 592, 256, 0, n->outf, out, npx));
    return VDI_OK;
}

/** d = g where the ReLU mask (the layer output) is positive, else zero; n a
 * multiple of 8. */
__global__ void masked_copy_k(float* __restrict__ d, const float* __restrict__ g, const bf16* __restrict__ mk, size_t n) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n / 8; i += size_t(gridDim.x) * blockDim.x) {
        const uint4 mv = reinterpret_cast<const uint4*>(mk)[i];
        const bf16* m = reinterpret_cast<const bf16*>(&mv);
        const float4 a = reinterpret_cast<const float4*>(g)[2 * i], b = reinterpret_cast<const float4*>(g)[2 * i + 1];
        float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (!(__bfloat162float(m[k]) > 0.f)) f[k] = 0.f;
        reinterpret_cast<float4*>(d)[2 * i] = make_float4(f[0], f[1], f[2], f[3]);
        reinterpret_cast<float4*>(d)[2 * i + 1] = make_float4(f[4], f[5], f[6], f[7]);
    }
}

/** Backward pass from the gradient in gact[NL-1]; accumulates weight and
 * bias gradients. Each output's gradient is written by its first contribution
 * (the skip's, where there is one, which comes from a later layer; else the
 * next layer's input gradient), so nothing is cleared first: direct inputs get
 * their gradient from the convolution itself, upsampled and pooled ones (the
 * pooled are the outputs with a skip) through one more pass. Adding the pooled
 * ones in the convolution's epilogue was slower (155 us instead of 37 and the
 * pass, 64 -> 32 channels at 64 x 128). */
static int net_backward(Net* n, cudaStream_t s, int B) {
    FlipArgs fa;
    int most = 0;
    for (int k = 0; k < NL; k++) {
        const Layer& l = n->L[k];
        fa.w[k] = l.wb;
        fa.wt[k] = l.wt;
        fa.cin[k] = l.cin;
        fa.cout[k] = l.cout;
        most = std::max(most, 9 * l.cin * l.cout);
    }
    flip_transpose_k<<<dim3((most + 255) / 256, NL), 256, 0, s>>>(fa);
    for (int k = NL - 1; k >= 0; k--) {
        const Layer& l = n->L[k];
        const bf16* ymask = l.relu ? n->act[k] : nullptr;
        const float* dy = n->gact[k];
        // skip connection: its gradient is the output gradient through the ReLU
        if (l.skip >= 0) {
            size_t na = size_t(B) * l.H * l.W * l.cout;
            masked_copy_k<<<1184, 256, 0, s>>>(n->gact[l.skip], dy, ymask, na);
            VDI_CUDA(cudaGetLastError());
        }
        // weight and bias gradients
        VDI_CUDA(wgrad_dispatch(s, l, layer_input(n, k), dy, ymask, B));
        if (k == 0) continue;   // no gradient needed for the network input
        // input gradient on the operating grid, through the resampling's adjoint
        const bool direct = l.mode == SRC_DIRECT;
        ConvArgs<float, float> a{dy, ymask, SRC_DIRECT, l.wt, nullptr, nullptr, 0, direct ? n->gact[l.src] : n->tmp,
                                 B,  l.H,   l.W};
        VDI_CUDA(conv_dispatch(s, l.cout, l.cin, a, false));
        if (l.mode == SRC_UP2) upsample_adjoint_k<<<1184, 256, 0, s>>>(n->tmp, n->gact[l.src], B, l.H, l.W, l.cin);
        if (l.mode == SRC_POOL2) pool_adjoint_add_k<<<1184, 256, 0, s>>>(n->tmp, n->gact[l.src], B, l.H, l.W, l.cin);
        VDI_CUDA(cudaGetLastError());
    }
    return VDI_OK;
}

}  // namespace unet
}  // namespace vdi

using namespace vdi;
using namespace vdi::unet;

struct vdi_unet {
    Net* net = nullptr;
    cudaStream_t s = nullptr;
};

extern "C" {

int vdi_unet_create(int H, int W, int batch, unsigned seed, void* stream, vdi_unet** out) {
    if (!out) return VDI_ERR_INVALID_ARGUMENT;
    vdi_unet* u = new vdi_unet();
    u->s = static_cast<cudaStream_t>(stream);
    int st = net_create(H, W, batch, seed, &u->net);
    if (st != VDI_OK) {
        delete u;
        return st;
    }
    *out = u;
    return VDI_OK;
}

int vdi_unet_destroy(vdi_unet* u) {
    if (!u) return VDI_OK;
    if (u->net) {
        net_free(u->net);
        delete u->net;
    }
    delete u;
    return VDI_OK;
}

long vdi_unet_param_count(const vdi_unet* u) {
    if (!u) return 0;
    long c = 0;
    for (int k = 0; k < NL; k++) c += 9L * u->net->L[k].cin * u->net->L[k].cout + u->net->L[k].cout;
    return c;
}

/** Reports a tensor-core wait that gave up (the kernels return without
 * their result rather than wait longer). */
static int tc_status(cudaStream_t s) {
    if (!use_tc()) return VDI_OK;
    int t = 0;
    VDI_CUDA(cudaMemcpyFromSymbolAsync(&t, tc::g_timeout, sizeof(int), 0, cudaMemcpyDeviceToHost, s));
    VDI_CUDA(cudaStreamSynchronize(s));
    if (t) {
        set_error("unet: a tensor-core convolution timed out waiting for its MMAs");
        return VDI_ERR_CUDA;
    }
    return VDI_OK;
}

int vdi_unet_tensor_path(void) { return use_tc() ? 1 : 0; }

int vdi_unet_forward(vdi_unet* u, const float* d_in, float* d_out, int batch) {
    if (!u || !d_in || !d_out || batch < 1 || batch > u->net->Bmax) return VDI_ERR_INVALID_ARGUMENT;
    Net* n = u->net;
    VDI_TRY(net_forward(n, u->s, d_in, d_out, batch));
    return tc_status(u->s);
}

int vdi_unet_train_step(vdi_unet* u, const float* d_in, const float* d_target, int batch, float lr, float* loss) {
    if (!u || !d_in || !d_target || batch < 1 || batch > u->net->Bmax) return VDI_ERR_INVALID_ARGUMENT;
    Net* n = u->net;
    cudaStream_t s = u->s;
    size_t npx = size_t(batch) * n->H * n->W;
    VDI_TRY(net_forward(n, s, d_in, nullptr, batch));
    VDI_CUDA(cudaMemsetAsync(n->loss, 0, sizeof(float), s));
    mse_k<<<592, 256, 0, s>>>(n->outf, d_target, n->gact[NL - 1], int(npx), 16, n->loss);
    VDI_CUDA(cudaGetLastError());
    VDI_TRY(net_backward(n, s, batch));
    n->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    float c1 = 1.f - std::pow(b1, float(n->step)), c2 = 1.f - std::pow(b2, float(n->step));
    static_assert(sizeof(AdamArgs::a) / sizeof(AdamArray) == 2 * NL, "weights and biases of every layer");
    AdamArgs aa;
    for (int k = 0; k < NL; k++) {
        const Layer& l = n->L[k];
        aa.a[2 * k] = AdamArray{l.w, l.wb, l.g, l.m1, l.m2, 9 * l.cin * l.cout};
        aa.a[2 * k + 1] = AdamArray{l.b, nullptr, l.gb, l.bm1, l.bm2, l.cout};
    }
    aa.lr = lr;
    aa.b1 = b1;
    aa.b2 = b2;
    aa.c1 = c1;
    aa.c2 = c2;
    aa.eps = 1e-8f;
    adam_k<<<dim3(36, 2 * NL), 256, 0, s>>>(aa);
    VDI_CUDA(cudaGetLastError());
    if (loss) {
        VDI_CUDA(cudaMemcpyAsync(loss, n->loss, sizeof(float), cudaMemcpyDeviceToHost, s));
        VDI_CUDA(cudaStreamSynchronize(s));
    }
    return tc_status(s);
}

/** Gradient check support: forward + loss + backward without an update;
 * copies layer k's weight gradient ([9][cout][cin], FP32) and the loss. */
int vdi_unet_gradients(vdi_unet* u, const float* d_in, const float* d_target, int batch, int layer, float* h_grad,
                       float* h_loss) {
    if (!u || layer < 0 || layer >= NL || batch < 1 || batch > u->net->Bmax) return VDI_ERR_INVALID_ARGUMENT;
    Net* n = u->net;
    cudaStream_t s = u->s;
    size_t npx = size_t(batch) * n->H * n->W;
    for (int k = 0; k < NL; k++) {
        Layer& l = n->L[k];
        VDI_CUDA(cudaMemsetAsync(l.g, 0, sizeof(float) * 9 * l.cin * l.cout, s));
        VDI_CUDA(cudaMemsetAsync(l.gb, 0, sizeof(float) * l.cout, s));
    }
    VDI_TRY(net_forward(n, s, d_in, nullptr, batch));
    VDI_CUDA(cudaMemsetAsync(n->loss, 0, sizeof(float), s));
    mse_k<<<592, 256, 0, s>>>(n->outf, d_target, n->gact[NL - 1], int(npx), 16, n->loss);
    VDI_TRY(net_backward(n, s, batch));
    Layer& l = n->L[layer];
    VDI_CUDA(cudaMemcpyAsync(h_grad, l.g, sizeof(float) * 9 * l.cin * l.cout, cudaMemcpyDeviceToHost, s));
    VDI_CUDA(cudaMemcpyAsync(h_loss, n->loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    VDI_CUDA(cudaStreamSynchronize(s));
    return VDI_OK;
}

/** Copies all parameters (per layer: weights [9][cout][cin] then bias, FP32)
 * to or from host memory. */
int vdi_unet_params(vdi_unet* u, float* h_buf, long count, int to_device) {
    if (!u || !h_buf || count != vdi_unet_param_count(u)) return VDI_ERR_INVALID_ARGUMENT;
    Net* n = u->net;
    long off = 0;
    for (int k = 0; k < NL; k++) {
        Layer& l = n->L[k];
        size_t nw = size_t(9) * l.cin * l.cout;
        if (to_device) {
            VDI_CUDA(cudaMemcpy(l.w, h_buf + off, nw * 4, cudaMemcpyHostToDevice));
            VDI_CUDA(cudaMemcpy(l.b, h_buf + off + nw, l.cout * 4, cudaMemcpyHostToDevice));
            std::vector<bf16> wb(nw);
            for (size_t q = 0; q < nw; q++) wb[q] = __float2bfloat16(h_buf[off + q]);
            VDI_CUDA(cudaMemcpy(l.wb, wb.data(), nw * 2, cudaMemcpyHostToDevice));
        } else {
            VDI_CUDA(cudaMemcpy(h_buf + off, l.w, nw * 4, cudaMemcpyDeviceToHost));
            VDI_CUDA(cudaMemcpy(h_buf + off + nw, l.b, l.cout * 4, cudaMemcpyDeviceToHost));
        }
        off += nw + l.cout;
    }
    return VDI_OK;
}

}  // extern "C"

namespace vdi {
namespace unet {

/** Network input: the residual averaged over factor x factor blocks, divided
 * by its RMS over the fine grid (norm / sqrt(m n)). */
__global__ void restrict_residual_k(const double* __restrict__ r, const double* rnorm, float* in, int m, int n,
                                    int f) {
    const int W = m / f, H = n / f;
    const double rms = *rnorm / sqrt(double(m) * n);
    const double inv = rms > 0 ? 1.0 / (rms * f * f) : 0.0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < W * H; p += gridDim.x * blockDim.x) {
        const int X = p % W, Y = p / W;
        double s = 0;
        for (int dj = 0; dj < f; dj++)
            for (int di = 0; di < f; di++) s += r[(X * f + di) + size_t(m) * (Y * f + dj)];
        in[p] = float(s * inv);
    }
}

/** z += scale * rms * (bilinear prolongation of the network output). */
__global__ void prolong_correction_k(const float* __restrict__ out, const double* rnorm, double* z, int m, int n,
                                     int f, double scale) {
    const int W = m / f, H = n / f;
    const double a = scale * (*rnorm / sqrt(double(m) * n));
    for (long k = blockIdx.x * long(blockDim.x) + threadIdx.x; k < long(m) * n; k += long(gridDim.x) * blockDim.x) {
        const int i = int(k % m), j = int(k / m);
        float X = (i + 0.5f) / f - 0.5f, Y = (j + 0.5f) / f - 0.5f;
        int I0 = int(floorf(X)), J0 = int(floorf(Y));
        float wx = X - I0, wy = Y - J0;
        int I1 = I0 + 1, J1 = J0 + 1;
        I0 = I0 < 0 ? 0 : (I0 > W - 1 ? W - 1 : I0);
        I1 = I1 < 0 ? 0 : (I1 > W - 1 ? W - 1 : I1);
        J0 = J0 < 0 ? 0 : (J0 > H - 1 ? H - 1 : J0);
        J1 = J1 < 0 ? 0 : (J1 > H - 1 ? H - 1 : J1);
        float v = (1 - wy) * ((1 - wx) * out[I0 + W * J0] + wx * out[I1 + W * J0]) +
                  wy * ((1 - wx) * out[I0 + W * J1] + wx * out[I1 + W * J1]);
        z[k] += a * double(v);
    }
}

}  // namespace unet

int unet_correct(vdi_unet* u, cudaStream_t s, const double* r, const double* d_rnorm, double* z, int m, int n,
                 int factor, double scale, float* in_buf, float* out_buf) {
    using namespace unet;
    Net* net = u->net;
    if (m / factor != net->W || n / factor != net->H) {
        set_error("unet: grid %dx%d / %d does not match the network's %dx%d", m, n, factor, net->W, net->H);
        return VDI_ERR_INVALID_ARGUMENT;
    }
    restrict_residual_k<<<592, 256, 0, s>>>(r, d_rnorm, in_buf, m, n, factor);
    VDI_TRY(net_forward(net, s, in_buf, out_buf, 1));
    prolong_correction_k<<<1184, 256, 0, s>>>(out_buf, d_rnorm, z, m, n, factor, scale);
    VDI_CUDA(cudaGetLastError());
    return VDI_OK;
}

int unet_kernels_per_correction() {
    return 4 + unet::NL;   // restrict, pack, one per layer, unpack, prolong
}

int unet_dims(const vdi_unet* u, int* H, int* W) {
    *H = u->net->H;
    *W = u->net->W;
    return VDI_OK;
}

}  // namespace vdi
