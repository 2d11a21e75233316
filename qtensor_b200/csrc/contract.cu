// Merged-index contractions of the reference's extended bucket backend
// (CMKLExtendedBackend, qtensor/ProcessingFrameworks.py:41-147), whose
// native dependency ``tcontract`` (an MKL C extension) is absent from the
// reference:
//
//   qtb_contract_outer_c64  c[n,m,k] = a[n,m] * b[n,k]          (mkl_contract_complex, :60-66)
//   qtb_contract_sum_c64    C[f,m,n] = sum_k A[k,f,m] * B[k,f,n] (mkl_contract_sum, :123-130)
//
// complex64 in and out.  The contract-sum is a batch of F complex GEMMs; with
// a large summed dimension it runs on the tcgen05 tensor cores:
//   * a pre-pass splits every operand into TF32 "hi" (rounded to nearest,
//     cvt.rna.tf32.f32) and "lo" (the rounded remainder) planes of the real
//     and imaginary parts, transposed to K-major and tiled 128 rows (of A) or
//     kN columns (of B) x 8 k in the canonical no-swizzle core-matrix layout
//     (8 rows x 16 bytes), zero padded to whole 32-k blocks;
//   * a cluster of 1 to 8 CTAs per (f, 128 x kN output tile), kN 64 or 128,
//     each CTA a contiguous part of the 32-k blocks: one lane stages tiles
//     with bulk copies (cp.async.bulk, mbarrier transaction count, bounded
//     waits), another issues tcgen05.mma kind::tf32 (M=128, N=2 kN, K=8) into
//     [Re | Im] accumulators in TMEM, FP32, while later tiles' copies land:
//       [Re | Im] += (Ar_hi + Ar_lo)[Br | Bi] + (Ai_hi + Ai_lo)[-Bi | Br]
//     with B split alike and the lo x lo terms dropped (3xTF32: Ootomo and
//     Yokota, "Recovering single precision accuracy from Tensor Cores while
//     surpassing the FP32 theoretical peak performance", IJHPCA 2022); B's
//     rows are stored once as [-Bi | Br | Bi], which holds both operands;
//   * every 32-k block goes to one of two TMEM buffers from zero; epilogue
//     warps read a finished buffer back (tcgen05.ld) and add it into FP32
//     registers with round-to-nearest while the next block fills the other
//     buffer, since the tensor cores' own accumulation rounds toward zero
//     (Ootomo and Yokota keep the long sum outside the tensor cores for the
//     same reason); the CTAs' sums meet in shared memory, in rank order, and
//     leave as whole rows of complex64.
// With a small summed dimension (the reference's own buckets sum one binary
// index, K = 2) a tile would be mostly padding, and a CUDA-core kernel
// computes the same sums in FP32.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <type_traits>

#include "plan.h"

namespace qtb {

// ----------------------------------------------------------------- CUDA cores
// The outputs of both kernels below are [F][M][N]; a thread takes a block of
// kRows rows (m) x 1 or 2 columns (n), then the block one grid width further.
// A block's index (f, row block, column block) is divided out once and every
// step adds the grid width in the same mixed radix, so that the loop has no
// division: two 64-bit divisions per output made the kernels issue-bound
// (1.8 TB/s of 6.5 for the outer product, 1.2 TB/s for K = 2).  Rows in a
// block share the load of their b, and with kPairs (N even, 16-byte aligned
// pointers) two columns load and store 16 bytes.  256 x 256 x 256 outer
// product: 73.6 -> 23.3 us; K = 2, F = 64, M = N = 512: 116 -> 26.7 us (134 MB
// written; a memset of it takes 20.6 us).
// I: 32-bit indices, or 64-bit where a dimension needs them.
template <typename I>
struct FlatIndex {
    uint64_t f;
    I m, n;
};

template <typename I>
struct FlatShape {
    uint64_t blocks;     // F x row blocks x column blocks
    I M, N;
    I rows, cols;        // row and column blocks
    FlatIndex<I> step;   // the grid width
};

template <typename I>
__device__ __forceinline__ FlatIndex<I> flat_start(uint64_t i, const FlatShape<I>& s) {
    const uint64_t row = i / s.cols;
    return FlatIndex<I>{row / s.rows, (I)(row % s.rows), (I)(i % s.cols)};
}

template <typename I>
__device__ __forceinline__ void flat_step(FlatIndex<I>& x, const FlatShape<I>& s) {
    x.n += s.step.n;
    x.m += s.step.m;
    x.f += s.step.f;
    if (x.n >= s.cols) {
        x.n -= s.cols;
        ++x.m;
    }
    if (x.m >= s.rows) {
        x.m -= s.rows;
        ++x.f;
    }
}

constexpr int kFlatThreads = 256;
constexpr int kFlatBlocksPerSm = 4;   // all resident at 64 registers (48 spill: K = 2 41 us; 74 and 8 per SM: 42)
constexpr int kFlatRows = 4;
// Outputs from here on are stored evict-first, when pairs of columns are (8-byte
// stores were not measured and stay plain).  What is gained is write-back that
// no longer waits for lines in L2 to be evicted: a call alone, or followed by
// work on other data, is faster, a reader of the output right behind it finds
// as little in L2 either way.  Plain against evict-first, and each with a
// reduction of the output behind it: K = 2 into 128 MiB 33.1 against 24.9 us
// and 67.9 / 68.1, the outer product 24.8 against 23.7 and 60.0 / 59.8; around
// the line K = 2 takes 26.2 and 27.3 us (100.8 and 103.8 MiB, plain), 22.2
// and 23.2 (104.8 and 111.8, evict-first), with the reduction 53.9, 55.2, 55.5
// and 59.8.  At 64 MiB, where a reader finds the output in L2, 18.9 against
// 14.6 but 33.1 / 39.2.
constexpr uint64_t kFlatStreamBytes = 104ull << 20;
static bool flat_stream(uint64_t outputs) { return outputs * sizeof(float2) >= kFlatStreamBytes; }

template <typename I>
static FlatShape<I> flat_shape(uint64_t F, uint64_t M, uint64_t N, int block_rows, int block_cols, unsigned* grid) {
    FlatShape<I> s{};
    s.M = (I)M;
    s.N = (I)N;
    s.rows = (I)((M + block_rows - 1) / block_rows);
    s.cols = (I)(N / block_cols);
    s.blocks = F * s.rows * s.cols;
    *grid = (unsigned)std::min<uint64_t>((s.blocks + kFlatThreads - 1) / kFlatThreads, 148ull * kFlatBlocksPerSm);
    const uint64_t width = (uint64_t)*grid * kFlatThreads;
    s.step = FlatIndex<I>{width / s.cols / s.rows, (I)(width / s.cols % s.rows), (I)(width % s.cols)};
    return s;
}

// Rows per thread: four where that still leaves every thread of the grid a
// block and the indices 32 bits, else one (below, the call is launch-bound:
// 8-9 us with either).
static int flat_rows(uint64_t outputs, uint64_t M, uint64_t N) {
    const uint64_t enough = 148ull * kFlatBlocksPerSm * kFlatThreads * kFlatRows;
    return outputs >= enough && M < (1ull << 30) && N < (1ull << 30) ? kFlatRows : 1;
}

template <bool kPairs>
__device__ __forceinline__ void flat_load(const float2* p, float2 (&v)[kPairs ? 2 : 1]) {
    if constexpr (kPairs) {
        const float4 q = *reinterpret_cast<const float4*>(p);
        v[0] = make_float2(q.x, q.y);
        v[1] = make_float2(q.z, q.w);
    } else {
        v[0] = *p;
    }
}

// kStream: evict-first, for an output that L2 (126 MB) does not hold anyway,
// so that its lines make room for one another as they are written back.
template <bool kPairs, bool kStream>
__device__ __forceinline__ void flat_store(float2* p, const float2 (&v)[kPairs ? 2 : 1]) {
    if constexpr (kPairs) {
        const float4 q = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
        if constexpr (kStream) __stcs(reinterpret_cast<float4*>(p), q);
        else *reinterpret_cast<float4*>(p) = q;
    } else {
        static_assert(!kStream, "single columns are stored plainly");
        *p = v[0];
    }
}

// c[f,m,n] = a[f,m] * b[f,n].
template <int kRows, bool kPairs, bool kStream, typename I>
__global__ void __launch_bounds__(kFlatThreads, kFlatBlocksPerSm) qtb_outer_kernel(const float2* __restrict__ a,
                                                                 const float2* __restrict__ b, float2* __restrict__ c,
                                                                 const FlatShape<I> s) {
    constexpr int kCols = kPairs ? 2 : 1;
    uint64_t i = blockIdx.x * (uint64_t)kFlatThreads + threadIdx.x;
    if (i >= s.blocks) return;
    FlatIndex<I> x = flat_start(i, s);
    for (; i < s.blocks; i += (uint64_t)gridDim.x * kFlatThreads, flat_step(x, s)) {
        const I m = x.m * kRows, n = x.n * kCols;
        float2 v[kCols], u[kRows];
        flat_load<kPairs>(b + x.f * s.N + n, v);
#pragma unroll
        for (int r = 0; r < kRows; ++r) u[r] = a[x.f * s.M + (kRows == 1 || m + r < s.M ? m + r : m)];
        float2* out = c + (x.f * s.M + m) * s.N + n;
#pragma unroll
        for (int r = 0; r < kRows; ++r, out += s.N) {
            float2 p[kCols];
#pragma unroll
            for (int e = 0; e < kCols; ++e)
                p[e] = make_float2(fmaf(u[r].x, v[e].x, -(u[r].y * v[e].y)), fmaf(u[r].y, v[e].x, u[r].x * v[e].y));
            if (kRows == 1 || m + r < s.M) flat_store<kPairs, kStream>(out, p);
        }
    }
}

// C[f,m,n] = sum_k A[k,f,m] B[k,f,n], FP32 sums over k in order.  kAhead k
// values are loaded together, so that a long sum over few outputs waits for
// memory once per kAhead terms.
template <int kRows, bool kPairs, bool kStream, int kAhead, typename I>
__global__ void __launch_bounds__(kFlatThreads, kFlatBlocksPerSm) qtb_contract_simt_kernel(const float2* __restrict__ A,
                                                                         const float2* __restrict__ B,
                                                                         float2* __restrict__ C, uint64_t K,
                                                                         uint64_t a_stride, uint64_t b_stride,
                                                                         int* status, const FlatShape<I> s) {
    constexpr int kCols = kPairs ? 2 : 1;
    if (blockIdx.x == 0 && threadIdx.x < 4) status[threadIdx.x] = 0;   // nothing here can fail
    uint64_t i = blockIdx.x * (uint64_t)kFlatThreads + threadIdx.x;
    if (i >= s.blocks) return;
    FlatIndex<I> x = flat_start(i, s);
    for (; i < s.blocks; i += (uint64_t)gridDim.x * kFlatThreads, flat_step(x, s)) {
        const I m = x.m * kRows, n = x.n * kCols;
        const float2* pa = A + x.f * s.M + m;
        const float2* pb = B + x.f * s.N + n;
        float2 sum[kRows][kCols];
#pragma unroll
        for (int r = 0; r < kRows; ++r)
#pragma unroll
            for (int e = 0; e < kCols; ++e) sum[r][e] = make_float2(0.f, 0.f);
        auto terms = [&](auto count) {
            constexpr int kCount = decltype(count)::value;
            float2 u[kCount][kRows], v[kCount][kCols];
#pragma unroll
            for (int k = 0; k < kCount; ++k) {
                flat_load<kPairs>(pb, v[k]);
#pragma unroll
                for (int r = 0; r < kRows; ++r) u[k][r] = pa[kRows == 1 || m + r < s.M ? r : 0];
                pa += a_stride;
                pb += b_stride;
            }
#pragma unroll
            for (int k = 0; k < kCount; ++k)
#pragma unroll
                for (int r = 0; r < kRows; ++r)
#pragma unroll
                    for (int e = 0; e < kCols; ++e) {
                        sum[r][e].x = fmaf(u[k][r].x, v[k][e].x, sum[r][e].x);
                        sum[r][e].x = fmaf(-u[k][r].y, v[k][e].y, sum[r][e].x);
                        sum[r][e].y = fmaf(u[k][r].x, v[k][e].y, sum[r][e].y);
                        sum[r][e].y = fmaf(u[k][r].y, v[k][e].x, sum[r][e].y);
                    }
        };
        uint64_t k = 0;
        for (; k + kAhead <= K; k += kAhead) terms(std::integral_constant<int, kAhead>());
        for (; k < K; ++k) terms(std::integral_constant<int, 1>());
        float2* out = C + (x.f * s.M + m) * s.N + n;
#pragma unroll
        for (int r = 0; r < kRows; ++r, out += s.N)
            if (kRows == 1 || m + r < s.M) flat_store<kPairs, kStream>(out, sum[r]);
    }
}

static bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// ----------------------------------------------------------------- tensor cores
constexpr uint32_t kTcM = 128;                        // output tile rows (A tile rows)
constexpr uint32_t kTcK = 32;                         // k per accumulation block (K padded to it)
constexpr uint32_t kTcStageK = 8;                     // k per staged tile (one MMA k step)
constexpr uint32_t kTcStagesPerBlock = kTcK / kTcStageK;
constexpr uint32_t kTcAPlanes = 4;                    // Ar_hi Ar_lo Ai_hi Ai_lo
constexpr uint32_t kTcBPlanes = 2;                    // [-Bi | Br | Bi]: hi, lo
constexpr uint32_t kTcAWords = kTcM * kTcStageK;      // 1024 x 32-bit = 4 KB per A plane and stage
constexpr uint32_t kTcChunks = kTcStageK / 4;         // 16-byte k chunks per row of a tile
constexpr uint32_t kTcSpinLimit = 1u << 24;           // bounded mbarrier waits (~1 s)
constexpr int kTcStatusTimeout = 2;

// What depends on the output tile's columns kN (complex).
template <uint32_t kN>
struct TcTile {
    static constexpr uint32_t kBWords = 3 * kN * kTcStageK;                        // per B plane and stage
    static constexpr uint32_t kStageWords = kTcAPlanes * kTcAWords + kTcBPlanes * kBWords;   // 40 or 28 KB
    static constexpr uint32_t kStages = kN == 128 ? 5 : 7;                         // about 200 KB
    static constexpr uint32_t kEpilogueWarps = kN / 16;                            // 64 columns x 32 rows each
    static constexpr uint32_t kThreads = 32 * (kEpilogueWarps + 2);                // + the MMA and the copy warp
    static constexpr uint32_t kBufCols = 2 * kN;                                   // one accumulator buffer [Re | Im]
    static constexpr uint32_t kTmemCols = 2 * kBufCols;
    // instruction descriptor: FP32 accumulator, TF32 A and B, both K-major,
    // N = 2 kN (>> 3 at bit 17), M = 128 (>> 4 at bit 24)
    static constexpr uint32_t kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((2 * kN >> 3) << 17) | ((kTcM >> 4) << 24);
    // the finished tile in the stages' place: rows of kN complex64, padded by
    // 16 bytes so that the rows of a warp's lanes start on different banks
    static constexpr uint32_t kRowBytes = kN * 8 + 16;
    static constexpr size_t kBarOffset = (size_t)kStages * kStageWords * 4;
    static constexpr size_t kSmemBytes = kBarOffset + (2 * kStages + 4) * 8 + 16;
    static_assert(kTcM * kRowBytes <= kBarOffset, "the tile fits the stages");
};

__device__ __forceinline__ uint32_t tf32_round(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

// TF32 hi / lo of one component: hi rounded to nearest, lo the rounded remainder.
__device__ __forceinline__ void tf32_split(float x, uint32_t& hi, uint32_t& lo) {
    hi = tf32_round(x);
    lo = tf32_round(x - __uint_as_float(hi));
}

// TF32 hi / lo of four k of one row: one 16-byte chunk of a core matrix each.
__device__ __forceinline__ void tf32_split4(const float (&x)[4], uint4& hi, uint4& lo) {
    tf32_split(x[0], hi.x, lo.x);
    tf32_split(x[1], hi.y, lo.y);
    tf32_split(x[2], hi.z, lo.z);
    tf32_split(x[3], hi.w, lo.w);
}

// The planes of A and of B.  A[k][f][m] -> tiles of 128 rows x 8 k, ordered
// (f, row tile, k tile), the four planes of a tile consecutive, so that one
// bulk copy stages all four; B[k][f][n] -> tiles of kN columns x 8 k, ordered
// (f, column tile, k tile), two planes of rows [-Bi | Br | Bi] (the negation
// is exact in TF32).  A thread takes four k of one row or column: its reads
// are coalesced over the rows, and its 16-byte writes fill 128-byte lines of
// eight rows, so nothing is exchanged between threads.  Element (r, k) of a
// plane: core matrix (r / 8, k / 4), 8 rows of 16 bytes each.  The first
// blocks split A, the others B; the status word is cleared for the kernel
// that follows.
template <uint32_t kN>
__global__ void __launch_bounds__(256) qtb_tc_split_kernel(const float2* __restrict__ A, const float2* __restrict__ B,
                                                           uint4* __restrict__ Ap, uint4* __restrict__ Bp, uint32_t K,
                                                           uint32_t F, uint32_t M, uint32_t N, uint32_t k_tiles,
                                                           uint32_t row_tiles, uint32_t col_tiles, uint32_t a_blocks,
                                                           int* status) {
    if (blockIdx.x == 0 && threadIdx.x < 4) status[threadIdx.x] = 0;
    const bool is_a = blockIdx.x < a_blocks;
    const uint32_t rows = is_a ? kTcM : kN, tiles = is_a ? row_tiles : col_tiles, width = is_a ? M : N;
    const uint64_t unit = (uint64_t)(is_a ? blockIdx.x : blockIdx.x - a_blocks) * 256u + threadIdx.x;
    const uint32_t r = (uint32_t)(unit % rows), c = (uint32_t)(unit / rows) % kTcChunks;
    const uint64_t tile = unit / (rows * kTcChunks);
    if (tile >= (uint64_t)F * tiles * k_tiles) return;
    const uint32_t kt = (uint32_t)(tile % k_tiles), rt = (uint32_t)(tile / k_tiles % tiles);
    const uint64_t f = tile / k_tiles / tiles;
    const uint64_t col = (uint64_t)rt * rows + r;
    const float2* src = is_a ? A : B;
    float re[4], im[4];
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) {
        const uint64_t kk = (uint64_t)kt * kTcStageK + 4u * c + e;
        const float2 v = (col < width && kk < K) ? src[(kk * F + f) * width + col] : make_float2(0.f, 0.f);
        re[e] = v.x;
        im[e] = v.y;
    }
    uint4 rh, rl, ih, il;
    tf32_split4(re, rh, rl);
    tf32_split4(im, ih, il);
    auto chunk = [&](uint32_t row) { return ((row >> 3) * kTcChunks + c) * 8u + (row & 7u); };
    if (is_a) {
        constexpr uint32_t kPlane = kTcAWords / 4;
        uint4* dst = Ap + tile * (kTcAPlanes * kPlane) + chunk(r);
        dst[0] = rh;
        dst[kPlane] = rl;
        dst[2 * kPlane] = ih;
        dst[3 * kPlane] = il;
    } else {
        constexpr uint32_t kPlane = TcTile<kN>::kBWords / 4;
        auto negated = [](uint4 v) {
            return make_uint4(v.x ^ 0x80000000u, v.y ^ 0x80000000u, v.z ^ 0x80000000u, v.w ^ 0x80000000u);
        };
        uint4* dst = Bp + tile * (kTcBPlanes * kPlane);
        dst[chunk(r)] = negated(ih);
        dst[chunk(kN + r)] = rh;
        dst[chunk(2 * kN + r)] = ih;
        dst[kPlane + chunk(r)] = negated(il);
        dst[kPlane + chunk(kN + r)] = rl;
        dst[kPlane + chunk(2 * kN + r)] = il;
    }
}

__device__ __forceinline__ uint32_t tc_smem(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor of a K-major, no-swizzle operand tile:
// start address, leading byte offset (next 16-byte k chunk: 128 B), stride
// byte offset (next 8-row group: kTcChunks chunks x 128 B), version 1.
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) |
           ((uint64_t)(kTcChunks * 128u >> 4) << 32) | (uint64_t(1) << 46);
}

__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

// Bounded wait for the mbarrier phase `parity`; false after `limit` polls.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
    uint32_t done = 0;
    for (uint32_t it = 0; it < limit; ++it) {
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if (it > 64) __nanosleep(64);
    }
    return false;
}

// 32 32-bit TMEM columns of this thread's lane at each of two addresses,
// one wait for both loads (a load's latency, not its width, is what costs
// while the MMAs run); the wait is in the same asm as the loads, so no use of
// the registers can be scheduled before it.
__device__ __forceinline__ void tc_ld2x32(uint32_t ta, uint32_t tb, uint32_t (&r)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,"
        "%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,"
        "%24,%25,%26,%27,%28,%29,%30,%31}, [%64];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%32,%33,%34,%35,%36,%37,%38,%39,"
        "%40,%41,%42,%43,%44,%45,%46,%47,"
        "%48,%49,%50,%51,%52,%53,%54,%55,"
        "%56,%57,%58,%59,%60,%61,%62,%63}, [%65];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
          "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
          "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
          "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
          "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
        : "r"(ta), "r"(tb)
        : "memory");
}

__device__ __forceinline__ void tc_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// Cluster of `split` CTAs (grid x = column tiles x split) per (f, 128 x kN
// tile of C); CTA `rank` takes its part of the 32-k blocks.
//   * One lane of the last warp stages tiles with bulk copies into kStages
//     shared-memory stages as they come free; one lane of the warp before it
//     issues the MMAs and never waits for one (a single lane doing both
//     waited for each tile's MMAs to refill its stage: 1150 of the 1550
//     cycles per tile, whatever the tile's MMAs).  kTcStagesPerBlock tiles
//     make one 32-k block, accumulated in one of two TMEM buffers from zero.
//   * The epilogue warps (32 TMEM lanes x 64 columns each) read a finished
//     block's buffer with tcgen05.ld and add it into FP32 registers with
//     round-to-nearest (the tensor cores' own accumulation rounds toward
//     zero, which over a long k range biases the sum: about 3e-5 relative at
//     K = 1000), while the next block's MMAs fill the other buffer.
// mbarriers: full[s] (stage s landed), empty[s] (stage s's MMAs done),
// tfull[b] (buffer b's block done), tempty[b] (buffer b read by every
// epilogue thread).  Every wait is bounded; on a timeout the status word is
// set, every role stops, and the CTA waits (bounded, in phase order) for its
// copies and MMAs in flight before freeing TMEM; it still meets its
// cluster's barriers, and no CTA of the cluster stores its part of the tile,
// whose sums are not finished.  kTest: the self-test's, whose CTAs of rank
// `stall` stage nothing and whose waits run out after spin_limit polls.
// What bounds it: shared memory.  A 128 x 128 tile's six MMAs take 768 tensor
// cycles per 8 k, read 72 KB of operands and see 40 KB written: 875 cycles at
// 128 bytes each (measured about 1100).  128 x 64 tiles with B stored as both
// [Br | Bi] and [-Bi | Br] also pulled 32 KB per 384 cycles through L2.
// K=1024, F=2, M=N=1024: 165 -> 112 us per call; K=500, F=3, M=333, N=190: 71 -> 23 us
// (4 CTAs per tile in place of 27 serial ones).  Measured and not kept: B as
// [Br | Bi] with the negative products through the descriptor's negate-A bit
// (32 KB per tile but N = 128 MMAs, 128 operand bytes per cycle: 116 us).
template <uint32_t kN, bool kTest>
__global__ void __launch_bounds__(TcTile<kN>::kThreads, 1)
qtb_tc_contract_kernel(const uint32_t* __restrict__ Ap, const uint32_t* __restrict__ Bp, float2* __restrict__ C,
                       uint32_t M, uint32_t N, uint32_t row_tiles, uint32_t col_tiles, uint32_t k_blocks,
                       uint32_t split, uint32_t vec, int* status, uint32_t spin_limit, uint32_t stall) {
    const uint32_t limit = kTest ? spin_limit : kTcSpinLimit;
    using T = TcTile<kN>;
    constexpr uint32_t NS = T::kStages;
    extern __shared__ __align__(1024) unsigned char smem[];
    // [stage 0: A planes x4 | B planes x2][stage 1] ..., the mbarriers, the TMEM slot
    uint32_t* stages = reinterpret_cast<uint32_t*>(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T::kBarOffset);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NS + 4);
    __shared__ volatile int s_ok;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t nt = blockIdx.x / split, rank = blockIdx.x % split, mt = blockIdx.y, f = blockIdx.z;
    const uint32_t block0 = k_blocks * rank / split, n_blocks = k_blocks * (rank + 1) / split - block0;
    const uint32_t n_tiles = n_blocks * kTcStagesPerBlock;
    auto full = [&](uint32_t s) { return tc_smem(&bars[s]); };
    auto empty = [&](uint32_t s) { return tc_smem(&bars[NS + s]); };
    auto tfull = [&](uint32_t b) { return tc_smem(&bars[2 * NS + b]); };
    auto tempty = [&](uint32_t b) { return tc_smem(&bars[2 * NS + 2 + b]); };
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < 2 * NS + 2; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&bars[i])));
        for (uint32_t b = 0; b < 2; ++b)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tempty(b)), "r"(32 * T::kEpilogueWarps));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_ok = 1;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(tmem_slot)),
                     "r"(T::kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tmem_slot;
    // launched while the split kernel still runs: its planes and the status
    // word are ready from here on
    asm volatile("griddepcontrol.wait;" ::: "memory");
    auto fail_once = [&]() {
        if (s_ok) atomicOr(status, kTcStatusTimeout);
        s_ok = 0;
    };
    float acc_re[64], acc_im[64];
    if (warp == T::kEpilogueWarps + 1) {   // the copies
        if (lane == 0) {
            // this CTA's tiles: (f, row tile, k tile) of A, (f, column tile, k tile) of B
            const uint64_t k_tiles = (uint64_t)k_blocks * kTcStagesPerBlock, kt0 = (uint64_t)block0 * kTcStagesPerBlock;
            const uint32_t* a_f = Ap + (((uint64_t)f * row_tiles + mt) * k_tiles + kt0) * (kTcAPlanes * kTcAWords);
            const uint32_t* b_f = Bp + (((uint64_t)f * col_tiles + nt) * k_tiles + kt0) * (kTcBPlanes * T::kBWords);
            uint32_t loaded = 0;
            for (; loaded < n_tiles && s_ok && !(kTest && rank == stall); ++loaded) {   // tile `loaded` into stage loaded % NS
                const uint32_t s = loaded % NS;
                if (loaded >= NS && !tc_wait(empty(s), (loaded / NS - 1u) & 1u, limit)) {
                    fail_once();   // the MMAs have not read the stage's previous tile
                    break;
                }
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full(s)),
                             "r"(T::kStageWords * 4u)
                             : "memory");
                // the tile's planes are consecutive in global memory and in the stage
                const uint32_t dst = tc_smem(stages + s * T::kStageWords);
                tc_bulk(dst, a_f + (uint64_t)loaded * kTcAPlanes * kTcAWords, kTcAPlanes * kTcAWords * 4u, full(s));
                tc_bulk(dst + kTcAPlanes * kTcAWords * 4u, b_f + (uint64_t)loaded * kTcBPlanes * T::kBWords,
                        kTcBPlanes * T::kBWords * 4u, full(s));
            }
            // no copy may still write shared memory when it is reused: wait
            // (bounded) for each stage's last one
            for (uint32_t i = loaded > NS ? loaded - NS : 0u; i < loaded; ++i)
                tc_wait(full(i % NS), (i / NS) & 1u, kTcSpinLimit);
        }
        __syncwarp();
    } else if (warp == T::kEpilogueWarps) {   // the MMAs
        if (lane == 0) {
            uint32_t committed = 0;
            for (uint32_t i = 0; i < n_tiles && s_ok; ++i) {
                const uint32_t s = i % NS, b = i / kTcStagesPerBlock, buf = b & 1u;
                const bool block_first = i % kTcStagesPerBlock == 0;
                if (block_first && b >= 2 && !tc_wait(tempty(buf), ((b - 2) >> 1) & 1u, limit)) {
                    fail_once();   // the epilogue has not read this buffer's previous block
                    break;
                }
                if (!tc_wait(full(s), (i / NS) & 1u, limit)) {
                    fail_once();
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                // A planes: 0 Ar_hi 1 Ar_lo 2 Ai_hi 3 Ai_lo.  B rows [-Bi | Br | Bi]:
                // from row kN on [Br | Bi], from row 0 on [-Bi | Br]
                const uint32_t abase = tc_smem(stages + s * T::kStageWords), bbase = abase + kTcAPlanes * kTcAWords * 4u;
                const uint32_t acc = tmem + buf * T::kBufCols;
                auto da = [&](uint32_t q) { return tc_desc(abase + q * kTcAWords * 4u); };
                auto db = [&](uint32_t q, uint32_t row) {
                    return tc_desc(bbase + q * T::kBWords * 4u + row * (kTcStageK * 4u));
                };
                tc_mma(acc, da(0), db(0, kN), T::kIdesc, block_first ? 0u : 1u);   // a block starts from zero
                tc_mma(acc, da(0), db(1, kN), T::kIdesc, 1u);
                tc_mma(acc, da(1), db(0, kN), T::kIdesc, 1u);
                tc_mma(acc, da(2), db(0, 0), T::kIdesc, 1u);
                tc_mma(acc, da(2), db(1, 0), T::kIdesc, 1u);
                tc_mma(acc, da(3), db(0, 0), T::kIdesc, 1u);
                tc_commit(empty(s));
                committed = i + 1;
                if (i % kTcStagesPerBlock == kTcStagesPerBlock - 1) tc_commit(tfull(buf));
            }
            // no MMA may still read shared memory or write TMEM when they are
            // reused or freed: wait (bounded) for each stage's last commit
            for (uint32_t i = committed > NS ? committed - NS : 0u; i < committed; ++i)
                tc_wait(empty(i % NS), (i / NS) & 1u, kTcSpinLimit);
        }
        __syncwarp();
    } else {
#pragma unroll
        for (uint32_t j = 0; j < 64; ++j) acc_re[j] = acc_im[j] = 0.f;
        // this warp's 32 TMEM lanes and 64 columns
        const uint32_t addr = tmem + (((warp & 3u) * 32u) << 16) + (warp >> 2) * 64u;
        for (uint32_t b = 0; b < n_blocks; ++b) {
            const uint32_t buf = b & 1u;
            if (!s_ok) break;
            if (!tc_wait(tfull(buf), (b >> 1) & 1u, limit)) {
                fail_once();
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
            for (uint32_t c0 = 0; c0 < 64; c0 += 32u) {
                uint32_t v[64];
                tc_ld2x32(addr + buf * T::kBufCols + c0, addr + buf * T::kBufCols + kN + c0, v);
#pragma unroll
                for (uint32_t j = 0; j < 32; ++j) {
                    acc_re[c0 + j] += __uint_as_float(v[j]);
                    acc_im[c0 + j] += __uint_as_float(v[32 + j]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tempty(buf)) : "memory");
        }
    }
    __syncthreads();   // no copy or MMA is left: the stages become the finished tile
    if (warp < T::kEpilogueWarps) {
        float4* row = reinterpret_cast<float4*>(smem + ((warp & 3u) * 32u + lane) * T::kRowBytes + (warp >> 2) * 512u);
#pragma unroll
        for (uint32_t j = 0; j < 64; j += 2) row[j / 2] = make_float4(acc_re[j], acc_im[j], acc_re[j + 1], acc_im[j + 1]);
    }
    auto cluster_sync = [&]() {
        if (split > 1)
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        else
            __syncthreads();
    };
    cluster_sync();
    // rows rank, rank + split, ... of the tile, the CTAs' sums added in rank
    // order; a warp stores whole rows, two columns per lane
    uint32_t ok = s_ok;
    for (uint32_t q = 0; q < split && split > 1; ++q) {   // a CTA that gave up leaves its part of the sums out
        uint32_t peer, peer_ok;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(tc_smem(const_cast<const int*>(&s_ok))), "r"(q));
        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(peer_ok) : "r"(peer) : "memory");
        ok &= peer_ok;
    }
    for (uint32_t r = rank + warp * split; r < kTcM; r += (T::kEpilogueWarps + 2) * split) {
        const uint32_t m = mt * kTcM + r;
        if (m >= M) break;
        float2* out = C + ((uint64_t)f * M + m) * N + (uint64_t)nt * kN;
        for (uint32_t c = 2u * lane; c < kN; c += 64u) {
            const uint32_t at = tc_smem(smem) + r * T::kRowBytes + c * 8u;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (uint32_t q = 0; q < split; ++q) {
                float4 x;
                if (split > 1) {
                    uint32_t peer;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(q));
                    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                                 : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(peer) : "memory");
                } else {
                    x = *reinterpret_cast<const float4*>(smem + r * T::kRowBytes + c * 8u);
                }
                v = q == 0 ? x : make_float4(v.x + x.x, v.y + x.y, v.z + x.z, v.w + x.w);
            }
            const uint32_t n = nt * kN + c;
            if (ok && vec && n + 1 < N) {
                *reinterpret_cast<float4*>(out + c) = v;
            } else if (ok) {
                if (n < N) out[c] = make_float2(v.x, v.y);
                if (n + 1 < N) out[c + 1] = make_float2(v.z, v.w);
            }
        }
    }
    cluster_sync();   // a CTA's shared memory is read until here
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::kTmemCols));
}

static uint64_t round_up(uint64_t x, uint64_t m) { return (x + m - 1) / m * m; }

// Whether the contract-sum runs on the tensor cores: mode 1 never, 2
// always, 0 when the summed dimension and both tile dimensions are large
// enough for the tiles to be mostly data.
static bool use_tensor_cores(int32_t mode, int64_t K, int64_t M, int64_t N) {
    if (mode == 1) return false;
    if (mode == 2) return true;
    return K >= 32 && M >= 64 && N >= 64;
}

// Tile columns and CTAs per tile of a shape: the smallest estimate of rounds
// of CTAs on 148 SMs x 32-k blocks per CTA x time per block (128 x 128 tiles
// take about 1.6 times as long per block as 128 x 64 ones: 40 against 28 KB
// through L2, 768 against 384 tensor cycles per 8 k, both partly hidden),
// plus the tile's epilogue (about four blocks' time) and the cluster's sums.
struct TcShape {
    uint32_t n, split;
    uint64_t k_blocks, row_tiles, col_tiles;
};

static TcShape tc_shape(int64_t K, int64_t F, int64_t M, int64_t N) {
    TcShape best{};
    double least = 1e300;
    for (uint32_t n : {128u, 64u})
        for (uint32_t split : {1u, 2u, 4u, 8u}) {
            TcShape s{n, split, round_up(K, kTcK) / kTcK, round_up(M, kTcM) / kTcM, round_up(N, n) / n};
            if (split > 1 && s.k_blocks < 2 * split) continue;
            const uint64_t ctas = (uint64_t)F * s.row_tiles * s.col_tiles * split;
            const double rounds = (double)((ctas + 147) / 148);
            const double cost = rounds * ((double)((s.k_blocks + split - 1) / split) + 4.0 + (split > 1 ? 1.0 : 0.0)) *
                                (n == 128 ? 1.6 : 1.0);
            if (cost < least) {
                least = cost;
                best = s;
            }
        }
    return best;
}

static int cuda_fail_c(cudaError_t e, const char* what) {
    return fail(QTB_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace qtb

using namespace qtb;

extern "C" {

int qtb_contract_outer_c64(const void* a, const void* b, void* c, int64_t n, int64_t m, int64_t k,
                           void* stream) {
    if (!a || !b || !c || n < 1 || m < 1 || k < 1) return fail(QTB_ERR_ARG, "contract_outer: bad arguments");
    const float2 *pa = static_cast<const float2*>(a), *pb = static_cast<const float2*>(b);
    float2* pc = static_cast<float2*>(c);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int rows = flat_rows((uint64_t)n * m * k, m, k);
    const bool pairs = rows > 1 && k % 2 == 0 && aligned16(b) && aligned16(c);
    const bool evict = flat_stream((uint64_t)n * m * k);
    unsigned grid = 0;
    if (rows > 1) {
        const FlatShape<uint32_t> s = flat_shape<uint32_t>(n, m, k, rows, pairs ? 2 : 1, &grid);
        const auto run = !pairs  ? qtb_outer_kernel<kFlatRows, false, false, uint32_t>
                        : evict ? qtb_outer_kernel<kFlatRows, true, true, uint32_t>
                                : qtb_outer_kernel<kFlatRows, true, false, uint32_t>;
        run<<<grid, kFlatThreads, 0, st>>>(pa, pb, pc, s);
    } else {
        const FlatShape<uint64_t> s = flat_shape<uint64_t>(n, m, k, 1, 1, &grid);
        qtb_outer_kernel<1, false, false><<<grid, kFlatThreads, 0, st>>>(pa, pb, pc, s);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? QTB_OK : cuda_fail_c(e, "contract_outer launch");
}

int qtb_contract_sum_scratch_bytes(int64_t K, int64_t F, int64_t M, int64_t N, int32_t mode, size_t* bytes) {
    if (!bytes || K < 1 || F < 1 || M < 1 || N < 1 || mode < 0 || mode > 2)
        return fail(QTB_ERR_ARG, "contract_sum_scratch_bytes: bad arguments");
    if (!use_tensor_cores(mode, K, M, N)) {
        *bytes = 16;
        return QTB_OK;
    }
    const TcShape s = tc_shape(K, F, M, N);
    // four planes of A, two of B with three rows per column
    *bytes = 256 + (uint64_t)F * (kTcAPlanes * s.row_tiles * kTcM + kTcBPlanes * 3 * s.col_tiles * s.n) * s.k_blocks * kTcK * 4;
    return QTB_OK;
}

}  // extern "C"

template <uint32_t kN, bool kTest>
static cudaError_t tc_launch(const TcShape& t, const float2* A, const float2* B, float2* C, int64_t K, int64_t F,
                             int64_t M, int64_t N, void* scratch, cudaStream_t st, uint32_t spin_limit, uint32_t stall) {
    using T = TcTile<kN>;
    int* status = static_cast<int*>(scratch);
    const uint64_t k_tiles = t.k_blocks * kTcStagesPerBlock;
    uint32_t* Ap = reinterpret_cast<uint32_t*>(static_cast<char*>(scratch) + 256);
    uint32_t* Bp = Ap + (uint64_t)F * t.row_tiles * k_tiles * kTcAPlanes * kTcAWords;
    const uint64_t a_blocks = (uint64_t)F * t.row_tiles * k_tiles;   // 128 rows x 2 chunks = 256 threads
    const uint64_t b_blocks = ((uint64_t)F * t.col_tiles * k_tiles * kN * kTcChunks + 255) / 256;
    qtb_tc_split_kernel<kN><<<(unsigned)(a_blocks + b_blocks), 256, 0, st>>>(
        A, B, reinterpret_cast<uint4*>(Ap), reinterpret_cast<uint4*>(Bp), (uint32_t)K, (uint32_t)F, (uint32_t)M,
        (uint32_t)N, (uint32_t)k_tiles, (uint32_t)t.row_tiles, (uint32_t)t.col_tiles, (uint32_t)a_blocks, status);
    // per device and cheap: set on every call
    cudaError_t e = cudaFuncSetAttribute(qtb_tc_contract_kernel<kN, kTest>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)T::kSmemBytes);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(t.col_tiles * t.split), (unsigned)t.row_tiles, (unsigned)F);
    cfg.blockDim = dim3(T::kThreads);
    cfg.dynamicSmemBytes = T::kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // griddepcontrol.wait in the kernel
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = t.split;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = t.split > 1 ? 2 : 1;
    const uint32_t vec = N % 2 == 0 && aligned16(C);
    return cudaLaunchKernelEx(&cfg, qtb_tc_contract_kernel<kN, kTest>, (const uint32_t*)Ap, (const uint32_t*)Bp, C, (uint32_t)M,
                              (uint32_t)N, (uint32_t)t.row_tiles, (uint32_t)t.col_tiles, (uint32_t)t.k_blocks, t.split,
                              vec, status, spin_limit, stall);
}

// The tensor-core contract-sum; arguments and scratch size checked by the caller.
template <bool kTest>
static int tc_sum(const TcShape& t, const void* A, const void* B, void* C, int64_t K, int64_t F, int64_t M, int64_t N,
                  void* scratch, cudaStream_t st, uint32_t spin_limit = 0, uint32_t stall = 0) {
    const uint64_t k_tiles = t.k_blocks * kTcStagesPerBlock;
    if (t.row_tiles > 65535 || F > 65535 || t.col_tiles * t.split > (1u << 30) || K > (1ll << 30) ||
        (uint64_t)F * (t.row_tiles + t.col_tiles) * k_tiles >= (1ull << 31))
        return fail(QTB_ERR_UNSUPPORTED, "contract_sum: shape beyond the tensor-core grid");
    const float2 *pa = static_cast<const float2*>(A), *pb = static_cast<const float2*>(B);
    float2* pc = static_cast<float2*>(C);
    cudaError_t e = t.n == 128 ? tc_launch<128, kTest>(t, pa, pb, pc, K, F, M, N, scratch, st, spin_limit, stall)
                               : tc_launch<64, kTest>(t, pa, pb, pc, K, F, M, N, scratch, st, spin_limit, stall);
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? QTB_OK : cuda_fail_c(e, "contract_sum launch");
}

extern "C" {

int qtb_contract_sum_c64(const void* A, const void* B, void* C, int64_t K, int64_t F, int64_t M, int64_t N,
                         int32_t mode, void* scratch, size_t scratch_bytes, void* stream) {
    if (!A || !B || !C || K < 1 || F < 1 || M < 1 || N < 1 || mode < 0 || mode > 2)
        return fail(QTB_ERR_ARG, "contract_sum: bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    size_t need = 0;
    int r = qtb_contract_sum_scratch_bytes(K, F, M, N, mode, &need);
    if (r) return r;
    if (!scratch || scratch_bytes < need)
        return fail(QTB_ERR_ARG, "contract_sum: scratch smaller than qtb_contract_sum_scratch_bytes");
    int* status = static_cast<int*>(scratch);
    if (!use_tensor_cores(mode, K, M, N)) {
        const float2 *pa = static_cast<const float2*>(A), *pb = static_cast<const float2*>(B);
        float2* pc = static_cast<float2*>(C);
        const int rows = flat_rows((uint64_t)F * M * N, M, N);
        const bool pairs = rows > 1 && N % 2 == 0 && aligned16(B) && aligned16(C);   // every k's rows too
        const bool evict = flat_stream((uint64_t)F * M * N);
        const uint64_t as = (uint64_t)F * M, bs = (uint64_t)F * N;
        unsigned grid = 0;
        if (rows > 1) {
            const FlatShape<uint32_t> s = flat_shape<uint32_t>(F, M, N, rows, pairs ? 2 : 1, &grid);
            const auto run = !pairs  ? qtb_contract_simt_kernel<kFlatRows, false, false, 2, uint32_t>
                            : evict ? qtb_contract_simt_kernel<kFlatRows, true, true, 2, uint32_t>
                                    : qtb_contract_simt_kernel<kFlatRows, true, false, 2, uint32_t>;
            run<<<grid, kFlatThreads, 0, st>>>(pa, pb, pc, K, as, bs, status, s);
        } else {
            const FlatShape<uint64_t> s = flat_shape<uint64_t>(F, M, N, 1, 1, &grid);
            qtb_contract_simt_kernel<1, false, false, 8><<<grid, kFlatThreads, 0, st>>>(pa, pb, pc, K, as, bs, status, s);
        }
        const cudaError_t e = cudaGetLastError();
        return e == cudaSuccess ? QTB_OK : cuda_fail_c(e, "contract_sum launch");
    }
    return tc_sum<false>(tc_shape(K, F, M, N), A, B, C, K, F, M, N, scratch, st);
}

int qtb_selftest_contract_timeout(const void* A, const void* B, void* C, int64_t K, int64_t F, int64_t M, int64_t N,
                                  void* scratch, size_t scratch_bytes, int32_t spin_limit, int32_t part, void* stream) {
    if (!A || !B || !C || K < 1 || F < 1 || M < 1 || N < 1 || spin_limit < 1 || part < 0)
        return fail(QTB_ERR_ARG, "selftest_contract_timeout: bad arguments");
    size_t need = 0;
    int r = qtb_contract_sum_scratch_bytes(K, F, M, N, 2, &need);
    if (r) return r;
    if (!scratch || scratch_bytes < need)
        return fail(QTB_ERR_ARG, "selftest_contract_timeout: scratch smaller than qtb_contract_sum_scratch_bytes");
    const TcShape t = tc_shape(K, F, M, N);
    if ((uint32_t)part >= t.split)
        return fail(QTB_ERR_ARG, "selftest_contract_timeout: the shape's K is in " + std::to_string(t.split) + " parts");
    return tc_sum<true>(t, A, B, C, K, F, M, N, scratch, static_cast<cudaStream_t>(stream), (uint32_t)spin_limit,
                        (uint32_t)part);
}

}  // extern "C"
