// mm8_seq on the integer path of the 5th-generation tensor cores (tcgen05 kind::i8): the packed matrix is multiplied as
// the bytes it is stored as.
//
//   y[t,n] = rx[n] * sum_k x'[t,k] (w[k,n] - 128) + rx[n]*128.5*SXR[t] + mx[n]*SX[t] + SXMY[t]
//
// with x' = x*ry, SX = sum_k x, SXR = sum_k x', SXMY = sum_k x*my (per row t), the factorisation of mm8_one.
//   * x' becomes a 24-bit fixed-point integer per row (the scale is the power of two that takes the row's largest
//     magnitude into [2^22, 2^23), so the fp32 products are scaled exactly and rounded once, to 2^-23 .. 2^-22 of the
//     row's maximum) and enters as three planes of signed base-256 digits.  A row in which a few elements tower over the
//     rest (outlier channels) is WIDE: it gets 32 bits, the last 8 as a fourth plane, for which a token tile that holds
//     such a row takes its K range a second time;
//   * W enters as the raw uint8 rows: TMA brings 128-column x 128-row boxes into shared memory in the layout the
//     tensor core reads as a transposed (MN-major) operand, with no conversion and no thread touching a weight;
//   * all sums are exact 32-bit integers (128 * 255 * K < 2^31 up to K = 65536), the planes and the K splits are
//     combined in exact 64-bit integers and rounded to fp32 once: the product part does not depend on the tiling, on the
//     split, on the form of the kernel or on the other rows.  (SX, SXR and SXMY are fp32 sums of the operand pass, whose
//     order depends on the launch's rows and on N.)
// W's 128 columns are the M side of the MMA and the tokens of all three planes its N side, so a launch of 16 tokens
// multiplies 48 columns instead of padding 16 rows to 128.
//
// One persistent kernel: the tiles (matrix, column tile, token tile) are dealt in whole waves to the CTAs (or pairs of
// CTAs, cta_group::2, sharing the token planes); the K range of the tiles left over is split so that they occupy the
// whole GPU too.  A split tile is finished by the CTA that arrives last (tickets, no waiting), which adds the others'
// 64-bit partial sums.
//   warps 0-15 epilogue: tcgen05.ld of 32 TMEM lanes (warp % 4) x every fourth chunk of 8 tokens, affine tail and
//              rounding into a shared-memory tile (the accumulators are free again), then the fused epilogue and the
//              stores in 16-byte pieces of rows
//   warp 16    TMEM allocation; tcgen05.mma and tcgen05.commit
//   warp 17    TMA loads (W ahead of the dependency wait: it was written before the launch)
// Bound by HBM up to about 64 rows and by the int8 tensor rate above 200 (760 clocks per K block of a pair's 256 x 128
// tile, 768 of tensor work).  Operator alone, operand pass included, fp16 path -> this one, (4096, 4096) / (4096, 16384) /
// (16384, 4096): 16 rows 16.7 -> 12.8 / 38.9 -> 16.4 / 49.3 -> 23.4 us, 1024 rows 67 -> 48 / 248 -> 135 / 245 -> 176 us.
// Every wait is bounded: on give-up the CTA raises an error word, skips the rest of its work and returns.
#include "common.cuh"
#include "seq_epi.cuh"
#include <algorithm>
#include <cmath>
#include <cuda.h>
#include "mm8_seq_i8.h"

namespace {

constexpr int BMC = 128;                        // columns of W per CTA
constexpr int BKI = 128;                        // K block
constexpr int kWTile = BMC * BKI;               // 16 KB
constexpr int kMaxTT = 128;                     // tokens per tile
constexpr int kEpiThreads = 512;
constexpr int kEpiWarps = kEpiThreads / 32;
constexpr int kThreadsI8 = kEpiThreads + 64;
constexpr int kMaxStages = 12;
constexpr int kSmemBudget = 226 * 1024;
constexpr unsigned kWaitLimitI8 = 1u << 22;
constexpr float kTopDigits = 8355711.f;         // 127 * 65536 + 127 * 256 + 127

struct alignas(16) RowConst { float scale, sx, sxr, sxmy; long long corr; int wide, pad; };     // corr = -128 * sum of the integers

struct I8Problem {
    const __half* mx; const __half* rx;
    __half* y; long long y_stride;
    SeqEpi epi;
    int M, tile0;                               // tile0: index of this matrix's first tile
    int vec;                                    // y, aux, aux2 allow 16-byte accesses
};
struct alignas(64) I8Args {
    CUtensorMap wmap[kSeqI8MaxProblems];
    CUtensorMap xmap[2];                        // the token planes as rows of 128 bytes, in boxes of the rows of each MMA
    CUtensorMap lmap;                           // the fourth planes
    I8Problem p[kSeqI8MaxProblems];
    const RowConst* consts;                     // [problem][T]
    unsigned* tickets;                          // [split tile][CTA of the pair]
    long long* slots;                           // [part of a split tile][CTA of the pair][TT][128]
    unsigned* error_flag;
    int nprob, T, TT, ntt, nkb, N1, N2, stages;
    int units, whole, parts, split;             // unit u: tiles u, u + units, ... < whole, then part u (< parts) of the rest, `split` parts a tile
    int bufcols;                                // TMEM columns between accumulator buffers (0: one buffer)
    int tmem_cols;
};

__device__ __forceinline__ uint32_t su(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t b, uint32_t n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(uint32_t b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b) : "memory"); }
__device__ __forceinline__ void bar_arrive_cluster(uint32_t b) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(b) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
}
template <bool CLUSTER = false>                // CLUSTER: acquire what the other CTA of the pair released
__device__ __forceinline__ bool bar_wait(uint32_t b, uint32_t parity) {
    for (unsigned it = 0; it < kWaitLimitI8; ++it) {
        uint32_t done;
        if (CLUSTER)
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                         "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(b), "r"(parity) : "memory");
        else
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                         "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(b), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
// One lane of a converged warp.  The roles that issue MMAs and TMA loads run as whole warps and elect a lane for each
// issue: descriptors then stay in uniform registers (issued from a lane == 0 branch, a K block cost 950 clocks).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
template <bool CLUSTER = false>                // the same answer in all lanes of a converged warp
__device__ __forceinline__ bool warp_wait(uint32_t b, uint32_t parity) { return __all_sync(0xffffffffu, bar_wait<CLUSTER>(b, parity)); }
__device__ __forceinline__ uint32_t in_cta(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// PAIR == 2: `bar` may be the barrier of the pair's first CTA, which counts the bytes of both
template <int PAIR> __device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    if constexpr (PAIR == 2)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(dst), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(dst), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// the same with an L2 eviction policy
template <int PAIR> __device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar, uint64_t policy) {
    if constexpr (PAIR == 2)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
                     ::"r"(dst), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar), "l"(policy) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
                     ::"r"(dst), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar), "l"(policy) : "memory");
}
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// Shared-memory matrix descriptor, 128-byte swizzle.  Both operands are stored as rows of 128 bytes whose 16-byte
// chunks are permuted by (row % 8): for W a row is one k and its bytes are columns (MN-major), for the token planes a
// row is one token and its bytes are k (K-major); 8-row groups follow each other at 1024 bytes.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t smem_addr) {
    uint64_t d = (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)(1024 >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;                     // descriptor version of sm_100
    d |= (uint64_t)2 << 61;                     // 128-byte swizzle
    return d;
}
// kind::i8: s32 accumulator, A unsigned 8 bit stored MN-major (transposed), B signed 8 bit stored K-major
__device__ __forceinline__ uint32_t i8_idesc(int m, int n) {
    return (2u << 4) | (0u << 7) | (1u << 10) | (1u << 15) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
template <int PAIR>
__device__ __forceinline__ void umma_i8(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accumulate) {
    if constexpr (PAIR == 2)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d), "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d), "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate) : "memory");
}
template <int PAIR> __device__ __forceinline__ void commit_i8(uint32_t bar) {
    if constexpr (PAIR == 2) {                  // the same barrier in both CTAs
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     ::"r"(bar), "h"((uint16_t)3) : "memory");
    } else {
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
    }
}
// fp32 of an exact 64-bit sum.  Three digits (below 2^47 up to K = 65536): both parts are exact, rounded once.  Four digits
// (below 2^54): above 2^48 the upper part is rounded to 24 bits before, which makes it one unit in the last place.
__device__ __forceinline__ float sum_to_f32(long long s) {
    return fmaf((float)(int)(s >> 24), 16777216.f, (float)((int)s & 0xffffff));
}
// the fused epilogue on eight neighbouring columns (v already rounded to fp16: seq_epilogue_with starts from that)
__device__ __forceinline__ void epi8(int mode, float scale, const __half (&v)[8], const __half (&x1)[8], const __half (&x2)[8], __half (&o)[8]) {
    if (mode == RWKV_EPI_STORE) {
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = v[e];
    } else if (mode == RWKV_EPI_MUL_RESIDUAL || mode == RWKV_EPI_RESIDUAL) {
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = seq_epilogue_with<__half>(mode, scale, __half2float(v[e]), __half2float(x1[e]), __half2float(x2[e]));
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = seq_epilogue_with<__half>(mode, scale, __half2float(v[e]), 0.f, 0.f);
    }
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory"); }
__device__ __forceinline__ bool epi_sync_or(bool v) {                    // the same, with the OR of `v` over its threads
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((uint32_t)v), "n"(kEpiThreads) : "memory");
    return r != 0;
}
__device__ __forceinline__ void tmem_ld8(int (&v)[8], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr) : "memory");
}

// ---- preparation: x' as digit planes, the row sums and scales ------------------------------------
// One block per row (or per row and matrix); a thread owns E neighbouring k.  What produces the row (LayerNorm + token
// shift, the one-step WKV, group norm + gate) runs in the same pass.  A block is a chain of latencies: one trip to memory,
// two to four reductions, and vectors and code that the streamed weights have evicted.  Few rows run with the weights'
// vectors fetched before the dependency wait and E = 8 (16 rows of 4096, LayerNorm + mix, from the wait to the end, in a 7B
// layer: 10 us with E = 16, 9 us with E = 4 whose 32 warps wait for each other in every reduction, 6.5 us with E = 8).
// With many rows what counts is how many blocks an SM holds: E = 16, rows kept as fp16, the vectors read when needed.
template <int E> struct HV {                     // E fp16 values
    __half2 h[E / 2];
    __device__ __forceinline__ float operator[](int e) const { return (e & 1) ? __high2float(h[e >> 1]) : __low2float(h[e >> 1]); }
    __device__ __forceinline__ void set(int e, float v) {
        const __half x = __float2half_rn(v);
        h[e >> 1] = (e & 1) ? __halves2half2(__low2half(h[e >> 1]), x) : __halves2half2(x, __high2half(h[e >> 1]));
    }
};
template <int BYTES> struct VecOf { typedef uint4 T; };
template <> struct VecOf<8> { typedef uint2 T; };
template <> struct VecOf<4> { typedef uint32_t T; };
template <int E> __device__ __forceinline__ HV<E> zero_hv() {
    HV<E> o;
#pragma unroll
    for (int i = 0; i < E / 2; ++i) o.h[i] = __float2half2_rn(0.f);
    return o;
}
template <int E, bool CONSTANT = false>          // CONSTANT: never written while kernels run (weights)
__device__ __forceinline__ HV<E> load_hv(const void* ptr, long long k0, int N, bool vec) {
    const __half* p = static_cast<const __half*>(ptr);
    HV<E> o = zero_hv<E>();
    if (vec && k0 + E <= N) {
        typedef typename VecOf<E * 2>::T V;
        const V* q = reinterpret_cast<const V*>(p + k0);
        V v[E * 2 / sizeof(V)];
#pragma unroll
        for (int i = 0; i < int(E * 2 / sizeof(V)); ++i) v[i] = CONSTANT ? __ldg(q + i) : q[i];
        memcpy(&o, v, sizeof(o));
    } else {
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (k0 + e < N) o.set(e, __half2float(p[k0 + e]));
    }
    return o;
}
template <int E> __device__ __forceinline__ void store_hv(void* ptr, int k0, int N, bool vec, const HV<E>& v) {
    __half* p = static_cast<__half*>(ptr);
    if (vec && k0 + E <= N) {
        typedef typename VecOf<E * 2>::T V;
        V o[E * 2 / sizeof(V)];
        memcpy(o, &v, sizeof(o));
#pragma unroll
        for (int i = 0; i < int(E * 2 / sizeof(V)); ++i) reinterpret_cast<V*>(p + k0)[i] = o[i];
    } else {
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (k0 + e < N) p[k0 + e] = __float2half_rn(v[e]);
    }
}
template <int E> __device__ __forceinline__ void load_f(const float* __restrict__ p, int k0, int N, bool vec, float (&out)[E]) {
    if (vec && k0 + E <= N) {
#pragma unroll
        for (int i = 0; i < E / 4; ++i) {
            const float4 v = reinterpret_cast<const float4*>(p + k0)[i];
            out[4 * i] = v.x; out[4 * i + 1] = v.y; out[4 * i + 2] = v.z; out[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < E; ++e) out[e] = (k0 + e < N) ? p[k0 + e] : 0.f;
    }
}
template <int E> __device__ __forceinline__ void store_f(float* p, int k0, int N, bool vec, const float (&v)[E]) {
    if (vec && k0 + E <= N) {
#pragma unroll
        for (int i = 0; i < E / 4; ++i) reinterpret_cast<float4*>(p + k0)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (k0 + e < N) p[k0 + e] = v[e];
    }
}
struct PrepProblem {
    rwkv_mm8_seq_prologue pro;                   // what makes the rows of x (RWKV_PRO_*)
    const void* x; long long x_stride;
    const __half* ry; const __half* my;
};
struct PrepArgs {
    PrepProblem p[kSeqI8MaxProblems];
    int nprob, T, N, nkb, TT, ntt, ntickets, vec;          // vec: every vector and row starts on a 16-byte boundary
    float narrow;                                // a row whose squared norm, in integer units of three digits, is below this is wide
    uint8_t* images; uint8_t* low; RowConst* consts; unsigned* tickets;
};
// Sums of NV values per thread over the block; every thread gets the results.
template <int NV>
__device__ __forceinline__ void block_reduce(float (&v)[NV], float (*sh)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = warp_sum(v[i]);
    __syncthreads();                                       // the previous use of sh is over
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) sh[i][warp] = v[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = warp_sum(lane < nwarp ? sh[i][lane] : 0.f);
}
// The row's maximum (of magnitudes: their bits order like integers) and four sums over the block, for every thread.  The sums
// run the butterfly of warp_sum with half of the values dropped at each step while there are several: the same pairs in the
// same order in 6 shuffles instead of 20, and again over the warps' parts.
__device__ __forceinline__ void row_reduce(float (&v)[5], float (*sh)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const bool b4 = (lane & 16) != 0, b3 = (lane & 8) != 0;
    auto fold = [&](float s0, float s1, float s2, float s3) {         // lanes 8 i .. 8 i + 7 get sum i
        float x = (b4 ? s2 : s0) + __shfl_xor_sync(0xffffffffu, b4 ? s0 : s2, 16);
        const float y = (b4 ? s3 : s1) + __shfl_xor_sync(0xffffffffu, b4 ? s1 : s3, 16);
        x = (b3 ? y : x) + __shfl_xor_sync(0xffffffffu, b3 ? x : y, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    };
    const float m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v[0])));
    const float s = fold(v[1], v[2], v[3], v[4]);
    __syncthreads();                                       // the previous use of sh is over
    if (lane == 0) sh[0][warp] = m;
    if ((lane & 7) == 0) sh[1 + (lane >> 3)][warp] = s;
    __syncthreads();
    const bool part = lane < nwarp;
    v[0] = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(part ? sh[0][lane] : 0.f)));
    const float t = fold(part ? sh[1][lane] : 0.f, part ? sh[2][lane] : 0.f, part ? sh[3][lane] : 0.f, part ? sh[4][lane] : 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[1 + i] = __shfl_sync(0xffffffffu, t, 8 * i);
}

// PRO: where the rows of x come from (RWKV_PRO_*).  LOOP (RWKV_PRO_PLAIN only): a thread owns every blockDim-th E k and
// reads the row twice (the second time from L1); else one chunk per thread.  PRE: the vectors of the first matrix and of
// the prologue are fetched ahead of the dependency wait.
template <int PRO, int E, bool LOOP, bool PRE, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) mm8_seq_i8_prep(const __grid_constant__ PrepArgs a) {
    asm volatile("griddepcontrol.launch_dependents;");
    const int t = blockIdx.x, tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarp = nthr >> 5;
    __shared__ float sh[5][32];
    __shared__ long long shq[32];
    const bool vec = a.vec != 0;
    const int N = a.N, k0 = tid * E;
    const int nchunk = a.nkb * (BKI / E);
    const bool mine = tid < nchunk;
    HV<E> ry = zero_hv<E>(), my = zero_hv<E>(), mix = zero_hv<E>(), lw = zero_hv<E>(), lb = zero_hv<E>();
    if (PRE && mine) {
        const PrepProblem& p = a.p[blockIdx.y];
        ry = load_hv<E, true>(p.ry, k0, N, vec);
        my = load_hv<E, true>(p.my, k0, N, vec);
        if constexpr (PRO == RWKV_PRO_LN_MIX) {
            if (p.pro.mode != 2) mix = load_hv<E, true>(p.pro.mix, k0, N, vec);
            lw = load_hv<E, true>(a.p[0].pro.ln_w, k0, N, vec);
            lb = load_hv<E, true>(a.p[0].pro.ln_b, k0, N, vec);
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (t == 0 && blockIdx.y == 0)
        for (int i = tid; i < a.ntickets; i += nthr) a.tickets[i] = 0;

    // ---- the row, common to all matrices of the launch
    HV<E> xx = zero_hv<E>(), prev = zero_hv<E>();
    if constexpr (PRO == RWKV_PRO_LN_MIX) {
        // LayerNorm + token shift, rounding as rwkv_ln_mix; the previous row's output is the state or computed again
        const rwkv_mm8_seq_prologue& q = a.p[0].pro;
        const bool shift = q.sx != nullptr, own = !shift || t == 0 || q.sx_stride != 0;
        const __half* x = static_cast<const __half*>(a.p[0].x) + (long long)t * a.p[0].x_stride;
        xx = load_hv<E>(x, k0, N, vec);
        if (shift) prev = own ? load_hv<E>(static_cast<const __half*>(q.sx) + (long long)t * q.sx_stride, k0, N, vec)
                              : load_hv<E>(x - a.p[0].x_stride, k0, N, vec);
        if (!PRE) {
            lw = load_hv<E, true>(q.ln_w, k0, N, vec);
            lb = load_hv<E, true>(q.ln_b, k0, N, vec);
        }
        float m[2] = {0.f, 0.f}, d[2] = {0.f, 0.f};
#pragma unroll
        for (int e = 0; e < E; ++e) { m[0] += xx[e]; m[1] += prev[e]; }
        block_reduce<2>(m, sh);
        m[0] /= float(N); m[1] /= float(N);
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (k0 + e < N) {
                d[0] = fmaf(xx[e] - m[0], xx[e] - m[0], d[0]);
                d[1] = fmaf(prev[e] - m[1], prev[e] - m[1], d[1]);
            }
        block_reduce<2>(d, sh);
        const float r0 = rsqrtf(d[0] / float(N) + 1e-5f), r1 = rsqrtf(d[1] / float(N) + 1e-5f);
#pragma unroll
        for (int e = 0; e < E; e += 2) {
            xx.h[e >> 1] = __floats2half2_rn((xx[e] - m[0]) * r0 * lw[e] + lb[e], (xx[e + 1] - m[0]) * r0 * lw[e + 1] + lb[e + 1]);
            if (!own) prev.h[e >> 1] = __floats2half2_rn((prev[e] - m[1]) * r1 * lw[e] + lb[e], (prev[e + 1] - m[1]) * r1 * lw[e + 1] + lb[e + 1]);
        }
        if (blockIdx.y == 0) {
            if (q.xx_out) store_hv<E>(static_cast<__half*>(q.xx_out) + (long long)t * q.xx_stride, k0, N, vec, xx);
            if (t == a.T - 1 && q.new_state) store_hv<E>(q.new_state, k0, N, vec, xx);
        }
    } else if constexpr (PRO == RWKV_PRO_WKV4) {
        // one step of the RWKV-4 recurrence per row, r * wkv with the roundings of rwkv_wkv4_seq; state in place
        const rwkv_mm8_seq_prologue& q = a.p[0].pro;
        const long long at = (long long)t * N;
        const HV<E> kk = load_hv<E>(static_cast<const __half*>(q.k) + at, k0, N, vec), vv = load_hv<E>(static_cast<const __half*>(q.v) + at, k0, N, vec);
        const HV<E> rr = load_hv<E>(static_cast<const __half*>(a.p[0].x) + (long long)t * a.p[0].x_stride, k0, N, vec);
        float w[E], u[E], aa[E], bb[E], pp[E];
        load_f<E>(q.aa + at, k0, N, vec, aa);
        load_f<E>(q.bb + at, k0, N, vec, bb);
        load_f<E>(q.pp + at, k0, N, vec, pp);
        load_f<E>(q.t_decay, k0, N, vec, w);
        load_f<E>(q.t_first, k0, N, vec, u);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            float ww = u[e] + kk[e];
            float p = fmaxf(pp[e], ww);
            float e1 = expf(pp[e] - p), e2 = expf(ww - p);
            const float y = (e1 * aa[e] + e2 * vv[e]) / (e1 * bb[e] + e2);
            xx.set(e, k0 + e < N ? rr[e] * r16(y) : 0.f);
            ww = w[e] + pp[e];
            p = fmaxf(ww, kk[e]);
            e1 = expf(ww - p); e2 = expf(kk[e] - p);
            aa[e] = e1 * aa[e] + e2 * vv[e];
            bb[e] = e1 * bb[e] + e2;
            pp[e] = p;
        }
        store_f<E>(q.aa + at, k0, N, vec, aa);
        store_f<E>(q.bb + at, k0, N, vec, bb);
        store_f<E>(q.pp + at, k0, N, vec, pp);
    } else if constexpr (PRO == RWKV_PRO_GN_GATE) {
        // group norm of each head (biased variance), ln_x in fp32, one rounding, times the gate: rwkv_v56_seq_gn_gate
        const rwkv_mm8_seq_prologue& q = a.p[0].pro;
        float y[E], gw[E], gb[E];
        load_f<E>(static_cast<const float*>(a.p[0].x) + (long long)t * a.p[0].x_stride, k0, N, vec, y);
        const HV<E> g = load_hv<E>(static_cast<const __half*>(q.gate) + (long long)t * q.gate_stride, k0, N, vec);
        load_f<E>(static_cast<const float*>(q.ln_w), k0, N, vec, gw);
        load_f<E>(static_cast<const float*>(q.ln_b), k0, N, vec, gb);
        const int per = q.head / E;                       // threads of a head: 1 to 32 neighbouring lanes (128 channels, E = 4)
        float s = 0.f, v = 0.f;
#pragma unroll
        for (int e = 0; e < E; ++e) s += y[e];
        for (int o = per >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float mean = s / float(q.head);
#pragma unroll
        for (int e = 0; e < E; ++e) v = fmaf(y[e] - mean, y[e] - mean, v);
        for (int o = per >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const float rstd = rsqrtf(v / float(q.head) + q.eps);
#pragma unroll
        for (int e = 0; e < E; ++e) xx.set(e, k0 + e < N ? r16((y[e] - mean) * rstd * gw[e] + gb[e]) * g[e] : 0.f);
    }

    // ---- digits, scale and sums for each matrix
    const int tt = t / a.TT, ti = t - tt * a.TT;
    const size_t plane = (size_t)a.TT * BKI;               // TT % 8 == 0: the three planes' rows share row % 8
    for (int prob = blockIdx.y; prob < a.nprob; prob += gridDim.y) {
        const PrepProblem& p = a.p[prob];
        const bool have = PRE && prob == (int)blockIdx.y;  // the vectors are in registers
        const __half* xrow = static_cast<const __half*>(p.x) + (long long)t * p.x_stride;      // RWKV_PRO_PLAIN
        HV<E> xv = zero_hv<E>();
        float red[5] = {0.f, 0.f, 0.f, 0.f, 0.f};          // maximum, SX, SXR, SXMY, sum of squares of x'
        auto first = [&](int c) {
            const int kc = c * E;
            if constexpr (PRO == RWKV_PRO_PLAIN) {
                xv = load_hv<E>(xrow, kc, N, vec);
            } else if constexpr (PRO == RWKV_PRO_LN_MIX) {
                if (!have && p.pro.mode != 2) mix = load_hv<E, true>(p.pro.mix, kc, N, vec);
                // every fp16 operation of the reference rounds once, as these do (_rn: never contracted)
                const __half2 one = __float2half2_rn(1.f);
#pragma unroll
                for (int i = 0; i < E / 2; ++i)
                    xv.h[i] = p.pro.mode == 2 ? xx.h[i]
                              : p.pro.mode == 0 ? __hadd2_rn(__hmul2_rn(xx.h[i], mix.h[i]), __hmul2_rn(prev.h[i], __hsub2_rn(one, mix.h[i])))
                                                : __hadd2_rn(xx.h[i], __hmul2_rn(__hsub2_rn(prev.h[i], xx.h[i]), mix.h[i]));
            } else {
                xv = xx;
            }
            if (!have) {
                ry = load_hv<E, true>(p.ry, kc, N, vec);
                my = load_hv<E, true>(p.my, kc, N, vec);
            }
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const float xe = xv[e], xp = xe * ry[e];
                red[1] += xe;
                red[2] += xp;
                red[3] = fmaf(xe, my[e], red[3]);
                red[4] = fmaf(xp, xp, red[4]);
                red[0] = fabsf(xp) <= 3.0e38f ? fmaxf(red[0], fabsf(xp)) : INFINITY;      // fmaxf would drop a NaN
            }
        };
        if constexpr (!LOOP) { if (mine) first(tid); }
        else for (int c = tid; c < nchunk; c += nthr) first(c);
        row_reduce(red, sh);
        // the power of two `up` that takes the maximum into [2^22, 2^23), or half of it if three digits would not hold it
        float up = 0.f, down = 0.f;
        bool wide = false;
        if (red[0] > 0.f && red[0] <= 3.0e38f) {
            int e = 22 - ilogbf(red[0]);
            if (ldexpf(red[0], e) > kTopDigits) --e;
            up = ldexpf(1.f, e);                            // |x'| >= 2^-48 or 0: e <= 70
            wide = red[4] * up * up < a.narrow;             // (see wide_norm)
            down = ldexpf(1.f, wide ? -e - 8 : -e);
        } else if (red[0] > 0.f) {
            down = NAN;                                     // a NaN or an infinity among the activations: the row is NaN
        }
        uint8_t* img = a.images + ((size_t)prob * a.ntt + tt) * a.nkb * (size_t)(3 * a.TT * BKI) + (size_t)ti * BKI;
        // balanced base-256 digits of four neighbouring k: the bytes of q + 128 * (1 + 256 + 65536), each minus 128
        auto digits = [&](const int (&q)[4], uint32_t& d0, uint32_t& d1, uint32_t& d2) {
            uint32_t u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) u[i] = (uint32_t)(q[i] + 0x808080);
            const uint32_t lo01 = __byte_perm(u[0], u[1], 0x5140), lo23 = __byte_perm(u[2], u[3], 0x5140);
            const uint32_t hi01 = __byte_perm(u[0], u[1], 0x0062), hi23 = __byte_perm(u[2], u[3], 0x0062);
            d0 = __byte_perm(lo01, lo23, 0x5410) ^ 0x80808080u;
            d1 = __byte_perm(lo01, lo23, 0x7632) ^ 0x80808080u;
            d2 = __byte_perm(hi01, hi23, 0x5410) ^ 0x80808080u;
        };
        auto in_row = [&](int kc) { return (size_t)((((kc >> 4) & 7) ^ (ti & 7)) << 4) + (kc & 15); };
        auto second = [&](int c, int& isum) {
            uint32_t d[3][E / 4];
#pragma unroll
            for (int e = 0; e < E; e += 4) {
                int q[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    q[i] = up > 0.f ? __float2int_rn(xv[e + i] * ry[e + i] * up) : 0;
                    isum += q[i];
                }
                digits(q, d[0][e >> 2], d[1][e >> 2], d[2][e >> 2]);
            }
            const int kc = c * E;
            uint8_t* dst = img + (size_t)(kc >> 7) * (3 * plane) + in_row(kc);
            typedef typename VecOf<E>::T V;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                V o;
                memcpy(&o, d[i], sizeof(o));
                *reinterpret_cast<V*>(dst + i * plane) = o;
            }
        };
        // a wide row: 32 bits, the first 24 as above and the last digit to the fourth plane (rare: kept small, four k at a time)
        auto second_wide = [&](int c) -> long long {
            const int kc = c * E;
            uint8_t* dst = img + (size_t)(kc >> 7) * (3 * plane) + in_row(kc);
            uint8_t* low = a.low + (((size_t)prob * a.ntt + tt) * a.nkb + (kc >> 7)) * plane + (size_t)ti * BKI + in_row(kc);
            const float up4 = up * 256.f;
            int isum = 0, lsum = 0;
#pragma unroll
            for (int e = 0; e < E; e += 4) {
                int q[4], l[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    q[i] = __float2int_rn(xv[e + i] * ry[e + i] * up4);
                    l[i] = (int8_t)q[i];
                    q[i] = (q[i] + 128) >> 8;               // (q - l) / 256
                    isum += q[i];
                    lsum += l[i];
                }
                uint32_t d[3];
                digits(q, d[0], d[1], d[2]);
#pragma unroll
                for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(dst + i * plane + e) = d[i];
                *reinterpret_cast<uint32_t*>(low + e) = __byte_perm(__byte_perm(l[0], l[1], 0x0040), __byte_perm(l[2], l[3], 0x0040), 0x5410);
            }
            return 256ll * isum + lsum;
        };
        long long qsum = 0;
        if (__builtin_expect(wide, 0)) {
            if constexpr (!LOOP) { if (mine) qsum = second_wide(tid); }
            else for (int c = tid; c < nchunk; c += nthr) {
                xv = load_hv<E>(xrow, c * E, N, vec);
                ry = load_hv<E, true>(p.ry, c * E, N, vec);
                qsum += second_wide(c);
            }
        } else if constexpr (!LOOP) {
            int isum = 0;
            if (mine) second(tid, isum);
            qsum = isum;
        } else {
            for (int c = tid; c < nchunk; c += nthr) {
                xv = load_hv<E>(xrow, c * E, N, vec);
                ry = load_hv<E, true>(p.ry, c * E, N, vec);
                int isum = 0;
                second(c, isum);
                qsum += isum;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) qsum += __shfl_xor_sync(0xffffffffu, qsum, o);
        __syncthreads();
        if (lane == 0) shq[warp] = qsum;
        __syncthreads();
        if (warp == 0) {
            qsum = lane < nwarp ? shq[lane] : 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) qsum += __shfl_xor_sync(0xffffffffu, qsum, o);
            if (lane == 0) {
                RowConst rc;
                rc.scale = down; rc.sx = red[1]; rc.sxmy = red[3]; rc.corr = -128 * qsum; rc.wide = wide ? 1 : 0; rc.pad = 0;
                rc.sxr = wide ? __ll2float_rn(qsum) * down : red[2];       // wide: the exact sum of the integers
                a.consts[(size_t)prob * a.T + t] = rc;
            }
        }
    }
}

// ---- the matmul ------------------------------------------------------------------------------------
struct Item { int prob, n0, tt, kb0, kb1, part; };        // part < 0: the whole K range
// The i-th piece of work of `unit`; false when there is none.
template <int PAIR> __device__ __forceinline__ bool item_of(const I8Args& a, int unit, int i, Item& t) {
    int tile = unit + i * a.units;
    t.kb0 = 0; t.kb1 = a.nkb; t.part = -1;
    if (tile >= a.whole) {
        if (unit >= a.parts || tile >= a.whole + a.units) return false;
        const int r = unit / a.split, k = unit - r * a.split;
        tile = a.whole + r;
        if (a.split > 1) {
            t.part = unit;
            t.kb0 = a.nkb * k / a.split;
            t.kb1 = a.nkb * (k + 1) / a.split;
        }
    }
    t.prob = 0;
#pragma unroll
    for (int q = 1; q < kSeqI8MaxProblems; ++q) t.prob += (q < a.nprob && tile >= a.p[q].tile0) ? 1 : 0;
    const int r = tile - a.p[t.prob].tile0, ct = r / a.ntt;
    t.tt = r - ct * a.ntt;
    t.n0 = ct * (BMC * PAIR);
    return true;
}

// Whether a token tile holds a wide row, in two steps so that the loads (of one warp) run beside other work.  The same
// answer in every role and in both CTAs of a pair.
struct WideFlags { int v[kMaxTT / 32]; };
__device__ __forceinline__ WideFlags wide_flags(const I8Args& a, const Item& tl, int lane) {
    WideFlags f;
    const int t0 = tl.tt * a.TT, n = min(a.TT, a.T - t0);
    const RowConst* rc = a.consts + (size_t)tl.prob * a.T + t0;
#pragma unroll
    for (int i = 0; i < kMaxTT / 32; ++i) f.v[i] = lane + 32 * i < n ? __ldcg(&rc[lane + 32 * i].wide) : 0;
    return f;
}
__device__ __forceinline__ bool any_wide(const WideFlags& f) {
    int v = 0;
#pragma unroll
    for (int i = 0; i < kMaxTT / 32; ++i) v |= f.v[i];
    return __any_sync(0xffffffffu, v != 0);
}

template <int PAIR>
__global__ void __launch_bounds__(kThreadsI8, 1) mm8_seq_i8_kernel(const __grid_constant__ I8Args a) {
    asm volatile("griddepcontrol.launch_dependents;");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024 - (su(smem_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t crank = PAIR == 2 ? (blockIdx.x & 1) : 0;
    const int unit = blockIdx.x / PAIR;
    const int S = a.stages;
    const int n1 = a.N1 / PAIR, n2 = a.N2 / PAIR;                 // token rows of each MMA that this CTA holds
    const uint32_t xbytes = (uint32_t)(n1 + n2) * BKI, stage_bytes = kWTile + xbytes;
    const int n3 = a.TT / PAIR;                                   // of the fourth plane
    uint8_t* bars = smem + (size_t)S * stage_bytes;
    const uint32_t full0 = su(bars), empty0 = full0 + kMaxStages * 8;
    const uint32_t acc_full0 = empty0 + kMaxStages * 8, acc_empty0 = acc_full0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages * 8 + 32);
    volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* last_flag = reinterpret_cast<int*>(tmem_slot + 2);
    RowConst* rowc = reinterpret_cast<RowConst*>(bars + 512);     // [2][TT]
    __half* tile = reinterpret_cast<__half*>(rowc + 2 * a.TT);    // [TT][128]: results before the fused epilogue

    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            bar_init(full0 + s * 8, 1);
            bar_init(empty0 + s * 8, 1);
        }
        for (int i = 0; i < 2; ++i) { bar_init(acc_full0 + i * 8, 1); bar_init(acc_empty0 + i * 8, kEpiWarps * PAIR); }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kEpiWarps) {
        if constexpr (PAIR == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su(tmem_slot)), "r"(a.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su(tmem_slot)), "r"(a.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if constexpr (PAIR == 2) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp < kEpiWarps) {
        // ================= epilogue =================
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int quarter = warp & 3, c_first = (warp >> 2) * 8;     // tokens c_first .. + 7, then 32 further on
        bool ok = true;
        Item tl;
        for (int seg = 0; item_of<PAIR>(a, unit, seg, tl); ++seg) {
            const I8Problem& p = a.p[tl.prob];
            const bool whole = tl.part < 0;
            const int buf = a.bufcols ? (seg & 1) : 0;
            const uint32_t par = a.bufcols ? ((seg >> 1) & 1) : (seg & 1);
            const int t0 = tl.tt * a.TT, n = tl.n0 + (int)crank * BMC + quarter * 32 + lane;
            const int nlive = min(a.TT, a.T - t0);                    // tokens of this tile that exist
            RowConst* rc = rowc + (seg & 1) * a.TT;
            // row constants of this tile (its K loop is running meanwhile)
            bool wide = false;                                        // of any row of this tile
            for (int i = tid; i < a.TT; i += kEpiThreads)
                if (t0 + i < a.T) {
                    const RowConst r = a.consts[(size_t)tl.prob * a.T + t0 + i];
                    rc[i] = r;
                    wide |= r.wide != 0;
                }
            const bool col = n < p.M;
            const float rxn = col ? __half2float(p.rx[n]) : 0.f, mxn = col ? __half2float(p.mx[n]) : 0.f;
            const float rx128 = rxn * 128.5f;
            wide = epi_sync_or(wide);                                 // (and the previous tile's stores have left `tile`)
            if (ok) ok = bar_wait(acc_full0 + buf * 8, par);
            if (!ok) *failed = 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tcol = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * a.bufcols);
            long long* slot = whole ? nullptr : a.slots + (((size_t)tl.part * PAIR + crank) * a.TT) * BMC + quarter * 32 + lane;
            __half* trow = tile + quarter * 32 + lane;
            auto put = [&](int ti, long long s) {
                const RowConst& r = rc[ti];
                const float val = fmaf(rxn, sum_to_f32(s + r.corr) * r.scale, fmaf(rx128, r.sxr, fmaf(mxn, r.sx, r.sxmy)));
                trow[ti * BMC] = __float2half_rn(val);
            };
            int q[2][3][8];                                           // the next chunk's loads run under this chunk's arithmetic
            auto fetch = [&](int (&d)[3][8], int c) {
#pragma unroll
                for (int i = 0; i < 3; ++i) tmem_ld8(d[i], tcol + i * a.TT + c);
            };
            auto emit = [&](int ti, long long s) {
                if (whole) put(ti, s);
                else if (ti < nlive) slot[(size_t)ti * BMC] = s;
            };
            auto finish = [&](const int (&d)[3][8], int c) {
#pragma unroll
                for (int e = 0; e < 8; ++e) emit(c + e, (long long)d[2][e] * 65536 + (long long)d[1][e] * 256 + d[0][e]);
            };
            if (__builtin_expect(!wide, 1)) {
                if (c_first < nlive) fetch(q[0], c_first);
#pragma unroll
                for (int k = 0; k < kMaxTT / 32; ++k) {
                    const int c = c_first + 32 * k;
                    if (c >= nlive) break;
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (c + 32 < nlive) fetch(q[(k + 1) & 1], c + 32);
                    finish(q[k & 1], c);
                }
            } else {
#pragma unroll 1
                for (int c = c_first; c < nlive; c += 32) {
                    fetch(q[0], c);
                    tmem_ld8(q[1][0], tcol + 3 * a.TT + c);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const long long s = (long long)q[0][2][e] * 65536 + (long long)q[0][1][e] * 256 + q[0][0][e];
                        emit(c + e, rc[c + e].wide ? s * 256 + q[1][0][e] : s);
                    }
                }
            }
            // the accumulators are read: the next tile's MMAs may overwrite them
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (PAIR == 2) bar_arrive_cluster(in_cta(acc_empty0 + buf * 8, 0));
                else bar_arrive(acc_empty0 + buf * 8);
            }
            if (!whole) {
                const int r = tl.part / a.split;                       // split tile
                __threadfence();
                epi_sync();
                if (tid == 0) *last_flag = ok && atomicAdd(a.tickets + (size_t)r * PAIR + crank, 1u) == (unsigned)(a.split - 1);
                epi_sync();
                if (*last_flag == 0) continue;
                __threadfence();
                // two neighbouring columns per thread and step, 16 loads in flight
                const size_t part_stride = (size_t)PAIR * a.TT * BMC / 2;
                const longlong2* first = reinterpret_cast<const longlong2*>(a.slots + ((size_t)r * a.split * PAIR + crank) * a.TT * BMC);
                const int n2c = tl.n0 + (int)crank * BMC + (tid & 63) * 2, end = min(a.TT, a.T - t0) * (BMC / 2);
                const bool c0 = n2c < p.M, c1 = n2c + 1 < p.M;
                const float rx0 = c0 ? __half2float(p.rx[n2c]) : 0.f, mx0 = c0 ? __half2float(p.mx[n2c]) : 0.f;
                const float rx1 = c1 ? __half2float(p.rx[n2c + 1]) : 0.f, mx1 = c1 ? __half2float(p.mx[n2c + 1]) : 0.f;
                for (int i = tid; i < end; i += 4 * kEpiThreads) {
                    longlong2 s[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) { const long long cr = rc[min(i + q * kEpiThreads, end - 1) >> 6].corr; s[q] = make_longlong2(cr, cr); }
#pragma unroll 4
                    for (int u = 0; u < a.split; ++u) {
                        longlong2 l[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            l[q] = i + q * kEpiThreads < end ? __ldcg(first + u * part_stride + i + q * kEpiThreads) : make_longlong2(0, 0);
#pragma unroll
                        for (int q = 0; q < 4; ++q) { s[q].x += l[q].x; s[q].y += l[q].y; }
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int j = i + q * kEpiThreads;
                        if (j >= end) break;
                        const RowConst& k = rc[j >> 6];
                        const float v0 = fmaf(rx0, sum_to_f32(s[q].x) * k.scale, fmaf(rx0 * 128.5f, k.sxr, fmaf(mx0, k.sx, k.sxmy)));
                        const float v1 = fmaf(rx1, sum_to_f32(s[q].y) * k.scale, fmaf(rx1 * 128.5f, k.sxr, fmaf(mx1, k.sx, k.sxmy)));
                        reinterpret_cast<__half2*>(tile)[j] = __halves2half2(__float2half_rn(v0), __float2half_rn(v1));
                    }
                }
            }
            epi_sync();                                               // the tile of results is complete
            if (!ok) continue;
            const int mode = p.epi.mode, M = p.M, nb = tl.n0 + (int)crank * BMC, tlive = min(a.TT, a.T - t0);
            const float scale = p.epi.out_scale;
            const bool has1 = mode == RWKV_EPI_RESIDUAL || mode == RWKV_EPI_MUL_RESIDUAL, has2 = mode == RWKV_EPI_MUL_RESIDUAL;
            __half* y = p.y + (long long)t0 * p.y_stride;
            const __half* x1p = static_cast<const __half*>(p.epi.aux) + (has1 ? (long long)t0 * p.epi.aux_stride : 0);
            const __half* x2p = static_cast<const __half*>(p.epi.aux2) + (has2 ? (long long)t0 * p.epi.aux2_stride : 0);
            const long long ys = p.y_stride, s1 = p.epi.aux_stride, s2 = p.epi.aux2_stride;
            const bool vec = p.vec != 0;
#pragma unroll 2
            for (int i = tid; i < tlive * (BMC / 8); i += kEpiThreads) {
                const int t = i >> 4, nn = nb + (i & 15) * 8, live = M - nn;
                if (live <= 0) continue;
                __half v[8], x1[8] = {}, x2[8] = {}, o[8];
                *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(tile + t * BMC + (i & 15) * 8);
                if (vec && live >= 8) {
                    if (has1) *reinterpret_cast<uint4*>(x1) = *reinterpret_cast<const uint4*>(x1p + t * s1 + nn);
                    if (has2) *reinterpret_cast<uint4*>(x2) = *reinterpret_cast<const uint4*>(x2p + t * s2 + nn);
                    epi8(mode, scale, v, x1, x2, o);
                    *reinterpret_cast<uint4*>(y + t * ys + nn) = *reinterpret_cast<const uint4*>(o);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (e < live) {
                            if (has1) x1[e] = x1p[t * s1 + nn + e];
                            if (has2) x2[e] = x2p[t * s2 + nn + e];
                        }
                    epi8(mode, scale, v, x1, x2, o);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (e < live) y[t * ys + nn + e] = o[e];
                }
            }
        }
    } else if (warp == kEpiWarps + 1) {
        // ================= TMA loads =================
        {
            bool ok = true;
            int s = 0;
            uint32_t ph = 1;                                           // the stages start empty
            const uint32_t smem0 = su(smem);
            const int xrows = 3 * a.TT;                                // rows of one K block of the token planes
            // With one token tile every byte of W is read once: it leaves L2 first, so that the activations, the norms' and
            // scale vectors and the code of the next layers are still there (a 7B layer streams 1.6 times the L2).
            const bool once = a.ntt == 1;
            const uint64_t policy = evict_first_policy();
            auto full_of = [&](int st) { return PAIR == 2 ? in_cta(full0 + st * 8, 0) : full0 + st * 8; };
            Item tl;
            for (int seg = 0; ok && item_of<PAIR>(a, unit, seg, tl); ++seg) {
                const CUtensorMap* map = &a.wmap[tl.prob];
                const int n0 = tl.n0 + (int)crank * BMC, nb = tl.kb1 - tl.kb0;
                int row = ((tl.prob * a.ntt + tl.tt) * a.nkb + tl.kb0) * xrows;
                auto load_w = [&](int i, int st, uint32_t bytes) {
                    if (elect_one()) {
                        if (crank == 0) bar_expect(full0 + st * 8, PAIR * bytes);
                        if (once) tma_load_2d_hint<PAIR>(smem0 + st * stage_bytes, map, n0, (tl.kb0 + i) * BKI, full_of(st), policy);
                        else tma_load_2d<PAIR>(smem0 + st * stage_bytes, map, n0, (tl.kb0 + i) * BKI, full_of(st));
                    }
                };
                auto load_x = [&](int st) {
                    const uint32_t dst = smem0 + st * stage_bytes + kWTile;
                    if (elect_one()) {
                        tma_load_2d<PAIR>(dst, &a.xmap[0], 0, row + (int)crank * n1, full_of(st));
                        if (n2) tma_load_2d<PAIR>(dst + n1 * BKI, &a.xmap[1], 0, row + a.N1 + (int)crank * n2, full_of(st));
                    }
                    row += xrows;
                };
                int i = 0;
                if (seg == 0) {                                        // W does not depend on the work before this launch
                    const int ahead = min(S, nb);
                    for (; i < ahead; ++i) load_w(i, i, stage_bytes);
                    asm volatile("griddepcontrol.wait;" ::: "memory");
                    asm volatile("fence.proxy.async;" ::: "memory");   // the planes were written by ordinary stores
                    for (int q = 0; q < ahead; ++q) load_x(q);
                    s = ahead == S ? 0 : ahead;
                    ph = ahead == S ? 0u : 1u;
                }
                const WideFlags flags = wide_flags(a, tl, lane);
                for (; i < nb; ++i) {
                    ok = warp_wait(empty0 + s * 8, ph);
                    if (!ok) break;
                    load_w(i, s, stage_bytes);
                    load_x(s);
                    if (++s == S) { s = 0; ph ^= 1; }
                }
                if (__builtin_expect(any_wide(flags), 0)) {            // the K range again, with the fourth plane
                    const uint32_t bytes = kWTile + (uint32_t)n3 * BKI;
                    const int lrow = ((tl.prob * a.ntt + tl.tt) * a.nkb + tl.kb0) * a.TT + (int)crank * n3;
                    for (i = 0; i < nb && ok; ++i) {
                        ok = warp_wait(empty0 + s * 8, ph);
                        if (!ok) break;
                        load_w(i, s, bytes);
                        if (elect_one()) tma_load_2d<PAIR>(smem0 + s * stage_bytes + kWTile, &a.lmap, 0, lrow + i * a.TT, full_of(s));
                        if (++s == S) { s = 0; ph ^= 1; }
                    }
                }
            }
            if (!ok) *failed = 1;
        }
    } else if (crank == 0) {
        // ================= MMA issuer =================
        const uint32_t id1 = i8_idesc(BMC * PAIR, a.N1), id2 = i8_idesc(BMC * PAIR, a.N2 ? a.N2 : a.N1), id3 = i8_idesc(BMC * PAIR, a.TT);
        bool ok = true;
        int s = 0;
        uint32_t ph = 0;
        const uint64_t ad0 = sw128_desc(su(smem)), xd0 = sw128_desc(su(smem) + kWTile);
        Item tl;
        for (int seg = 0; ok && item_of<PAIR>(a, unit, seg, tl); ++seg) {
            const int nb = tl.kb1 - tl.kb0;
            const int buf = a.bufcols ? (seg & 1) : 0;
            const uint32_t par = a.bufcols ? ((seg >> 1) & 1) : (seg & 1);
            ok = warp_wait<PAIR == 2>(acc_empty0 + buf * 8, par ^ 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d = tmem + (uint32_t)(buf * a.bufcols);
            WideFlags flags = {};
            for (int i = 0; i < nb && ok; ++i) {
                ok = warp_wait(full0 + s * 8, ph);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t ad = ad0 + ((uint32_t)s * stage_bytes >> 4), xd = xd0 + ((uint32_t)s * stage_bytes >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int j = 0; j < BKI / 32; ++j) {           // one UMMA consumes K = 32: 32 rows of W, 32 bytes of the planes
                        const uint32_t acc = (i > 0 || j > 0) ? 1u : 0u;
                        umma_i8<PAIR>(d, ad + (j * 32 * 128 >> 4), xd + (j * 32 >> 4), id1, acc);
                        if (n2) umma_i8<PAIR>(d + a.N1, ad + (j * 32 * 128 >> 4), xd + ((n1 * BKI + j * 32) >> 4), id2, acc);
                    }
                    commit_i8<PAIR>(empty0 + s * 8);
                }
                __syncwarp();
                if (i == 0) {                                      // behind the first block's MMAs: asked for before them, the flags cost
                    if (seg == 0) asm volatile("griddepcontrol.wait;" ::: "memory");     // 1.5 % of a step of 16 rows
                    flags = wide_flags(a, tl, lane);
                }
                if (++s == S) { s = 0; ph ^= 1; }
            }
            if (ok && __builtin_expect(any_wide(flags), 0)) {      // the K range again, with the fourth plane
                for (int i = 0; i < nb && ok; ++i) {
                    ok = warp_wait(full0 + s * 8, ph);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = ad0 + ((uint32_t)s * stage_bytes >> 4), xd = xd0 + ((uint32_t)s * stage_bytes >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int j = 0; j < BKI / 32; ++j)
                            umma_i8<PAIR>(d + 3 * a.TT, ad + (j * 32 * 128 >> 4), xd + (j * 32 >> 4), id3, (i > 0 || j > 0) ? 1u : 0u);
                        commit_i8<PAIR>(empty0 + s * 8);
                    }
                    __syncwarp();
                    if (++s == S) { s = 0; ph ^= 1; }
                }
            }
            if (ok && elect_one()) commit_i8<PAIR>(acc_full0 + buf * 8);
            __syncwarp();
        }
        if (!ok) *failed = 1;
    }

    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if constexpr (PAIR == 2) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
    if (*failed) {                                                 // a wait gave up: give copies still in flight time to land
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == kEpiWarps) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if constexpr (PAIR == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols) : "memory");
    }
    if (tid == 0 && *failed) atomicExch(a.error_flag, 1u);
}

// ---- host side -------------------------------------------------------------------------------------
struct Plan {
    int TT, ntt, nkb, pair, N1, N2, stages, smem, units, whole, parts, split, ntiles, bufcols, tmem_cols;
    size_t tickets, consts, images, low, slots, bytes;                 // offsets in the workspace, its size
};

// Estimated time of a tile whose K blocks are dealt to `k` CTAs, `ctas` of them at work: a block takes the tensor cores
// 0.28 us (0.39 us with 128 tokens) and HBM 16 KB per CTA; parts cost the exchange through L2.
double split_cost_us(int nkb, int k, int TT, int ctas) {
    const double block = std::max(std::max(0.28, 0.39 * TT / 128), 0.0025 * ctas);
    return (nkb + k - 1) / k * block + (k > 1 ? 2.5 + 0.02 * TT + 0.1 * k : 0.0);
}

// A row is wide when three digits would represent it worse than the fp16 path's hi + lo pairs do.  Three digits round each
// element to a unit (step), so the sum's error relative to the row's norm is sqrt(N / 12) steps over the norm.  The hi + lo
// path's, measured against fp64 below the fp16 store in rows with a peak above ten times their RMS: 5.2e-7 at N = 768, 9.4e-7
// to 1.3e-6 at 4096, 2.9e-6 at 16384 (sums in fp32 tensor-core accumulators); of this the fp32 row sums, common to both
// paths, are 2.5e-7, 4e-7 and 1.2e-6.  The line leaves the total below it; a peak of 5.6 to 12 (N = 768), 12 to 24 (4096) or 31 to
// 62 times the RMS (16384) crosses it, depending on how it lies to the power of two.  Without a fourth plane a channel 300
// times the rest cost 1.9e-5 at N = 4096 in columns whose weight there is the middle code, against 9.4e-7 (now 1.3e-6).
// Returned: the squared norm in steps below which the row is wide.
float wide_norm(int64_t N) { return float(double(N) / 12 / std::pow(3.6e-7 + 1.1e-10 * double(N), 2)); }

Plan make_plan(int nprob, int64_t T, int64_t N, const int64_t* M, bool single) {
    Plan p;
    const int sms = rwkv_sm_count();
    p.nkb = int((N + BKI - 1) / BKI);
    p.ntt = int((T + kMaxTT - 1) / kMaxTT);
    const int per = int((T + p.ntt - 1) / p.ntt);
    // Pairs halve the token planes each CTA fetches and reads; up to 32 rows these are small and single CTAs spread a matrix
    // over twice as many units (4096 x 4096: 16 rows 13.9 against 15.0 us, 64 rows equal, 1024 rows 64 against 56 us).
    p.pair = !single && per > 32 ? 1 : 0;
    const int unit = p.pair ? 32 : 16;
    p.TT = (per + unit - 1) / unit * unit;
    const int n = 3 * p.TT;
    p.N1 = n <= 256 ? n : (n / 2 + unit - 1) / unit * unit;
    p.N2 = n - p.N1;
    const int pc = p.pair ? 2 : 1;
    const int stage = kWTile + n / pc * BKI;
    const int tail = 512 + p.TT * (2 * int(sizeof(RowConst)) + BMC * 2);
    p.stages = std::min(kMaxStages, (kSmemBudget - 1024 - tail) / stage);
    p.smem = 1024 + p.stages * stage + tail;
    p.bufcols = 4 * p.TT <= 256 ? 256 : 0;                         // columns: three planes in two MMAs, then the fourth
    p.tmem_cols = 512;
    p.ntiles = 0;
    for (int i = 0; i < nprob; ++i) p.ntiles += int((M[i] + BMC * pc - 1) / (BMC * pc)) * p.ntt;
    // whole waves, then the rest split along K (at least two K blocks a part) over the units
    const int umax = sms / pc;
    p.whole = p.ntiles / umax * umax;
    const int rest = p.ntiles - p.whole;
    p.split = 1;
    double best = 1e30;
    for (int k = 1; rest > 0 && k <= std::max(1, std::min(umax / rest, p.nkb / 2)); ++k) {
        const double t = split_cost_us(p.nkb, k, p.TT, rest * k * pc);
        if (t < best) { best = t; p.split = k; }
    }
    p.parts = rest * p.split;
    p.units = p.whole > 0 ? umax : p.parts;
    auto up = [](size_t v) { return (v + 1023) / 1024 * 1024; };
    p.tickets = 1024;
    p.consts = up(p.tickets + size_t(umax) * pc * 4);
    p.images = up(p.consts + size_t(nprob) * T * sizeof(RowConst));
    p.low = up(p.images + size_t(nprob) * p.ntt * p.nkb * size_t(n) * BKI);
    p.slots = up(p.low + size_t(nprob) * p.ntt * p.nkb * size_t(p.TT) * BKI);
    p.bytes = p.slots + (p.split > 1 ? size_t(p.parts) * pc * p.TT * BMC * 8 : 0);
    return p;
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
    static EncodeFn fn = []() -> EncodeFn {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult st;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &st) != cudaSuccess || st != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        return reinterpret_cast<EncodeFn>(f);
    }();
    return fn;
}

bool g_i8_single = false;                // one CTA per tile always (set through rwkv_mm8_seq_set_path)

}  // namespace

void rwkv_mm8_seq_i8_set_single_cta(bool single) { g_i8_single = single; }

size_t rwkv_mm8_seq_i8_workspace_bytes(int nprob, int64_t T, int64_t N, const int64_t* M) {
    if (nprob < 1 || nprob > kSeqI8MaxProblems || T < 1 || N < 1 || N > 65536) return 0;
    return std::max(make_plan(nprob, T, N, M, false).bytes, make_plan(nprob, T, N, M, true).bytes);
}

int rwkv_mm8_seq_i8(int nprob, const SeqI8Problem* probs, int64_t T, int64_t N, void* workspace, size_t workspace_bytes, void* stream) {
    RWKV_CHECK_ARG(nprob >= 1 && nprob <= kSeqI8MaxProblems && T >= 1 && N >= 1);
    if (N > 65536 || T > (1 << 18)) return RWKV_ERR_UNSUPPORTED;
    int64_t M[kSeqI8MaxProblems];
    for (int i = 0; i < nprob; ++i) {
        const SeqI8Problem& q = probs[i];
        if (reinterpret_cast<uintptr_t>(q.w) % 16 != 0 || q.w_stride % 16 != 0) return RWKV_ERR_UNSUPPORTED;   // TMA rows
        M[i] = q.M;
    }
    if (encode_fn() == nullptr) return RWKV_ERR_UNSUPPORTED;
    static int use_pair = -1;            // RWKV_B200_SEQ_PAIR=0: never the CTA-pair form (same results)
    if (use_pair < 0) { const char* e = getenv("RWKV_B200_SEQ_PAIR"); use_pair = (e != nullptr && e[0] == '0') ? 0 : 1; }
    const Plan p = make_plan(nprob, T, N, M, !use_pair || g_i8_single);
    if (workspace == nullptr || workspace_bytes < p.bytes) return RWKV_ERR_WORKSPACE;
    RWKV_CHECK_ALIGN(workspace, 256);
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    I8Args a;
    memset(&a, 0, sizeof(a));
    PrepArgs pa;
    memset(&pa, 0, sizeof(pa));
    const int pc = p.pair ? 2 : 1;
    int tile = 0;
    bool vec = true;
    const int pro = probs[0].pro.kind;
    auto al = [](const void* ptr, int64_t stride_bytes) { return reinterpret_cast<uintptr_t>(ptr) % 16 == 0 && stride_bytes % 16 == 0; };
    for (int i = 0; i < nprob; ++i) {
        const SeqI8Problem& q = probs[i];
        const cuuint64_t dims[2] = {(cuuint64_t)q.M, (cuuint64_t)N}, strides[1] = {(cuuint64_t)q.w_stride};
        const cuuint32_t box[2] = {BMC, BKI}, es[2] = {1, 1};
        if (encode_fn()(&a.wmap[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(q.w), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return RWKV_ERR_UNSUPPORTED;
        I8Problem& d = a.p[i];
        d.mx = static_cast<const __half*>(q.mx); d.rx = static_cast<const __half*>(q.rx);
        d.vec = al(q.y, q.y_stride * 2) && (q.epi.aux == nullptr || al(q.epi.aux, q.epi.aux_stride * 2)) &&
                (q.epi.aux2 == nullptr || al(q.epi.aux2, q.epi.aux2_stride * 2));
        d.y = static_cast<__half*>(q.y); d.y_stride = q.y_stride; d.epi = q.epi; d.M = int(q.M); d.tile0 = tile;
        tile += int((q.M + BMC * pc - 1) / (BMC * pc)) * p.ntt;
        PrepProblem& r = pa.p[i];
        r.pro = q.pro; r.x = q.x; r.x_stride = q.x_stride;
        r.ry = static_cast<const __half*>(q.ry); r.my = static_cast<const __half*>(q.my);
        const int xel = pro == RWKV_PRO_GN_GATE ? 4 : 2;
        vec = vec && al(q.x, q.x_stride * xel) && al(q.ry, 0) && al(q.my, 0) && al(q.pro.sx, q.pro.sx_stride * 2) && al(q.pro.ln_w, 0) &&
              al(q.pro.ln_b, 0) && al(q.pro.mix, 0) && al(q.pro.xx_out, q.pro.xx_stride * 2) && al(q.pro.new_state, 0) &&
              al(q.pro.gate, q.pro.gate_stride * 2) && al(q.pro.k, 0) && al(q.pro.v, 0) && al(q.pro.t_decay, 0) && al(q.pro.t_first, 0) &&
              al(q.pro.aa, 0) && al(q.pro.bb, 0) && al(q.pro.pp, 0);
    }
    if (pro == RWKV_PRO_WKV4 && N % 8 != 0) vec = false;          // rows N apart
    pa.nprob = nprob; pa.vec = vec ? 1 : 0; pa.T = int(T); pa.N = int(N); pa.nkb = p.nkb; pa.TT = p.TT; pa.ntt = p.ntt;
    pa.ntickets = p.split > 1 ? p.parts / p.split * pc : 0;
    pa.narrow = wide_norm(N); pa.low = ws + p.low;
    pa.images = ws + p.images; pa.consts = reinterpret_cast<RowConst*>(ws + p.consts); pa.tickets = reinterpret_cast<unsigned*>(ws + p.tickets);
    const long long xrows = (long long)nprob * p.ntt * p.nkb * 3 * p.TT;
    if (xrows >= (1ll << 31)) return RWKV_ERR_UNSUPPORTED;
    for (int i = 0; i < (p.N2 ? 2 : 1); ++i) {
        const cuuint64_t dims[2] = {BKI, (cuuint64_t)xrows}, strides[1] = {BKI};
        const cuuint32_t box[2] = {BKI, (cuuint32_t)((i ? p.N2 : p.N1) / pc)}, es[2] = {1, 1};
        if (encode_fn()(&a.xmap[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, pa.images, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return RWKV_ERR_UNSUPPORTED;
    }
    {
        const cuuint64_t dims[2] = {BKI, (cuuint64_t)(xrows / 3)}, strides[1] = {BKI};
        const cuuint32_t box[2] = {BKI, (cuuint32_t)(p.TT / pc)}, es[2] = {1, 1};
        if (encode_fn()(&a.lmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, pa.low, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return RWKV_ERR_UNSUPPORTED;
    }
    a.consts = pa.consts; a.tickets = pa.tickets; a.slots = reinterpret_cast<long long*>(ws + p.slots);
    a.error_flag = reinterpret_cast<unsigned*>(ws);
    a.nprob = nprob; a.T = int(T); a.TT = p.TT; a.ntt = p.ntt; a.nkb = p.nkb; a.N1 = p.N1; a.N2 = p.N2; a.stages = p.stages;
    a.units = p.units; a.whole = p.whole; a.parts = p.parts; a.split = p.split;
    a.bufcols = p.bufcols; a.tmem_cols = p.tmem_cols;

    static bool configured[64] = {};         // function attributes are per device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) { cudaGetLastError(); return RWKV_ERR_LAUNCH; }
    if (dev >= 64 || !configured[dev]) {
        if (cudaFuncSetAttribute(mm8_seq_i8_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget) != cudaSuccess ||
            cudaFuncSetAttribute(mm8_seq_i8_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget) != cudaSuccess) {
            cudaGetLastError();
            return RWKV_ERR_LAUNCH;
        }
        if (dev < 64) configured[dev] = true;
    }
    // Few rows: a block per (row, matrix), so that they run side by side (E: see above).
    // Many rows: the row is normalised once for all matrices, and as many blocks as fit an SM matter more than what one of
    // them takes (1024 rows of 4096, LayerNorm + 2 matrices: 47 us with 2 blocks of 128 registers a thread on an SM).
    const bool few = T * nprob <= 2 * rwkv_sm_count();
    const dim3 pgrid((unsigned)T, (unsigned)(few ? nprob : 1));
    const int Np = p.nkb * BKI;
    if (pro != RWKV_PRO_PLAIN && Np > 16384) return RWKV_ERR_UNSUPPORTED;
    const int E = (few || pro == RWKV_PRO_WKV4) && Np <= 1024 ? 4 : (few || pro == RWKV_PRO_WKV4) && Np <= 8192 ? 8 : 16;
    const int threads = std::min(1024, (Np / E + 31) / 32 * 32);
    auto prep = [&](auto kernel, int n) { return rwkv_launch_pdl(kernel, pgrid, dim3(n), 0, st, pa); };
    int rc;
    if (pro == RWKV_PRO_PLAIN) {
        if (E == 4) rc = prep(mm8_seq_i8_prep<RWKV_PRO_PLAIN, 4, false, true, 1024, 2>, threads);
        else if (E == 8) rc = prep(mm8_seq_i8_prep<RWKV_PRO_PLAIN, 8, false, true, 1024, 1>, threads);
        else if (few) rc = prep(mm8_seq_i8_prep<RWKV_PRO_PLAIN, 8, true, false, 1024, 1>, 1024);
        else rc = prep(mm8_seq_i8_prep<RWKV_PRO_PLAIN, 16, true, false, 256, 4>, std::min(256, threads));
    } else if (pro == RWKV_PRO_LN_MIX) {
        if (E == 4) rc = prep(mm8_seq_i8_prep<RWKV_PRO_LN_MIX, 4, false, true, 1024, 2>, threads);
        else if (E == 8) rc = prep(mm8_seq_i8_prep<RWKV_PRO_LN_MIX, 8, false, true, 1024, 1>, threads);
        else if (threads > 512) rc = prep(mm8_seq_i8_prep<RWKV_PRO_LN_MIX, 16, false, false, 1024, 1>, threads);
        else if (threads > 256) rc = prep(mm8_seq_i8_prep<RWKV_PRO_LN_MIX, 16, false, false, 512, 2>, threads);
        else rc = prep(mm8_seq_i8_prep<RWKV_PRO_LN_MIX, 16, false, false, 256, 4>, threads);
    } else if (pro == RWKV_PRO_WKV4) {
        if (E == 4) rc = prep(mm8_seq_i8_prep<RWKV_PRO_WKV4, 4, false, true, 1024, 2>, threads);
        else if (E == 8) rc = prep(mm8_seq_i8_prep<RWKV_PRO_WKV4, 8, false, true, 1024, 1>, threads);
        else rc = prep(mm8_seq_i8_prep<RWKV_PRO_WKV4, 16, false, false, 1024, 1>, threads);
    } else {
        if (E == 4) rc = prep(mm8_seq_i8_prep<RWKV_PRO_GN_GATE, 4, false, true, 1024, 2>, threads);
        else if (E == 8) rc = prep(mm8_seq_i8_prep<RWKV_PRO_GN_GATE, 8, false, true, 1024, 1>, threads);
        else if (threads > 512) rc = prep(mm8_seq_i8_prep<RWKV_PRO_GN_GATE, 16, false, false, 1024, 1>, threads);
        else if (threads > 256) rc = prep(mm8_seq_i8_prep<RWKV_PRO_GN_GATE, 16, false, false, 512, 2>, threads);
        else rc = prep(mm8_seq_i8_prep<RWKV_PRO_GN_GATE, 16, false, false, 256, 4>, threads);
    }
    if (rc != RWKV_OK) return rc;
    if (!p.pair) return rwkv_launch_pdl(mm8_seq_i8_kernel<1>, dim3(p.units), dim3(kThreadsI8), size_t(p.smem), st, a);
    return rwkv_launch_pdl_clustered(2, mm8_seq_i8_kernel<2>, dim3(p.units * 2), dim3(kThreadsI8), size_t(p.smem), st, a);
}
