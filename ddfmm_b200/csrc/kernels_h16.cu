// Mixed-form high-frequency GEMM on the FP16 tensor cores (tcgen05 kind::f16).
//
// Problem (as in umma_cgemm_kernel): Y[:, c] += A X[:, c] for gathered columns c,
// complex FP32.  Every vector (and every operator row) is scaled by a power of
// two to a largest component in [2^13, 2^14) and written as two FP16 planes,
// hi = FP16(x), lo = FP16(x - hi): 22 bits of every component that is not more
// than 2^17 below the largest, and an absolute 2^-39 of the largest below that.
// Outgoing vectors' components differ by more at P = 8: they and the operators on them
// are evened out by the vectors' profiles first, as in kernels_i8.cu (on a K = 8 cluster at
// P = 8 M2L products are 1.1e-6 off with them, 1.7e-5 without, split TF32 2.2e-6; elsewhere
// 0.4-2.4e-6 by pass on evals' own vectors, split TF32 0.8-4.5e-6).  A product is hi hi + lo hi + hi lo in FP32, like the three TF32 products of
// umma_cgemm_kernel with rounded instead of truncated halves, at twice their
// rate and half their operand bytes.  On random products of 16 to 400 terms the
// result is 0.2-2.9e-6 from a long-double one in relative 2-norm, that kernel's
// 0.3-5.8e-6.
//
// What that kernel waited for was mostly its own latency: a tile's columns came
// through registers, split on the way, behind a chain of tile, problem and column
// offset loads.  Here the planes are written once per vector (h16_slice_kernel:
// 128-byte granules, 16 complex numbers' hi then lo) and gathered by 16-byte
// cp.async straight into the swizzled layout, a tile is one self-contained 32-byte
// record read a tile ahead, and three slots of 32 reals are in flight.
//
// Tile: 128 gathered columns (M, a TMEM lane each) x up to 112 complex rows (N =
// 2 rows real rows, interleaved as in umma_pack_kernel), two accumulators of 256
// TMEM columns, so a tile's epilogue overlaps the next one's main loop.
// Persistent, one block per SM.  Warps:
//   0 .. 2  operands: warp w owns ring slot w; the operator block by one bulk
//           copy, the columns by cp.async (8 lanes fill two 64-byte rows)
//   3       MMA issue, one thread
//   4 .. 7  epilogue on TMEM lanes 32 (w % 4) ..: TMEM -> scaled -> parking area;
//           each lane adds its column's piece with one bulk reduction
// Measured, the passes of a K = 64, P = 6 sphere: 9.6 ms in all against 14.2 for
// umma_cgemm_kernel (m 100, k 152, 3.76 million columns: 1.7 ms, 269 TF/s of complex
// products).  With the outputs dropped the 9.6 are 7.0, which is the operand copies'
// rate (43 KB a K block of a 100-row tile, 9.3 TB/s over the chip; the MMAs need
// half of it).  The rest is the reductions, whose cost is by piece: pieces of 16
// rows make it 13.2 ms, of 32 rows 11.9, so a tile parks up to 56 rows at once and
// the ring has three slots, not four (float4 atomics of parked rows: 13.9 ms).
// Every mbarrier wait is bounded as in umma_cgemm_kernel; a block that gives up
// drains its copies, frees its TMEM and sets *err.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.cuh"
#include "umma.cuh"

namespace ddfmm {

namespace {
constexpr int HM = 128;
constexpr int HNMAX = 2 * H16_TILE_ROWS;
constexpr int HSLOTS = 3;
constexpr int H_X_PLANE = HM * 64;               // bytes of one plane of a column block
constexpr int H_X_BYTES = 2 * H_X_PLANE;
constexpr int H_SLOT_BYTES = H_X_BYTES + 2 * HNMAX * 64;
constexpr int HCH = H16_TILE_ROWS / 2;           // most complex rows parked per column
constexpr int HPS = HCH + 2;                     // parked column's stride (complex): 16-byte stores of 8 lanes hit all banks
constexpr int H_PARK_WARP = 32 * HPS * 8;
constexpr int H_SMEM = HSLOTS * H_SLOT_BYTES + 4 * H_PARK_WARP + 1024;
static_assert(H_SMEM + 6144 <= 232448, "shared memory per block");
static_assert(H_SLOT_BYTES % 1024 == 0, "swizzle atoms");
constexpr int HTHREADS = 256;

// K-major descriptors of 64-byte rows: swizzled columns (layout 4) and the operator's
// core matrices (no swizzle; K-adjacent ones 128 bytes apart); 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t h16_desc_x(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)4 << 61);
}
__device__ __forceinline__ uint64_t h16_desc_b(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3FFF) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void h16_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u)
        : "memory");
}

// Scale of a vector whose largest |x| has the bits `top`: x s in [2^13, 2^14) for that
// component; NaN for a vector holding an infinity or a NaN.  A vector with nothing above
// 2^-63 is brought up by 2^100 first (low), so subnormals keep their bits.  With |x| < 2^e
// (before that) an output is the sum of planes' products times 2^(e - 14) for the vector and
// for the operator row: stored as 2^(e - 1) (h16_out, exact for every FP32 vector) and 2^(e - 27).
constexpr int H_UP = 100;
constexpr uint32_t H_LOW = 64u << 23;  // top below it: low
struct H16Scale {
    float s;
    int b;  // e + 126
};
__device__ __forceinline__ float h16_pow2(int e) {  // 2^e; 0 below 2^-149
    return e >= -126 ? __uint_as_float((uint32_t)(127 + e) << 23) : e >= -149 ? __uint_as_float(1u << (e + 149)) : 0.f;
}
__device__ __forceinline__ H16Scale h16_scale(uint32_t top, bool low) {
    H16Scale r;
    const int be = (int)(top >> 23);
    if (be == 255) {
        r.s = 0.f;
        r.b = 255;
        return r;
    }
    const int b1 = top == 0 ? 127 : be < 13 ? 13 : be;  // boosted by 2^100 it is 18 or more
    r.s = h16_pow2(140 - b1);
    r.b = b1 - (low ? H_UP : 0);
    return r;
}
__device__ __forceinline__ float h16_out(const H16Scale& S, int by) {  // 2^(e - by)
    return S.b == 255 ? __uint_as_float(0x7fc00000u) : h16_pow2(S.b - 126 - by);
}
// two values: hi and lo halves of each
__device__ __forceinline__ void h16_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }

template <class T>
__device__ __forceinline__ int sub_of(const T* prefix, int nsub, T i) {
    int lo = 0, hi = nsub - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= i)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}
}  // namespace

// ---------------------------------------------------------------- planes
// One warp per vector, four lanes per granule (4 complex numbers each: 16 bytes
// of hi, 16 of lo); a vector of up to 128 numbers is read once and kept in registers.
// Bound by HBM: 8 bytes read and 8 written per complex number; 4.3-4.4 TB/s on 2.5
// million vectors of 100 (16-byte loads: the same; two vectors a warp: 2% faster
// there, a tenth slower where vectors do not fill the SMs).
// A vector's planes by one warp; UP: components brought up by 2^UP first.  False, and nothing
// written, where the vector is low and was not brought up.
template <bool PROF, int UP>
__device__ __forceinline__ bool h16_slice_vector(const float2* x, const unsigned char* prof, float* cx, char* out, int len,
                                                 int lane) {
    float2 v[4];
    auto load = [&](int j0) {
        uint32_t b = 0x7f7f7f7fu;
        if (PROF && j0 < len) b = __ldg(reinterpret_cast<const uint32_t*>(prof + j0));
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = j0 + i < len ? x[j0 + i] : make_float2(0.f, 0.f);
        if (PROF || UP) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float f = __uint_as_float((((b >> (8 * i)) & 255u) + UP) << 23);
                v[i] = make_float2(v[i].x * f, v[i].y * f);
            }
        }
    };
    uint32_t top = 0;
    for (int j0 = 0; j0 < len; j0 += 128) {
        load(j0 + lane * 4);
#pragma unroll
        for (int i = 0; i < 4; ++i) top = max(top, max(abs_bits(v[i].x), abs_bits(v[i].y)));
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (!UP && top < H_LOW) return false;
    const H16Scale C = h16_scale(top, UP > 0);
    if (lane == 0) *cx = h16_out(C, 1);
    for (int j0 = 0; j0 < len; j0 += 128) {
        if (len > 128) load(j0 + lane * 4);
        const int g = (j0 >> 4) + (lane >> 2);
        if (g * 16 < len) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) h16_split(v[i].x * C.s, v[i].y * C.s, hi[i], lo[i]);
            char* o = out + g * H16_GRANULE + (lane & 3) * 16;
            *reinterpret_cast<uint4*>(o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(o + 64) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
    }
    return true;
}
// rare: out of the kernel's way, which runs six blocks an SM at 40 registers (the outgoing
// vectors of a K = 64 sphere 0.84 ms; five blocks 1.00)
template <bool PROF>
__device__ __noinline__ void h16_slice_low(const float2* x, const unsigned char* prof, float* cx, char* out, int len,
                                           int lane) {
    h16_slice_vector<PROF, H_UP>(x, prof, cx, out, len, lane);
}
struct HSliceRef {  // vector w of a launch
    const float2* x;
    const unsigned char* prof;
    float* cx;
    char* out;
    int len;
};
template <bool PROF>
__device__ __forceinline__ HSliceRef h16_slice_ref(const HSliceSub& S, int i) {
    const I8Vec V = S.vecs[i];
    return HSliceRef{S.X + V.src, PROF ? S.prof.prof + (size_t)(V.profile - 1) * S.prof.stride : nullptr, S.cx + V.gran,
                     S.X16 + (size_t)V.gran * H16_GRANULE, V.len};
}
template <bool PROF>  // finds the vector again: nothing of it has to be kept for this
__device__ __noinline__ void h16_slice_low_multi(const HSliceSub* subs, const int* prefix, int nsub, int w) {
    const int j = sub_of(prefix, nsub, w);
    const HSliceRef R = h16_slice_ref<PROF>(subs[j], w - prefix[j]);
    h16_slice_vector<PROF, H_UP>(R.x, R.prof, R.cx, R.out, R.len, threadIdx.x & 31);
}

// PROF: the vectors have profiles (a launch's all do or none does).
template <bool MULTI, bool PROF>
__global__ void __launch_bounds__(256, 6) h16_slice_kernel(const HSliceSub one, const HSliceSub* __restrict__ subs,
                                                           const int* __restrict__ prefix, int nsub, int n,
                                                           const int* __restrict__ active) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= n) return;
    const int j = MULTI ? sub_of(prefix, nsub, w) : 0;
    const HSliceSub& S = MULTI ? subs[j] : one;
    if (active && !active[S.inst]) return;
    const HSliceRef R = h16_slice_ref<PROF>(S, MULTI ? w - prefix[j] : w);
    if (h16_slice_vector<PROF, 0>(R.x, R.prof, R.cx, R.out, R.len, lane)) return;
    if (MULTI)
        h16_slice_low_multi<PROF>(subs, prefix, nsub, (blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    else
        h16_slice_low<PROF>(R.x, R.prof, R.cx, R.out, R.len, lane);
}

void launch_h16_slice(const HSliceSub* subs, const int* prefix, int nsub, int n, const int* active, cudaStream_t s,
                      const HSliceSub& one) {
    if (n <= 0) return;
    auto kernel = nsub == 1 ? (one.prof.prof ? h16_slice_kernel<false, true> : h16_slice_kernel<false, false>)
                            : (one.prof.prof ? h16_slice_kernel<true, true> : h16_slice_kernel<true, false>);
    kernel<<<(unsigned)((n + 7) / 8), 256, 0, s>>>(one, subs, prefix, nsub, n, active);
}

int h16_tile_rows(int m) {
    const int n = (m + H16_TILE_ROWS - 1) / H16_TILE_ROWS;
    return ((m + n - 1) / n + 7) / 8 * 8;
}
int h16_row_tiles(int m) { return (m + h16_tile_rows(m) - 1) / h16_tile_rows(m); }
size_t h16_packed_floats(int m, int k) {  // planes, then the rows' output scales
    return (size_t)h16_row_tiles(m) * ((k + 15) / 16) * 2 * 2 * h16_tile_rows(m) * 16 + (m + 3) / 4 * 4;
}
const float* h16_scales(const float* packed, int m, int k) {
    return packed + h16_packed_floats(m, k) - (m + 3) / 4 * 4;
}

// Operator planes (setup only): block (row tile, job).  K block kb of a row tile:
// hi plane then lo plane, each 2 rows_t real rows of 64 bytes in core-matrix order.
__global__ void __launch_bounds__(256) h16_pack_kernel(const H16PackJob* __restrict__ jobs, int njobs) {
    __shared__ uint32_t tops[2][128];
    __shared__ H16Scale sc[128];
    __shared__ bool low[128];
    const int tid = threadIdx.x;
    for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
        const H16PackJob J = jobs[j];
        const int row0 = blockIdx.x * J.rows_t;
        if (row0 >= J.m) continue;  // uniform over the block
        // column k as the vectors' profile leaves it, brought up where the row is low
        auto entry = [&](int r, int k, bool up) {
            const float2 a = J.A[(size_t)k * J.lda + row0 + r];
            const float f = h16_pow2(J.prof ? 127 - J.prof[k] : 0), g = h16_pow2(up ? H_UP : 0);
            return make_float2(a.x * f * g, a.y * f * g);
        };
        for (int up = 0; up < 2; ++up) {
            __syncthreads();
            const int r = tid & 127;
            uint32_t top = 0;
            if (r < J.rows_t && row0 + r < J.m && (up == 0 || low[r]))
                for (int k = tid >> 7; k < J.k; k += 2) {
                    const float2 a = entry(r, k, up);
                    top = max(top, max(abs_bits(a.x), abs_bits(a.y)));
                }
            tops[tid >> 7][r] = top;
            __syncthreads();
            if (tid < J.rows_t) {
                const uint32_t t = max(tops[0][tid], tops[1][tid]);
                if (up == 0) low[tid] = t < H_LOW;
                if (up == 0 || low[tid]) sc[tid] = h16_scale(t, up);
            }
        }
        if (tid < J.rows_t && row0 + tid < J.m) J.ra[row0 + tid] = h16_out(sc[tid], 27);
        __syncthreads();
        const int nkb = (J.k + 15) / 16, nq = nkb * 4, N = 2 * J.rows_t;
        char* dst = reinterpret_cast<char*>(J.dst) + (size_t)blockIdx.x * nkb * 2 * N * 64;
        for (int e = tid; e < nq * J.rows_t; e += 256) {
            const int r = e % J.rows_t, q4 = e / J.rows_t, k0 = q4 * 4;
            const H16Scale C = sc[r];
            uint32_t h0[4], l0[4], h1[4], l1[4];  // rows [Ar, -Ai] and [Ai, Ar]
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool ok = row0 + r < J.m && k0 + i < J.k;
                const float2 a = ok ? entry(r, k0 + i, low[r]) : make_float2(0.f, 0.f);
                const float re = a.x * C.s, im = a.y * C.s;
                h16_split(re, -im, h0[i], l0[i]);
                h16_split(im, re, h1[i], l1[i]);
            }
            char* blk = dst + (size_t)(q4 >> 2) * 2 * N * 64;
            const int n = 2 * r, o = (n >> 3) * 512 + (q4 & 3) * 128 + (n & 7) * 16;
            *reinterpret_cast<uint4*>(blk + o) = make_uint4(h0[0], h0[1], h0[2], h0[3]);
            *reinterpret_cast<uint4*>(blk + o + 16) = make_uint4(h1[0], h1[1], h1[2], h1[3]);
            *reinterpret_cast<uint4*>(blk + N * 64 + o) = make_uint4(l0[0], l0[1], l0[2], l0[3]);
            *reinterpret_cast<uint4*>(blk + N * 64 + o + 16) = make_uint4(l1[0], l1[1], l1[2], l1[3]);
        }
    }
}

void launch_h16_pack(const H16PackJob* jobs, int njobs, int max_tiles, cudaStream_t s) {
    if (njobs > 0) h16_pack_kernel<<<dim3(max_tiles, njobs < 32768 ? njobs : 32768), 256, 0, s>>>(jobs, njobs);
}

void h16_tiles(const float* packed, int m, int k, int col0, int ncol, std::vector<H16Tile>& out) {
    const int nrt = h16_row_tiles(m), rt = h16_tile_rows(m), nkb = (k + 15) / 16;
    const float* ra = h16_scales(packed, m, k);
    for (int c = 0; c < ncol; c += HM)
        for (int r = 0; r < nrt; ++r)
            out.push_back(H16Tile{packed + (size_t)r * nkb * 2 * 2 * rt * 16, ra + r * rt, col0 + c, r * rt,
                                  (unsigned short)(ncol - c < HM ? ncol - c : HM),
                                  (unsigned short)(m - r * rt < rt ? m - r * rt : rt), (unsigned short)(2 * rt),
                                  (unsigned short)k});
}

// ---------------------------------------------------------------- GEMM
namespace {
struct HTileRef {
    H16Tile t;
    int sub;
};
constexpr int H_SUBS_SMEM = 64;

// Tile ti of the launch: its sub-launch (order[ti] = sub << 24 | tile, or by the
// prefix sums) and record; past the end, tile 0 (read ahead, never used)
template <bool MULTI>
__device__ __forceinline__ HTileRef h16_tile(const HSub& one, const HSub* subs, const int* prefix, int nsub, int ntiles,
                                             const int* __restrict__ order, int ti) {
    if (ti >= ntiles) ti = 0;
    HTileRef r;
    r.sub = 0;
    int t = ti;
    if (MULTI) {
        if (order) {
            const unsigned e = (unsigned)__ldg(order + ti);
            r.sub = (int)(e >> 24);
            t = (int)(e & 0xFFFFFFu);
        } else {
            r.sub = sub_of(prefix, nsub, ti);
            t = ti - prefix[r.sub];
        }
    }
    union {
        int4 w[2];
        H16Tile t;
    } u;
    static_assert(sizeof(H16Tile) == 32, "two 16-byte loads");
    const int4* p = reinterpret_cast<const int4*>((MULTI ? subs[r.sub] : one).tiles + t);
    u.w[0] = __ldg(p);
    u.w[1] = __ldg(p + 1);
    r.t = u.t;
    return r;
}
}  // namespace

template <bool MULTI>
__global__ void __launch_bounds__(HTHREADS, 1) h16_gemm_kernel(const HSub one, const HSub* __restrict__ gsubs,
                                                               const int* __restrict__ gprefix, int nsub, int ntiles,
                                                               const int* __restrict__ order,
                                                               const int* __restrict__ active, int* err,
                                                               unsigned long long wait_ns, int withhold) {
    extern __shared__ __align__(1024) unsigned char hsm_raw[];
    __shared__ HSub ssubs[MULTI ? H_SUBS_SMEM : 1];
    __shared__ int sprefix[MULTI ? H_SUBS_SMEM + 1 : 1];
    __shared__ __align__(8) uint64_t full[HSLOTS], empty[HSLOTS], acc_full[2], acc_empty[2], drained;
    __shared__ uint32_t tmem_base;
    __shared__ int failed_s;
    volatile int* failed = &failed_s;
    const bool cached = MULTI && nsub <= H_SUBS_SMEM;
    if (cached) {
        for (int i = threadIdx.x; i < nsub; i += blockDim.x) ssubs[i] = gsubs[i];
        for (int i = threadIdx.x; i <= nsub; i += blockDim.x) sprefix[i] = gprefix[i];
    }
    const HSub* subs = cached ? ssubs : gsubs;
    const int* prefix = cached ? sprefix : gprefix;
    unsigned char* sm = (unsigned char*)(((uintptr_t)hsm_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        failed_s = 0;
        for (int s = 0; s < HSLOTS; ++s) {
            mbar_init(&full[s], 2);   // the operator copy's bytes, the gathered columns
            mbar_init(&empty[s], 1);  // tcgen05.commit
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);   // tcgen05.commit
            mbar_init(&acc_empty[a], 4);  // epilogue warps
        }
        mbar_init(&drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_base;
    auto tile_at = [&](int ti) { return h16_tile<MULTI>(one, subs, prefix, nsub, ntiles, order, ti); };
    auto sub_at = [&](int j) -> const HSub& { return MULTI ? subs[j] : one; };
    HTileRef next = tile_at(blockIdx.x);

    if (warp < HSLOTS) {
        // ------------------------------------------------ operands
        // lane l copies 16-byte piece l % 4 of both planes of columns l / 4 + 8 i
        const int piece = lane & 3, sub = lane >> 2;
        const uint32_t dst = smem_u32(sm) + warp * H_SLOT_BYTES + sub * 64 + ((piece ^ ((sub >> 1) & 3)) << 4);
        uint32_t parity = 1;  // of empty[warp]; the first wait passes
        int slot = 0;  // of the next K block
        bool ok = true;
        int ahead[16];  // the next tile's columns' first granules, -1 past the last one
        auto granules = [&](const HTileRef& R) {
            const int* g = sub_at(R.sub).xgran + R.t.col;
#pragma unroll
            for (int i = 0; i < 16; ++i) ahead[i] = sub + 8 * i < R.t.ncol ? __ldg(g + sub + 8 * i) : -1;
        };
        granules(next);
        for (int ti = blockIdx.x; ti < ntiles && ok; ti += gridDim.x) {
            const HTileRef R = next;
            int gran[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) gran[i] = ahead[i];
            next = tile_at(ti + gridDim.x);
            granules(next);
            const HSub& S = sub_at(R.sub);
            if (active && !active[S.inst]) continue;
            const H16Tile T = R.t;
            const char* X16 = S.X16 + piece * 16;
            const uint32_t bytes = (uint32_t)T.n * 128;
            const int nkb = (T.k + 15) >> 4;
            for (int kb = 0; kb < nkb; ++kb) {
                const bool own = slot == warp;
                slot = slot + 1 < HSLOTS ? slot + 1 : 0;
                if (!own) continue;
                if (!warp_wait(&empty[warp], parity, failed, wait_ns)) {
                    *failed = 1;
                    ok = false;
                    break;
                }
                parity ^= 1;
                if (lane == 0 && !(withhold && blockIdx.x == 0)) {  // withheld: full[warp] never completes
                    mbar_expect_tx(&full[warp], bytes);
                    bulk_g2s(sm + warp * H_SLOT_BYTES + H_X_BYTES, reinterpret_cast<const char*>(T.B) + (size_t)kb * bytes,
                             bytes, &full[warp]);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const char* a = X16 + (gran[i] < 0 ? 0 : (size_t)(gran[i] + kb) * H16_GRANULE);
                    const int n = gran[i] < 0 ? 0 : 16;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst + i * 512), "l"(a), "r"(n));
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst + H_X_PLANE + i * 512),
                                 "l"(a + 64), "r"(n));
                }
                asm volatile("cp.async.wait_all;\n" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[warp]);
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    } else if (warp == 3) {
        if (lane == 0) {
            // -------------------------------------------- MMA issue
            uint32_t slot = 0, fpar = 0, ready = 0;
            int it = 0;
            bool ok = true;
            for (int ti = blockIdx.x; ti < ntiles && ok; ti += gridDim.x) {
                const HTileRef R = next;
                next = tile_at(ti + gridDim.x);
                if (active && !active[sub_at(R.sub).inst]) continue;
                const int k = R.t.k, N = R.t.n, nkb = (k + 15) >> 4;
                const uint32_t idesc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(HM >> 4) << 24);
                const uint64_t blo = (uint64_t)(N * 4);  // hi plane to lo plane of the operator, 16-byte units
                const int a = it & 1;
                ok = mbar_wait(&acc_empty[a], ((it >> 1) & 1) ^ 1, failed, wait_ns);  // the first of each passes
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t d = tmem + (uint32_t)(a * 256);
                for (int kb = 0; kb < nkb; ++kb) {
                    if (!ready) ok = mbar_wait(&full[slot], fpar, failed, wait_ns);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t base = smem_u32(sm) + slot * H_SLOT_BYTES;
                    const uint64_t dx = h16_desc_x(base), db = h16_desc_b(base + H_X_BYTES);
                    uint64_t* const done = &empty[slot];
                    slot = slot + 1 < HSLOTS ? slot + 1 : 0;
                    fpar ^= slot == 0;
                    const bool two = k - kb * 16 > 8;  // the second K step holds k
                    h16_mma(d, dx, db, idesc, kb > 0);
                    h16_mma(d, dx + (H_X_PLANE >> 4), db, idesc, 1u);
                    ready = mbar_peek(&full[slot], fpar);  // answered while the rest runs
                    h16_mma(d, dx, db + blo, idesc, 1u);
                    if (two) {  // 32 bytes on: 2 of the swizzled rows' units, two core matrices of the operator's
                        h16_mma(d, dx + 2, db + 16, idesc, 1u);
                        h16_mma(d, dx + 2 + (H_X_PLANE >> 4), db + 16, idesc, 1u);
                        h16_mma(d, dx + 2, db + 16 + blo, idesc, 1u);
                    }
                    umma_commit(done);
                }
                if (!ok) break;
                umma_commit(&acc_full[a]);
                ++it;
            }
            if (!ok) {  // let the MMAs already issued finish before TMEM is freed
                *failed = 1;
                umma_commit(&drained);
                mbar_wait(&drained, 0, nullptr, wait_ns);
            }
        }
    } else {
        // ------------------------------------------------ epilogue
        const int qw = warp & 3, col = qw * 32 + lane;
        float2* const park = reinterpret_cast<float2*>(sm + HSLOTS * H_SLOT_BYTES + qw * H_PARK_WARP) + lane * HPS;
        int it = 0;
        for (int ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
            const HTileRef R = next;
            next = tile_at(ti + gridDim.x);
            const HSub& S = sub_at(R.sub);
            if (active && !active[S.inst]) continue;
            const H16Tile T = R.t;
            const int a = it & 1;
            float c = 0.f;
            float2* y = nullptr;  // this thread's column of the output
            if (col < T.ncol) {
                y = S.Y + __ldg(S.yoff + T.col + col) + T.row0;
                c = __ldg(S.cx + __ldg(S.xgran + T.col + col));
            }
            const bool aligned = (reinterpret_cast<uintptr_t>(y) & 15) == 0;
            if (!warp_wait(&acc_full[a], (it >> 1) & 1, failed, wait_ns)) {
                *failed = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t src = tmem + ((uint32_t)(qw * 32) << 16) + (uint32_t)(a * 256);
            // rows parked at once: the tile's, or half of them (long pieces: a bulk reduction
            // costs 18 clocks of the SM and 8 per 128 bytes)
            const int hc = T.n <= 2 * HCH ? T.n >> 1 : ((T.n >> 2) + 7) & ~7;
            for (int r0 = 0; 2 * r0 < T.n; r0 += hc) {
                asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");  // `park` has been read
#pragma unroll
                for (int h = 0; h < HCH; h += 8) {
                    if (h < hc && 2 * (r0 + h) < T.n) {  // n and 2 hc are multiples of 16
                        uint32_t v[16];
                        asm volatile(
                            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
                            "%15}, [%16];\n"
                            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                              "=r"(v[14]), "=r"(v[15])
                            : "r"(src + (uint32_t)(2 * (r0 + h)))
                            : "memory");
                        float f[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) f[i] = r0 + h + i < T.rows ? __ldg(T.ra + r0 + h + i) : 0.f;
                        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                        for (int e = 0; e < 8; e += 2)
                            *reinterpret_cast<float4*>(park + h + e) = make_float4(
                                __uint_as_float(v[2 * e]) * f[e] * c, __uint_as_float(v[2 * e + 1]) * f[e] * c,
                                __uint_as_float(v[2 * e + 2]) * f[e + 1] * c, __uint_as_float(v[2 * e + 3]) * f[e + 1] * c);
                    }
                }
                if (2 * (r0 + hc) >= T.n) {  // last chunk read: accumulator back to the MMA issuer
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[a]);
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                const int n = min(hc, T.rows - r0);
                if (y && n > 0) {
                    const int bulk = aligned ? n & ~1 : 0;  // whole 16-byte pieces
                    if (bulk)
                        asm volatile(
                            "cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;\n" ::"l"(y + r0),
                            "r"(smem_u32(park)), "r"(bulk * 8)
                            : "memory");
                    for (int i = bulk; i < n; ++i) atomicAdd(y + r0 + i, park[i]);
                }
                asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
            }
            ++it;
        }
        asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    if (*failed && tid == 0) {
        // bounded drain of operator copies still in flight, then report
        const unsigned long long t0 = gtimer();
        while (gtimer() - t0 < 200000ull) __nanosleep(1000);
        atomicExch(err, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
}

static int g_h16_sms = 0;

void h16_init() {
    cudaFuncSetAttribute(h16_gemm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, H_SMEM);
    cudaFuncSetAttribute(h16_gemm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, H_SMEM);
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_h16_sms, cudaDevAttrMultiProcessorCount, dev);
}

void launch_h16_gemm(const HSub* subs, const int* prefix, int nsub, int ntiles, const int* active, int* err,
                     cudaStream_t s, const HSub& one, const int* order, unsigned long long wait_ns, int withhold) {
    if (ntiles == 0) return;
    if (wait_ns == 0) wait_ns = U_WAIT_NS;
    const int sms = g_h16_sms > 0 ? g_h16_sms : 148;
    const int grid = ntiles < sms ? ntiles : sms;
    if (nsub == 1)
        h16_gemm_kernel<false><<<grid, HTHREADS, H_SMEM, s>>>(one, subs, prefix, nsub, ntiles, nullptr, active, err, wait_ns,
                                                                 withhold);
    else
        h16_gemm_kernel<true><<<grid, HTHREADS, H_SMEM, s>>>(HSub{}, subs, prefix, nsub, ntiles, order, active, err, wait_ns,
                                                                withhold);
}

}  // namespace ddfmm
