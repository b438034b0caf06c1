// FP64 complex GEMM on the integer tensor cores (tcgen05 kind::i8).
//
// Problem (as in zgemm_kernel): Y[:, c] += A X[:, c] for gathered columns c, A
// an m x k complex operator.  The FP64 tensor path peaks at 37 TF/s; the int8
// path does 34 exact integer products per FP64 product at over 100 times that
// rate.  Every column (and every operator row) is written as
//     x_j = 2^(ex - 55) q_j,   q_j = sum_{i=0}^{6} d_i 256^(6-i),  d_i in [-128, 127],
// 2^ex above the vector's largest component: 55 bits below it (54 where its mantissa
// is above 1.988), a quarter of the largest FP64 entry's last place.  With X's digits d and A's
// digits e, a product of two numbers is sum_{i,j} d_i e_j 256^(12-i-j); the terms
// i + j <= 7 are kept (34 of 49; the dropped ones are below 2^-58 of the largest
// product).  Those of one diagonal i + j are summed over k by the tensor core in
// int32 without any rounding, the eight diagonals joined in int64 and rounded to
// FP64 twice per output, so the sums over k carry no rounding error at all.
//
// 55 bits below the largest component are worth as many of each product only where
// the components are of one size.  Outgoing vectors' are not: w stands for the
// equivalent densities E1 w, of one size, and E1 = inv(R1) of a pivoted QR has columns that
// grow by up to 10^8.  The sizes 1 / max |E1 column j| are a class's profile: component j is scaled
// by a power of two that evens it out before it becomes digits, column j of an operator by the
// inverse.  (They are within 0.75-1.25 of the row maxima of the M2M operators into a class, and
// come with the operator files: no session's geometry shows in them.)  Against long-double products, on
// the operators and vectors of evals (spheres, ellipsoids and clusters, K = 8 .. 32, both
// kernels, P = 4, 6, 8, four kinds of densities), the relative 2-norm error is 5e-17 to
// 7e-16 by pass, the three-MMA FP64 form's 3e-16 to 1.6e-15 and larger in each of them; M2L
// products without the scaling were off by 4e-14, 5e-12 and 1e-10 at P = 4, 6, 8.
//
// One tile is 128 gathered columns (the MMA's M, one TMEM lane each) x up to 56
// complex operator rows; operator row i becomes the int8 rows [Ar, -Ai] and
// [Ai, Ar] (N = 2 rows), K = 2k interleaved real and imaginary digits.  int32
// accumulators of eight diagonals would need 8 N of the 512 TMEM columns, so a
// tile runs its K loop twice: diagonals 4 .. 7 (24 MMAs per 32-wide K block,
// 4 N <= 448 columns; drained to one FP64 per output), then 0 .. 3 (10 MMAs, of
// which only the first four planes are loaded).
//
// Operands sit in shared memory K-major in the 32-byte swizzled layout, one
// plane per digit.  Digits come from memory: the operator's are packed at setup
// in the order a K block is consumed (one bulk copy per block), a vector's are
// written once by i8_slice_kernel as 224-byte granules (16 complex numbers x 7
// digit planes) and gathered by every column that uses it with 16-byte
// cp.async (eight lanes fill four 32-byte rows: all banks once).
//
// Persistent, one 512-thread block per SM.  Warp groups (registers moved from
// the first two to the last two):
//   0     operands: warps 0 .. 2 fill ring slot 0 .. 2, the operator block by one
//         bulk copy, the columns by cp.async
//   1     warp 4: MMA issue, one thread
//   2, 3  epilogue: warp w on TMEM lanes 32 (w % 4) .., group 2 on the tile's
//         first half of the rows, group 3 on the second.  After the second K
//         loop a thread holds its column's outputs as FP64 in registers, hands
//         the accumulators back, then scales and parks 14 rows at a time in
//         shared memory and adds each column's piece with one bulk reduction
//         (warp-wide FP64 atomics from the parked rows took twice as long: their
//         shared loads queue behind the tensor core's operand reads).
// Measured (m 100, k 152, 491,520 gathered columns): 1.02 ms, 59 TF/s of complex
// products against 28 for zgemm_kernel; 105 clocks an MMA, of which 60 are the
// operand reads (4 KB + 32 N bytes at 128 a clock; the MMA itself needs 56), 19
// the slots' fill, 11 the drain of the accumulators.
// Every mbarrier wait is bounded as in umma_cgemm_kernel (1 s, or until another
// role failed); a block that gives up drains its copies, frees its TMEM and
// sets *err.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdint>
#include <stdexcept>

#include "kernels.cuh"
#include "umma.cuh"

namespace ddfmm {

namespace {
constexpr int IS = I8_DIGITS;                 // digit planes
constexpr int IM = 128;                       // gathered columns per tile
constexpr int INMAX = 2 * I8_TILE_ROWS;       // int8 operator rows per tile
constexpr int ISTAGES = 3;                    // ring depth
constexpr int I_X_PLANE = IM * 32;            // bytes of one digit plane of a column block
constexpr int I_X_BYTES = IS * I_X_PLANE;
constexpr int I_B_BYTES = IS * INMAX * 32;
constexpr int I_STAGE_BYTES = I_X_BYTES + I_B_BYTES;
constexpr int IPR = 14;                       // complex rows parked per column
constexpr int IPS = IPR * 16 + 16;            // bytes per parked column: 16-byte stores of 8 lanes hit all banks
constexpr int I_PARK_WARP = 32 * IPS;
constexpr int I_SMEM = ISTAGES * I_STAGE_BYTES + 8 * I_PARK_WARP + 1024;
static_assert(I_SMEM + 1024 <= 232448, "shared memory per block");
constexpr int ITHREADS = 512;
constexpr int ICH = 8;                        // accumulator columns per TMEM load
constexpr int ICHUNKS = INMAX / 2 / ICH;      // chunks of a warp's half tile
static_assert(I_STAGE_BYTES % 256 == 0 && INMAX % 16 == 0 && INMAX <= 128, "swizzle atoms");

// byte offset of byte b (0 .. 31) of row r in a 32-byte swizzled K-major plane:
// 8-row groups of 256 bytes, the row's two 16-byte halves exchanged in rows 4 .. 7
__host__ __device__ __forceinline__ int i8_off(int r, int b) { return r * 32 + ((((b >> 4) ^ ((r >> 2) & 1)) << 4) | (b & 15)); }

// K-major operand descriptor, 32-byte swizzle (layout type 6), 8-row groups 256
// bytes apart: the low word holds the address, the high word is constant
__device__ __forceinline__ uint32_t i8_desc(uint32_t saddr) { return ((saddr >> 4) & 0x3FFF) | (1u << 16); }
constexpr uint32_t I_DESC_HI = (256 >> 4) | (1u << 14) | (6u << 29);
// D s32 (bits 4-5 = 2), A and B s8 (bits 7-9, 10-12 = 1), N >> 3 at 17, M >> 4 at 24
__device__ constexpr uint32_t i8_idesc(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(IM >> 4) << 24);
}
__device__ __forceinline__ void i8_mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %6};\n\tmov.b64 db, {%2, %6};\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %3, {%5, %5, %5, %5}, p;\n\t}\n" ::"r"(d),
        "r"(a), "r"(b), "r"(idesc), "r"(acc), "r"(0u), "r"(I_DESC_HI)
        : "memory");
}
// The MMA issuer's place in the ring: slot, its parity, and whether the slot is
// already known to be full.
struct I8Ring {
    uint32_t slot, parity, ready;
};

// One K loop of a tile: diagonals 4 .. 7 (PH 0) or 0 .. 3 (PH 1), per K block a
// chain of plane pairs i + j = d on accumulator d % 4.  One thread issues
// everything and the tensor core's queue is short, so what it does between two
// MMAs shows: N is a template argument (every address is the slot's plus a
// constant), slot and parity are counted rather than divided out, and the next
// slot's barrier -- whose answer takes some 250 clocks beside the operand reads --
// is asked before the block's last MMAs.
template <int N, int PH>
__device__ __forceinline__ bool i8_phase(uint32_t tmem, uint32_t dx0, int nkb, I8Ring& R, uint64_t* full, uint64_t* empty,
                                         uint64_t* acc_full, volatile int* failed, unsigned long long wait_ns) {
    for (int kb = 0; kb < nkb; ++kb) {
        if (!R.ready && !mbar_wait(full + R.slot, R.parity, failed, wait_ns)) return false;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t dx = dx0 + R.slot * (I_STAGE_BYTES >> 4), db = dx + (I_X_BYTES >> 4);
        uint64_t* const done = empty + R.slot;
        const bool wrap = R.slot == ISTAGES - 1;
        R.slot = wrap ? 0 : R.slot + 1;
        R.parity ^= wrap;
#pragma unroll
        for (int d = PH ? 0 : 4; d < (PH ? 4 : 8); ++d) {
            const int i0 = d < IS ? 0 : d - IS + 1;
            if (d == (PH ? 2 : 7)) R.ready = mbar_peek(full + R.slot, R.parity);
#pragma unroll
            for (int i = i0; i <= d - i0; ++i)
                i8_mma(tmem + (uint32_t)((d & 3) * N), dx + i * (I_X_PLANE >> 4), db + (d - i) * (N * 2), i8_idesc(N),
                       i > i0 ? 1u : (uint32_t)kb);
        }
        umma_commit(done);
    }
    umma_commit(acc_full);
    return true;
}

// ---------------------------------------------------------------- digits
// The seven balanced base-256 digits of q, |q| <= 0.996 2^55: adding 128 to every
// digit place makes them the bytes of one sum; flipping each byte's top bit
// takes the 128 off again.  Byte i of the result is digit 6 - i.
constexpr unsigned long long I_BIAS = 0x0080808080808080ull;
__device__ __forceinline__ unsigned long long i8_digits(long long q) { return ((unsigned long long)q + I_BIAS) ^ I_BIAS; }

// Scale of a vector (operator row) whose largest component has the high word `top` (sign
// off): s = 2^(55 - ex), which makes it an integer below 0.9942 2^55 (seven balanced digits
// reach 0.9960 2^55), and out = 2^(ex - 1).  A vector with nothing above 2^-823 is brought up by
// 2^200 first (low), so subnormals keep their bits.  NaN when the vector holds an infinity or
// a NaN.
constexpr int I_UP = 200;
constexpr uint32_t I_LOW = 200u << 20;  // top below it: low
struct I8Scale {
    double s, out;
};
__device__ __forceinline__ double i8_pow2(int e) { return __longlong_as_double((long long)(1023 + e) << 52); }
__device__ __forceinline__ I8Scale i8_scale(uint32_t top, bool low) {
    I8Scale r;
    const int be = (int)(top >> 20);
    if (be == 0x7ff) {
        r.s = 0.0;
        r.out = __longlong_as_double(0x7ff8000000000000ll);
        return r;
    }
    if (top == 0) {  // zero
        r.s = r.out = 1.0;
        return r;
    }
    const int b1 = be + ((top & 0xfffffu) >= 0xfd000u);  // ex + 1022
    r.s = __longlong_as_double((long long)(2100 - b1) << 52);
    const int bo = b1 - (low ? I_UP : 0);
    r.out = bo >= 1 ? __longlong_as_double((long long)bo << 52) : __longlong_as_double(bo >= -51 ? 1ll << (bo + 51) : 0ll);
    return r;
}
__device__ __forceinline__ long long i8_quant(double x, const I8Scale& S) { return __double2ll_rn(x * S.s); }
__device__ __forceinline__ uint32_t top_word(double x) { return (uint32_t)__double2hiint(x) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t top_of(double2 v) { return max(top_word(v.x), top_word(v.y)); }

// eight digit bytes, place p of eight numbers: byte p of w[0..7]
__device__ __forceinline__ uint2 gather_bytes(const unsigned long long (&w)[8], int p) {
    uint32_t r[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = p < 4 ? (uint32_t)w[4 * h + j] : (uint32_t)(w[4 * h + j] >> 32);
        const int b = p & 3;
        const uint32_t lo = __byte_perm(v[0], v[1], b | ((b + 4) << 4));
        const uint32_t hi = __byte_perm(v[2], v[3], b | ((b + 4) << 4));
        r[h] = __byte_perm(lo, hi, 0x5410);
    }
    return make_uint2(r[0], r[1]);
}
}  // namespace

// Digits of vectors: one warp per vector, four lanes per granule of 16 complex
// numbers (each lane 4 of them: 8 bytes in each of the 7 planes).  Bound by
// HBM: 16 bytes read and 14 written per complex number; the profiles come from L2.
// PROF: the vectors have profiles (a launch's all do or none does).
template <bool PROF>
__global__ void __launch_bounds__(256) i8_slice_kernel(const I8Vec* __restrict__ vecs, int n,
                                                       const double2* __restrict__ X, char* __restrict__ X8,
                                                       double* __restrict__ cx, const I8Profiles T) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= n) return;
    const I8Vec V = vecs[w];
    const double2* x = X + V.src;
    const unsigned char* prof = PROF ? T.prof + (size_t)(V.profile - 1) * T.stride : nullptr;
    double2 v[4];
    auto load = [&](int j0, int up) {
        uint32_t b = 0x7f7f7f7fu;
        if (PROF && j0 < V.len) b = __ldg(reinterpret_cast<const uint32_t*>(prof + j0));
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = j0 + j < V.len ? x[j0 + j] : make_double2(0.0, 0.0);
        if (PROF || up) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double f = __hiloint2double((int)(((b >> (8 * j)) & 255u) + (uint32_t)(896 + up)) << 20, 0);
                v[j] = make_double2(v[j].x * f, v[j].y * f);
            }
        }
    };
    int up = 0;
    uint32_t top;  // of the whole vector
    while (true) {
        top = 0;
        for (int j0 = 0; j0 < V.len; j0 += 128) {
            load(j0 + lane * 4, up);
#pragma unroll
            for (int i = 0; i < 4; ++i) top = max(top, top_of(v[i]));
        }
        top = __reduce_max_sync(0xffffffffu, top);
        if (top >= I_LOW || up) break;
        up = I_UP;
    }
    const I8Scale S = i8_scale(top, up > 0);
    if (lane == 0) cx[V.gran] = S.out;
    for (int j0 = 0; j0 < V.len; j0 += 128) {
        if (V.len > 128) load(j0 + lane * 4, up);
        const int g = (j0 >> 4) + (lane >> 2);
        if (g * 16 < V.len) {
            unsigned long long q[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                q[2 * j] = i8_digits(i8_quant(v[j].x, S));
                q[2 * j + 1] = i8_digits(i8_quant(v[j].y, S));
            }
            char* o = X8 + (size_t)(V.gran + g) * I8_GRANULE + (lane & 3) * 8;
#pragma unroll
            for (int p = 0; p < IS; ++p) *reinterpret_cast<uint2*>(o + p * 32) = gather_bytes(q, IS - 1 - p);
        }
    }
}

void launch_i8_slice(const I8Vec* vecs, int n, const double2* X, char* X8, double* cx, const I8Profiles& T,
                     cudaStream_t s) {
    if (n <= 0) return;
    auto kernel = T.prof ? i8_slice_kernel<true> : i8_slice_kernel<false>;
    kernel<<<(unsigned)(((size_t)n * 32 + 255) / 256), 256, 0, s>>>(vecs, n, X, X8, cx, T);
}

// 127 - (e_j - e0), e_j the exponent of size j and e0 the smallest of them but no less than
// the largest one - 60; sizes that are no positive number count as the smallest.  (Vectors are scaled
// down only: none overflows.)
std::vector<unsigned char> i8_profile(const double* size, int n, int stride) {
    std::vector<unsigned char> row(stride, 127);
    auto expo = [](double v) { return v > 0.0 && v <= DBL_MAX ? std::ilogb(v) : INT_MIN; };
    int lo = INT_MAX, hi = INT_MIN;
    for (int j = 0; j < n; ++j) {
        const int e = expo(size[j]);
        if (e == INT_MIN) continue;
        lo = std::min(lo, e);
        hi = std::max(hi, e);
    }
    const int e0 = hi == INT_MIN ? 0 : std::max(lo, hi - 60);
    for (int j = 0; j < n; ++j) row[j] = (unsigned char)(127 - (std::max(expo(size[j]), e0) - e0));
    return row;
}

// Operator digits (setup only): block (row tile, job).  Row scales first, then
// 4 complex numbers of a row at a time into K block order: block kb of a row
// tile holds plane p of its 2 rows_t int8 rows at p * rows_t * 64.
__global__ void __launch_bounds__(256) i8_pack_kernel(const I8PackJob* __restrict__ jobs, int njobs) {
    __shared__ uint32_t tops[4][64];
    __shared__ I8Scale sc[64];
    __shared__ bool low[64];
    const int tid = threadIdx.x;
    for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
        const I8PackJob J = jobs[j];
        const int row0 = blockIdx.x * J.rows_t;
        if (row0 >= J.m) continue;  // uniform over the block
        // column k as the vectors' profile leaves it, brought up where the row is low
        auto entry = [&](int r, int k, bool up) {
            const double2 a = J.A[(size_t)k * J.lda + row0 + r];
            const double f = i8_pow2((J.prof ? 127 - J.prof[k] : 0) + (up ? I_UP : 0));
            return make_double2(a.x * f, a.y * f);
        };
        for (int up = 0; up < 2; ++up) {
            __syncthreads();
            const int r = tid & 63;
            uint32_t top = 0;
            if (r < J.rows_t && row0 + r < J.m && (up == 0 || low[r]))
                for (int k = tid >> 6; k < J.k; k += 4) top = max(top, top_of(entry(r, k, up)));
            tops[tid >> 6][r] = top;
            __syncthreads();
            if (tid < J.rows_t) {
                const uint32_t t = max(max(tops[0][tid], tops[1][tid]), max(tops[2][tid], tops[3][tid]));
                if (up == 0) low[tid] = t < I_LOW;
                if (up == 0 || low[tid]) sc[tid] = i8_scale(t, up);
            }
        }
        // the output scale of a row: 2^(ea - 1) 2^-36 (the epilogue's sums count units
        // of diagonal 3: 256^9 2^(ex - 55) 2^(ea - 55) = 2^(ex + ea - 38), and cx = 2^(ex - 1))
        if (tid < J.rows_t && row0 + tid < J.m) J.ra[row0 + tid] = sc[tid].out * 0x1p-36;
        __syncthreads();
        const int nq = J.nkb * 4, N = 2 * J.rows_t;
        char* dst = J.dst + (size_t)blockIdx.x * J.nkb * IS * N * 32;
        for (int e = tid; e < nq * J.rows_t; e += 256) {
            const int r = e % J.rows_t, q4 = e / J.rows_t, k0 = q4 * 4;
            const I8Scale S = sc[r];
            unsigned long long w0[8], w1[8];  // rows [Ar, -Ai] and [Ai, Ar]
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool ok = row0 + r < J.m && k0 + i < J.k;
                const double2 a = ok ? entry(r, k0 + i, low[r]) : make_double2(0.0, 0.0);
                const long long qr = i8_quant(a.x, S), qi = i8_quant(a.y, S);
                w0[2 * i] = w1[2 * i + 1] = i8_digits(qr);
                w0[2 * i + 1] = i8_digits(-qi);
                w1[2 * i] = i8_digits(qi);
            }
            char* blk = dst + (size_t)(q4 >> 2) * IS * N * 32;
            const int b = (q4 & 3) * 8;
#pragma unroll
            for (int p = 0; p < IS; ++p) {
                *reinterpret_cast<uint2*>(blk + p * N * 32 + i8_off(2 * r, b)) = gather_bytes(w0, IS - 1 - p);
                *reinterpret_cast<uint2*>(blk + p * N * 32 + i8_off(2 * r + 1, b)) = gather_bytes(w1, IS - 1 - p);
            }
        }
    }
}

int i8_row_tiles(int m) { return (m + I8_TILE_ROWS - 1) / I8_TILE_ROWS; }
int i8_tile_rows(int m) { return ((m + i8_row_tiles(m) - 1) / i8_row_tiles(m) + 7) / 8 * 8; }
size_t i8_packed_bytes(int m, int k) {
    return (size_t)i8_row_tiles(m) * ((k + 15) / 16) * IS * 2 * i8_tile_rows(m) * 32;
}

void i8_tiles(const char* B, const double* ra, int m, int k, int col0, int ncol, std::vector<I8Tile>& out) {
    const int nrt = i8_row_tiles(m), rt = i8_tile_rows(m), nkb = (k + 15) / 16;
    for (int c = 0; c < ncol; c += IM)
        for (int r = 0; r < nrt; ++r)  // adjacent: the row tiles of a column block read its digits from L2 together
            out.push_back(I8Tile{B + (size_t)r * nkb * IS * 2 * rt * 32, ra + r * rt, col0 + c, r * rt,
                                 (unsigned short)(ncol - c < IM ? ncol - c : IM),
                                 (unsigned short)(m - r * rt < rt ? m - r * rt : rt), (unsigned short)(2 * rt),
                                 (unsigned short)nkb});
}

void launch_i8_pack(const I8PackJob* jobs, int njobs, int max_tiles, cudaStream_t s) {
    if (njobs > 0) i8_pack_kernel<<<dim3(max_tiles, njobs < 32768 ? njobs : 32768), 256, 0, s>>>(jobs, njobs);
}

// ---------------------------------------------------------------- GEMM
namespace {
__device__ __forceinline__ I8Tile i8_tile(const I8Sub& S, int ti) {
    union {
        int4 w[2];
        I8Tile t;
    } u;
    static_assert(sizeof(I8Tile) == 32, "two 16-byte loads");
    const int4* p = reinterpret_cast<const int4*>(S.tiles + (ti < S.ntiles ? ti : 0));
    u.w[0] = __ldg(p);
    u.w[1] = __ldg(p + 1);
    return u.t;
}
// four diagonals as one FP64 number, in units of the last, exactly (below 2^51)
__device__ __forceinline__ double join4(int a, int b, int c, int d) {
    return (double)(((long long)a * 256 + b) * 65536 + ((long long)c * 256 + d));
}
// a warp's copies of NP digit planes of K block kb: 128 columns, zero where absent
template <int NP>
__device__ __forceinline__ void i8_copy(uint32_t dst, const int (&gran)[8], const char* X8, int kb) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const char* a = X8 + (gran[j] < 0 ? 0 : (size_t)(gran[j] + kb) * I8_GRANULE);
        const int n = gran[j] < 0 ? 0 : 16;
#pragma unroll
        for (int p = 0; p < NP; ++p)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst + p * I_X_PLANE + j * 512),
                         "l"(a + p * 32), "r"(n));
    }
}
template <int R>
__device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(R)); }
__device__ __forceinline__ void tmem_ld8(uint32_t addr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr)
                 : "memory");
}
// eight columns of four accumulators n columns apart
__device__ __forceinline__ void tmem_ld4(uint32_t addr, int n, int (&d)[4][8]) {
#pragma unroll
    for (int a = 0; a < 4; ++a) tmem_ld8(addr + (uint32_t)(a * n), d[a]);
}
}  // namespace

__global__ void __launch_bounds__(ITHREADS, 1) i8_gemm_kernel(const I8Sub S, int* err, unsigned long long wait_ns, int withhold) {
    extern __shared__ __align__(1024) unsigned char ism_raw[];
    __shared__ __align__(8) uint64_t full[ISTAGES], empty[ISTAGES], acc_full, acc_empty, drained;
    __shared__ uint32_t tmem_base;
    __shared__ int failed_s;
    volatile int* failed = &failed_s;
    unsigned char* sm = (unsigned char*)(((uintptr_t)ism_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        failed_s = 0;
        for (int s = 0; s < ISTAGES; ++s) {
            mbar_init(&full[s], 2);        // the operator copy's bytes, the gathered columns
            mbar_init(&empty[s], 1);       // tcgen05.commit
        }
        mbar_init(&acc_full, 1);     // tcgen05.commit
        mbar_init(&drained, 1);      // tcgen05.commit, after a failure
        mbar_init(&acc_empty, 8);    // epilogue warps
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_base;

    if (warp < 4) {
        reg_dec<48>();
        // ------------------------------------------------ operands
        // warp w owns ring slot w, so all slots are filled at once and none waits for the
        // next one to become free (one owner a slot: a warp that could run a second
        // phase ahead would read the slot's empty barrier by the wrong parity).  Lane l
        // copies half l % 2 of the 32-byte rows of columns l / 2 + 16 j
        const int hf = lane & 1;
        const uint32_t dst = smem_u32(sm) + i8_off(lane >> 1, hf * 16);
        int g = 0;
        bool ok = true;
        I8Tile Tn = i8_tile(S, blockIdx.x);
        for (int ti = blockIdx.x; ti < S.ntiles && ok && warp < ISTAGES; ti += gridDim.x) {
            const I8Tile T = Tn;
            Tn = i8_tile(S, ti + gridDim.x);
            int gran[8];  // the columns' first granules, -1 past the last one
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int c = (lane >> 1) + 16 * j;
                gran[j] = c < T.ncol ? __ldg(S.xgran + T.col + c) : -1;
            }
            for (int ph = 0; ph < 2 && ok; ++ph)
                for (int kb = 0; kb < T.nkb; ++kb, ++g) {
                    const int s = g % ISTAGES;
                    if (s != warp) continue;
                    if (g >= ISTAGES && !warp_wait(&empty[s], ((g / ISTAGES) - 1) & 1, failed, wait_ns)) {
                        *failed = 1;
                        ok = false;
                        break;
                    }
                    if (lane == 0 && !(withhold && blockIdx.x == 0)) {  // withheld: full[s] never completes
                        const uint32_t bytes = (uint32_t)(ph == 0 ? IS : 4) * T.n * 32;
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;\n" ::"r"(bytes),
                                     "r"(smem_u32(&full[s]))
                                     : "memory");
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                                smem_u32(sm + s * I_STAGE_BYTES + I_X_BYTES)),
                            "l"(T.B + (size_t)kb * IS * T.n * 32), "r"(bytes), "r"(smem_u32(&full[s]))
                            : "memory");
                    }
                    const uint32_t so = dst + s * I_STAGE_BYTES;
                    if (ph == 0)
                        i8_copy<IS>(so, gran, S.X8 + hf * 16, kb);
                    else
                        i8_copy<4>(so, gran, S.X8 + hf * 16, kb);
                    asm volatile("cp.async.wait_all;\n" ::: "memory");
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[s]);
                }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    } else if (warp < 8) {
        reg_dec<48>();
        if (warp == 4 && lane == 0) {
            // -------------------------------------------- MMA issue
            I8Ring R{0, 0, 0};
            const uint32_t dx0 = i8_desc(smem_u32(sm));
            uint32_t parity = 1;  // of acc_empty; the first wait passes
            bool ok = true;
            I8Tile T = i8_tile(S, blockIdx.x);
            for (int ti = blockIdx.x; ti < S.ntiles && ok; ti += gridDim.x) {
                const int N = T.n, nkb = T.nkb;
                T = i8_tile(S, ti + gridDim.x);  // read while this tile's MMAs run
#define DDFMM_I8_PHASE(n, ph) i8_phase<n, ph>(tmem, dx0, nkb, R, full, empty, &acc_full, failed, wait_ns)
#define DDFMM_I8_CASE(n) \
    case n: ok = ph == 0 ? DDFMM_I8_PHASE(n, 0) : DDFMM_I8_PHASE(n, 1); break;
                for (int ph = 0; ph < 2 && ok; ++ph) {
                    ok = mbar_wait(&acc_empty, parity, failed, wait_ns);
                    parity ^= 1;
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    switch (N) {
                        DDFMM_I8_CASE(112)
                        DDFMM_I8_CASE(96)
                        DDFMM_I8_CASE(80)
                        DDFMM_I8_CASE(64)
                        DDFMM_I8_CASE(48)
                        DDFMM_I8_CASE(32)
                        DDFMM_I8_CASE(16)
                    }
                }
#undef DDFMM_I8_CASE
#undef DDFMM_I8_PHASE
            }
            if (!ok) {  // let the MMAs already issued finish before TMEM is freed
                *failed = 1;
                umma_commit(&drained);
                mbar_wait(&drained, 0, nullptr, wait_ns);
            }
        }
    } else {
        reg_inc<208>();
        // ------------------------------------------------ epilogue
        const int ew = warp - 8, qw = warp & 3, half = ew >> 2;
        unsigned char* park = sm + ISTAGES * I_STAGE_BYTES + ew * I_PARK_WARP;
        unsigned char* mine = park + lane * IPS;
        int q = 0;
        // a tile's column (granule, output element) and scale are read one tile ahead
        I8Tile T = i8_tile(S, blockIdx.x);
        const int col = qw * 32 + lane;
        double c = 0.0;
        long long yo = 0;
        if (col < T.ncol) {
            c = __ldg(S.cx + __ldg(S.xgran + T.col + col));
            yo = __ldg(S.yoff + T.col + col);
        }
        for (int ti = blockIdx.x; ti < S.ntiles; ti += gridDim.x) {
            const I8Tile Tn = i8_tile(S, ti + gridDim.x);
            const int hN = T.n >> 1;  // this warp's accumulator columns: half hN .. (half + 1) hN
            double2* y = col < T.ncol ? S.Y + yo + T.row0 + half * (hN >> 1) : nullptr;
            const uint32_t base = tmem + ((uint32_t)(qw * 32) << 16) + (uint32_t)(half * hN);
            double v[ICHUNKS * ICH];
            if (!warp_wait(&acc_full, q & 1, failed, wait_ns)) {
                *failed = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            // diagonals 4 .. 7 (at most 50 bits), in units of diagonal 7; the loads of a
            // chunk are in flight while the previous one is joined
            int d[2][4][8];
            tmem_ld4(base, T.n, d[0]);
#pragma unroll
            for (int ch = 0; ch < ICHUNKS; ++ch)
                if (ch * ICH < hN) {
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    if (ch + 1 < ICHUNKS && (ch + 1) * ICH < hN) tmem_ld4(base + (ch + 1) * ICH, T.n, d[(ch + 1) & 1]);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        v[ch * ICH + e] = join4(d[ch & 1][0][e], d[ch & 1][1][e], d[ch & 1][2][e], d[ch & 1][3][e]);
                }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty);
            ++q;
            if (!warp_wait(&acc_full, q & 1, failed, wait_ns)) {
                *failed = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            // diagonals 0 .. 3 in units of diagonal 3, then both parts in one rounding
            tmem_ld4(base, T.n, d[0]);
#pragma unroll
            for (int ch = 0; ch < ICHUNKS; ++ch)
                if (ch * ICH < hN) {
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    if (ch + 1 < ICHUNKS && (ch + 1) * ICH < hN) tmem_ld4(base + (ch + 1) * ICH, T.n, d[(ch + 1) & 1]);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        v[ch * ICH + e] = fma(v[ch * ICH + e], 0x1p-32,
                                              join4(d[ch & 1][0][e], d[ch & 1][1][e], d[ch & 1][2][e], d[ch & 1][3][e]));
                }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty);
            ++q;
            int gn = 0;
            if (col < Tn.ncol) {
                gn = __ldg(S.xgran + Tn.col + col);
                yo = __ldg(S.yoff + Tn.col + col);
            }
            // scale, park, add: rows of this half tile, IPR at a time
            const int r0 = half * (hN >> 1), nr = min(hN >> 1, (int)T.rows - r0);
            const double* ra = T.ra + r0;
#pragma unroll
            for (int b = 0; b < ICHUNKS * ICH / 2; b += IPR) {
                if (b < nr) {
                    asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");  // this lane's last piece was read
#pragma unroll
                    for (int i = 0; i < IPR; ++i)
                        if (b + i < ICHUNKS * ICH / 2 && b + i < nr) {
                            const double f = __ldg(ra + b + i);
                            *reinterpret_cast<double2*>(mine + i * 16) =
                                make_double2(v[2 * (b + i)] * f * c, v[2 * (b + i) + 1] * f * c);
                        }
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    if (y)
                        asm volatile(
                            "cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;\n" ::"l"(y + b),
                            "r"(smem_u32(mine)), "r"(min(IPR, nr - b) * 16)
                            : "memory");
                    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                }
            }
            T = Tn;
            if (col < T.ncol) c = __ldg(S.cx + gn);
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

static int g_i8_sms = 0;

void i8_init() {
    cudaFuncSetAttribute(i8_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, I_SMEM);
    // the register split (2 x 48 + 2 x 208 a thread) needs what the block was launched with
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, i8_gemm_kernel) == cudaSuccess && a.numRegs * ITHREADS < 128 * (2 * 48 + 2 * 208))
        throw std::runtime_error("int8 GEMM kernel built with too few registers for its register split");
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_i8_sms, cudaDevAttrMultiProcessorCount, dev);
}

void launch_i8_gemm(const I8Sub& S, int* err, cudaStream_t s, unsigned long long wait_ns, int withhold) {
    if (S.ntiles == 0) return;
    const int sms = g_i8_sms > 0 ? g_i8_sms : 148;
    i8_gemm_kernel<<<S.ntiles < sms ? S.ntiles : sms, ITHREADS, I_SMEM, s>>>(S, err, wait_ns ? wait_ns : U_WAIT_NS, withhold);
}

}  // namespace ddfmm
