// Device kernels of the directional FMM eval and their launch descriptors.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <vector>

namespace ddfmm {

enum KernelType { KERNEL_HELM = 0, KERNEL_EXPR = 1 };  // include/kernel3d.hpp:24-27
enum GemmMode { GEMM_SET = 0, GEMM_ADD = 1, GEMM_ATOMIC = 2 };

// One shared operator A (m x k, column-major, leading dimension lda) applied
// to ncol gathered columns: y[yoff[c]..] (op)= A * x[xoff[c]..].
struct GemmProblem {
    const double2* A;
    int m, k, lda;
    int col0;  // first entry in the column arrays
    int ncol;
    const float* packed;  // tcgen05 form: an already packed copy of A (A may then be null)
    int profile;          // int8 and FP16 paths: 1 + the row of the profile table that scales its columns' vectors; 0: none
};
// A launch is a list of output tiles of up to GEMM_TILE_M rows x GEMM_TILE_N columns.
constexpr int GEMM_TILE_M = 64, GEMM_TILE_N = 64;
void gemm_init();
struct GemmTile {
    int prob;
    int row0;
    int col0;  // relative to the problem's first column
    int pad;
};

// Kernel-matrix generation job: out(i,j) = G(trg_i + ts, src_j + ss),
// trg/src are 3 x n point arrays (coordinate fastest), out column-major.
struct KmatJob {
    const double* trg;
    const double* src;
    double2* out;
    double ts[3];
    double ss[3];
    int m, k;
    long long elem0;  // prefix offset of this job's elements in the launch
};

// A set of points: p_k = scale * x[3k..3k+2] + shift.
struct PtSet {
    const double* x;
    double shift[3];
    double scale;
    int n;
};
// Point-interaction work item: out[t] += sum_s G(trg_t, src_s) den[s] over
// the source segments src_begin..src_end of the item.
struct PtItem {
    PtSet trg;
    double2* out;
    int src_begin, src_end;
};
struct PtSrc {
    PtSet src;
    const double2* den;
};

void launch_kmat(const KmatJob* jobs_dev, int njobs, long long total, int kernel, cudaStream_t s);
// Columns of a setup product: column c of the span's is X + bx + c sx and Y + cy + c sy.
struct ColumnSpan {
    long long first, bx, cy;  // first: the span's first column in the launch
    int sx, sy;
};
void launch_list_columns(const ColumnSpan* spans_dev, int nspans, long long ncols, long long* xoff, long long* yoff,
                         cudaStream_t s);
void launch_gemm(const GemmProblem* probs_dev, const GemmTile* tiles_dev, int ntiles,
                 const long long* xoff, const long long* yoff, const double2* X, double2* Y, int mode,
                 cudaStream_t s);
// Products with few columns: tiles of `rows` (64 or 128) operator rows x 8 columns; kmax: the
// launch's longest k, narrow_smem(kmax) <= NARROW_SMEM.
constexpr int NARROW_SMEM = 72 << 10;
constexpr size_t narrow_smem(int k) { return sizeof(double2) * 8 * ((size_t)(k + 7) / 8 * 8 + 4); }
// every operator's m and k are at most the largest skeleton rank (OperatorLib::validate) or surface
static_assert(narrow_smem(400) <= NARROW_SMEM, "shared memory of the longest column");
// Y[off[c] ..] = B (A X[off[c] ..]) for ncol columns: A r x m, B m x r, column-major and dense, m, r <= GEMM_PAIR_MAX
constexpr int GEMM_PAIR_MAX = 64;
struct GemmPair {
    const double2* A;
    const double2* B;
    int m, r, ncol;
    const long long* off;
    const double2* X;
    double2* Y;
};
void launch_gemm_pair(const GemmPair& P, cudaStream_t s);
void launch_gemm_narrow(const GemmProblem* probs_dev, const GemmTile* tiles_dev, int ntiles, const long long* xoff,
                        const long long* yoff, const double2* X, double2* Y, int mode, int kmax, int rows,
                        cudaStream_t s);
// tpi: the launch shape, chosen per step by the session's autotuner: 4, 8, 16 or
// 32 threads per item, each thread taking targets and walking the sources in
// global memory; or one warp per item with the item's sources staged in
// shared memory, lanes over targets (PT_WARP_TARGETS: 4 targets a lane;
// PT_WARP_TARGETS2: 2, fewer registers) or over sources with a warp-shuffle
// reduction per target (PT_WARP_SOURCES: 8 targets a pass; PT_WARP_SOURCES4: 4)
constexpr int PT_WARP_TARGETS = 1001, PT_WARP_SOURCES = 1002, PT_WARP_TARGETS2 = 1003, PT_WARP_SOURCES4 = 1004;
__host__ __device__ constexpr bool pt_warp_shape(int tpi) { return tpi >= PT_WARP_TARGETS && tpi <= PT_WARP_SOURCES4; }
void launch_pt(const PtItem* items_dev, int nitems, const PtSrc* srcs_dev, int kernel, cudaStream_t s, int tpi = 32);

// FFT-based low-frequency M2L on a G^3 grid (G = 2P), see kernels.cu.
struct VlistLevel {
    int G, P;
    int nE;                 // equivalent / check points per box
    const int* cube_idx;    // nE indices of the uep (== dcp) nodes in the P^3 corner cube [P, 2P)^3
    const double2* tns;     // 343 x G^3 FFT'd translation tensors (zero when near)
    const double2* twf;     // G forward twiddles exp(-2 pi i m / G)
    const double2* twb;     // G backward twiddles exp(+2 pi i m / G)
};
void vlist_init(int G);
// The forward and inverse transforms take one box per block and one thread per
// (ka, kb) line of the grid; their shared memory holds the twiddles (G P) and
// the three partial transforms (P^3, P^2 G, P G^2 elements of es bytes).
__host__ __device__ constexpr int vt_threads(int G) { return ((G * G + 31) / 32) * 32; }
size_t vt_smem(int G, size_t es);
void launch_vlist_forward(const VlistLevel& L, const int* boxes, int nbox, const double2* upeq,
                          double2* spec, cudaStream_t s);
// The V-list sums in Fourier space, by target parent: the target boxes of a
// level are grouped by their parent (the groups in Morton order of the
// parents); a group lists the union of its targets' V-list sources, each as
//   {spectrum row of the source, (tbase << 8) | mask}
// where bit c of mask says that the child at position c = 4a + 2b + c' of
// the parent (offset (a, b, c') from twice the parent's index) has the
// source in its V list, and tbase is the translation-tensor index of that
// pair for child position 0; child position c adds a + 7b + 49c'.
// tsp[t] (G^3 per target, rows in group order) receives the summed spectrum
// of target t, overwritten each eval.
constexpr int VGROUP_WARPS = 8;  // target parents per block of the sums
// Launches with fewer (group, 32-frequency chunk) pairs than this give a pair a
// whole block, its entries dealt to the 8 warps: a warp alone walks 40 to 190
// entries of two dependent loads each, and so few warps do not fill the SMs.
// Measured: K = 4, P = 4 (800 pairs) 86 -> 80 us a matvec, a K = 8 adaptive cluster
// (five levels) 681 -> 643 us, but K = 8, P = 4 (2900 pairs) 399 -> 409 us: the line
// lies at 12 warps an SM.
constexpr long long VGROUP_SPLIT = 148 * 12;
struct VlistGroups {
    const int* gptr;   // ngroups + 1: the source entries of each group
    const int2* gsrc;  // the source entries
    const int* gtrg;   // ngroups x 8: row of tsp of each child position, -1 where none
    int ngroups;
};
void launch_vlist_group(const VlistLevel& L, const VlistGroups& V, const double2* spec, double2* tsp,
                        cudaStream_t s);
// dnchk[trg[t]] += pruned inverse DFT of tsp[t] / G^3 at the corner-cube nodes
void launch_vlist_inverse(const VlistLevel& L, const int* trg, int ntrg, const double2* tsp, double2* dnchk,
                          cudaStream_t s);

// mixed-precision form (kernels_mixed.cu): complex FP32 data behind the same
// descriptors; GemmProblem::A, PtItem::out, PtSrc::den and VlistLevel::tns /
// twf / twb then point to float2 data.
// PRECISION_MIXED multiplies on tcgen05 (kernels_umma.cu); PRECISION_MIXED_MMA_SYNC
// is the same form with the warp-level mma.sync GEMM (cgemm_kernel), kept for comparison.
enum Precision { PRECISION_FP64 = 0, PRECISION_MIXED = 1, PRECISION_MIXED_MMA_SYNC = 2 };
void cgemm_init();
void launch_cgemm(const GemmProblem* probs_dev, const GemmTile* tiles_dev, int ntiles, const long long* xoff,
                  const long long* yoff, const void* X, void* Y, int mode, cudaStream_t s);

// Multi-instance launches of the mixed form.  A launch is a device array of
// per-instance sub-launches plus the prefix sums of their work items (nsub + 1
// entries); a sub-launch is skipped when `active` (indexed by `inst`) is given
// and holds 0.  A single session is a launch with one sub-launch.
struct PtSub {
    const PtItem* items;
    const PtSrc* srcs;
    int nitems;
    int kernel;  // KERNEL_HELM / KERNEL_EXPR
    int inst;
    int pad;
};
struct VfSub {  // V-list source spectra, one work item per source box
    VlistLevel L;
    const int* boxes;
    const float2* upeq;
    float2* spec;
    int nbox;
    int inst;
};
struct VaSub {  // V-list sums by target parent (VlistGroups), one work item per group
    VlistLevel L;
    const int* gptr;
    const int2* gsrc;
    const int* gtrg;
    const float2* spec;
    float2* tsp;
    int ngroups;
    int inst;
};
struct ViSub {  // V-list inverse transforms, one work item per target box
    VlistLevel L;
    const int* trg;
    const float2* tsp;
    float2* dnchk;
    int ntrg;
    int inst;
};
struct MoveSub {  // complex64 point data between point-id and leaf order
    const void* in;
    const int* perm;
    void* out;
    int n;
    int inst;
};
struct ZeroSub {
    void* p;
    long long n8;  // 8-byte words
    int inst;
    int pad;
};
void launch_pt32(const PtSub* subs, const int* prefix, int nsub, int nitems, const int* active, cudaStream_t s,
                 int tpi = 32);
void vlist32_init(int G);
// A launch with nsub == 1 passes its sub-launch as `one` (host copy, sent as
// a kernel parameter); `subs` / `prefix` are then not read.
void launch_vlist_forward32(const VfSub* subs, const int* prefix, int nsub, int nbox, int G, const int* active,
                            void* spec_override, cudaStream_t s, const VfSub* one);
// work items: groups (launch_vlist_group32) or targets (launch_vlist_inverse32)
void launch_vlist_group32(const VaSub* subs, const int* prefix, int nsub, int ngroups, int G, const int* active,
                          const void* spec_override, cudaStream_t s, const VaSub* one);
void launch_vlist_inverse32(const ViSub* subs, const int* prefix, int nsub, int ntrg, int G, const int* active,
                            cudaStream_t s, const ViSub* one);
void launch_move32(const MoveSub* subs, const int* prefix, int nsub, int n, const int* active, int scatter,
                   const int* err, cudaStream_t s);
void launch_zero(const ZeroSub* subs, const long long* prefix, int nsub, long long n8, const int* active,
                 cudaStream_t s);
void launch_gather32(const void* den, const int* perm, void* out, int n, int c64, cudaStream_t s);
void launch_scatter32(const void* in, const int* perm, void* val, int n, int c64, const int* err, cudaStream_t s);
void launch_to_c64(const double2* a, float2* b, long long n, cudaStream_t s);

// mixed-form low-frequency GEMM on tcgen05 (kernels_umma.cu): 128 gathered columns x up to
// 128 complex operator rows per tile, operator packed at setup as split TF32.
struct UmmaProblem {
    const float* B;      // packed operator (umma_pack_kernel layout)
    size_t tile_stride;  // floats between 128-row tiles of the packed operator
    int m, k, nkb;       // complex rows, complex columns, 16-wide real K blocks
    int col0, ncol;      // gathered columns, as in GemmProblem
};
struct UmmaTile {
    int prob;
    int rtile;  // 128-row tile of the operator
    int row0;   // = 128 * rtile
    int rows;   // complex rows of this tile (<= 128)
    int col0;   // relative to the problem's first column
    int pad;
};
struct UmmaSub {  // one instance's part of a multi-instance GEMM launch
    const UmmaProblem* probs;
    const UmmaTile* tiles;
    const long long* xoff;
    const long long* yoff;
    const float2* X;
    float2* Y;
    int ntiles;
    int mode;
    int inst;
    int pad;
};
struct UmmaPackJob {
    const float2* A;  // complex FP32 operator, column-major
    float* dst;
    size_t tile_stride;
    int m, k, lda, nkb;
};
void umma_init();
int umma_nkb(int k);
size_t umma_tile_stride(int k);
size_t umma_packed_floats(int m, int k);
void launch_umma_pack(const UmmaPackJob* jobs_dev, int njobs, cudaStream_t s);
// nsub == 1: `one` is that sub-launch (host copy, sent as a kernel parameter).
// wait_ns bounds every pipeline wait (0: 1 s); withhold != 0 is the failure-path
// test hook: block 0 issues no operator copies, so its first wait runs out, the
// block drains, frees its tensor memory and sets *err.  order (nsub > 1,
// optional): the launch's tiles in the order the blocks take them, entry
// j << 24 | t for tile t of sub-launch j (j < 256, t < 2^24).
void launch_umma_cgemm(const UmmaSub* subs, const int* prefix, int nsub, int ntiles, const int* active, int* err,
                       cudaStream_t s, const UmmaSub* one, unsigned long long wait_ns = 0, int withhold = 0,
                       const int* order = nullptr);

// FP64 GEMM on the int8 tensor path (kernels_i8.cu): 128 gathered columns x up to
// I8_TILE_ROWS complex operator rows per tile; both operands as seven int8 digit
// planes under a power-of-two scale per vector / operator row.
constexpr int I8_DIGITS = 7;
constexpr int I8_TILE_ROWS = 56;
constexpr int I8_GRANULE = 16 * 2 * I8_DIGITS;  // bytes of the digits of 16 complex numbers
struct alignas(16) I8Vec {  // a vector to write as digits
    long long src;  // its first element in X
    int gran;       // its first granule (and its entry of cx)
    unsigned short len;      // complex numbers
    unsigned short profile;  // as in GemmProblem; a launch's vectors all have one or none has
};
// Profile table: a row of `stride` biased exponents b = 67 .. 127 (as FP32 has them) for each class
// of vectors.  Component j of a vector of row p is scaled by 2^(b - 127), b = prof[p * stride + j],
// before it is written as digits, column j of an operator on it by the inverse (kernels_i8.cu).
struct I8Profiles {
    const unsigned char* prof;
    int stride;
};
// the row of a class from the typical sizes of its n components, padded with 127 to `stride`
std::vector<unsigned char> i8_profile(const double* size, int n, int stride);
void launch_i8_slice(const I8Vec* vecs, int n, const double2* X, char* X8, double* cx, const I8Profiles& T,
                     cudaStream_t s);
struct alignas(16) I8Tile {  // everything about a tile, so that its next one can be read ahead
    const char* B;         // the row tile's packed operator (i8_pack_kernel)
    const double* ra;      // output scales of its rows
    int col, row0;         // first column (of xgran, yoff), first operator row
    unsigned short ncol, rows, n, nkb;  // columns, valid complex rows, int8 rows, 16-wide complex K blocks
};
struct I8Sub {
    const I8Tile* tiles;
    const int* xgran;        // first granule of each column's vector
    const long long* yoff;   // element of Y each column adds into
    const char* X8;
    const double* cx;
    double2* Y;
    int ntiles;
};
struct I8PackJob {
    const double2* A;  // complex operator, column-major
    char* dst;
    double* ra;
    int m, k, lda, nkb, rows_t;
    const unsigned char* prof;  // of its columns, or null
};
void i8_init();
int i8_row_tiles(int m);
int i8_tile_rows(int m);
size_t i8_packed_bytes(int m, int k);
// the tiles of one problem: m x k operator packed at B with row scales ra, columns col0 .. col0 + ncol
void i8_tiles(const char* B, const double* ra, int m, int k, int col0, int ncol, std::vector<I8Tile>& out);
void launch_i8_pack(const I8PackJob* jobs_dev, int njobs, int max_tiles, cudaStream_t s);
// *err is set when a block gave up waiting on its pipeline; wait_ns, withhold as in launch_umma_cgemm
void launch_i8_gemm(const I8Sub& sub, int* err, cudaStream_t s, unsigned long long wait_ns = 0, int withhold = 0);
// gemm_test.cu: Y += A X through one of the GEMM kernels (paths as in ddfmm.h)
void test_gemm(const double2* A, int m, int k, const double2* X, int ncol, int path, double2* Y);

// Mixed-form high-frequency GEMM on the FP16 tensor cores (kernels_h16.cu): 128
// gathered columns x up to H16_TILE_ROWS complex operator rows per tile; both
// operands as two FP16 planes under a power-of-two scale per vector / operator row.
constexpr int H16_TILE_ROWS = 112;
constexpr int H16_GRANULE = 128;  // bytes of the planes of 16 complex numbers: 64 of hi, 64 of lo
struct HSliceSub {  // one instance's vectors to write as planes
    const I8Vec* vecs;
    const float2* X;
    char* X16;
    float* cx;  // output scale of the vector that starts at a granule
    int n;
    int inst;
    I8Profiles prof;  // prof.prof null: no vector has a profile, in any sub-launch of the launch
};
struct alignas(16) H16Tile {  // everything about a tile, so that its next one can be read ahead
    const float* B;           // the row tile's packed operator (h16_pack_kernel)
    const float* ra;          // output scales of its rows
    int col, row0;            // first column (of xgran, yoff), first operator row
    unsigned short ncol, rows, n, k;  // columns, valid complex rows, real rows, complex K
};
struct HSub {
    const H16Tile* tiles;
    const int* xgran;       // first granule of each column's vector
    const long long* yoff;  // element of Y each column adds into
    const char* X16;
    const float* cx;
    float2* Y;
    int ntiles;
    int inst;
};
struct H16PackJob {
    const float2* A;  // complex FP32 operator, column-major
    float* dst;
    float* ra;
    int m, k, lda, rows_t;
    const unsigned char* prof;  // of its columns, or null
};
void h16_init();
int h16_row_tiles(int m);
int h16_tile_rows(int m);
size_t h16_packed_floats(int m, int k);
const float* h16_scales(const float* packed, int m, int k);  // the row scales of a packed operator
void h16_tiles(const float* packed, int m, int k, int col0, int ncol, std::vector<H16Tile>& out);
void launch_h16_pack(const H16PackJob* jobs_dev, int njobs, int max_tiles, cudaStream_t s);
// nsub == 1: `one` is that sub-launch (sent as a kernel parameter); order, wait_ns, withhold as in launch_umma_cgemm
void launch_h16_slice(const HSliceSub* subs, const int* prefix, int nsub, int n, const int* active, cudaStream_t s,
                      const HSliceSub& one);
void launch_h16_gemm(const HSub* subs, const int* prefix, int nsub, int ntiles, const int* active, int* err,
                     cudaStream_t s, const HSub& one, const int* order = nullptr, unsigned long long wait_ns = 0,
                     int withhold = 0);

// gather/scatter helpers.  err: the int that the pipelined GEMM launches of an eval set
// when a block gave up on its pipeline; zero at the eval's start.  Outputs are then
// incomplete, and an enqueued eval has no status to return, so the scatter that ends it
// writes NaN for every value.
void launch_gather_den(const double2* den, const int* perm, double2* out, int n, cudaStream_t s);
void launch_scatter_val(const double2* in, const int* perm, double2* val, int n, const int* err, cudaStream_t s);
void launch_direct(const double* pos, const double2* den, int n, const int* chk, int nchk,
                   double2* out, int kernel, cudaStream_t s);

}  // namespace ddfmm
