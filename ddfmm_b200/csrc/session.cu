// Plan flattening and the eval launch sequence (see session.hpp).
//
// Pass structure and data flow follow Wave3d::eval (src/wave3d_eval.cpp:299-415):
//   1. low-frequency upward, widths ascending        (EvalUpwardLow :418-490)
//   2. high-frequency upward, widths ascending       (EvalUpwardHigh :773-854)
//   3. high-frequency downward, widths descending    (EvalDownwardHigh :996-1040,
//      HighFrequencyM2L :876-928, HighFrequencyL2L :931-993)
//   4. low-frequency downward, widths descending     (EvalDownwardLow :493-583 with
//      U/V/W/X lists :585-718)
// The reference walks directions recursively (pre-order up, post-order down,
// :721-751); every (box, wedge) only depends on its children (up) or its
// parent (down), so processing whole widths at a time gives the same sums.
// Operators are the reference's: Mlib3d::*Fetch (src/mlib3d.cpp:106-280).
#include "session.hpp"

#include "plan.hpp"

#include <algorithm>
#include <array>
#include <cctype>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <exception>
#include <set>
#include <stdexcept>
#include <thread>
#include <unordered_map>
#include <unordered_set>

namespace ddfmm {

#define CK(x)                                                                                      \
    do {                                                                                           \
        cudaError_t e_ = (x);                                                                      \
        if (e_ != cudaSuccess)                                                                     \
            throw std::runtime_error(std::string("CUDA error: ") + cudaGetErrorString(e_) + " (" + \
                                     #x + ")");                                                    \
    } while (0)

static int accu_to_p(int accu) {
    if (accu < 1 || accu > 3) throw std::runtime_error("ACCU must be 1, 2 or 3");  // src/wave3d.cpp:149
    return accu == 1 ? 4 : (accu == 2 ? 6 : 8);
}

template <class T>
T* Session::dalloc(size_t count) {
    if (count == 0) count = 1;
    void* p = nullptr;
    const auto t0 = std::chrono::steady_clock::now();
    CK(cudaMalloc(&p, count * sizeof(T)));
    t_malloc_ += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    ++n_malloc_;
    allocs_.push_back(p);
    alloc_bytes_[p] = count * sizeof(T);
    stats_.device_bytes += count * sizeof(T);
    return static_cast<T*>(p);
}

void Session::dfree(const void* p) {
    auto it = alloc_bytes_.find(p);
    if (it == alloc_bytes_.end()) return;  // not an allocation of this session (or an interior pointer)
    CK(cudaFree(const_cast<void*>(p)));
    stats_.device_bytes -= it->second;
    alloc_bytes_.erase(it);
    allocs_.erase(std::remove(allocs_.begin(), allocs_.end(), p), allocs_.end());
}

template <class T>
T* Session::upload_n(const T* src, size_t count) {
    const size_t bytes = count * sizeof(T);
    if (bytes > kArenaMax) {
        const auto t0 = std::chrono::steady_clock::now();
        T* d = nullptr;
        if (bytes <= kMidMax) {
            const size_t need = (bytes + 255) & ~(size_t)255;
            if (mid_used_ + need > mid_cap_) {  // chunks of 4 MiB doubling to 64 MiB: small sessions stay small
                const size_t cap = std::max(need, std::min(kMidChunk, std::max((size_t)kMidMax, 2 * mid_cap_)));
                void* chunk = nullptr;
                CK(cudaMalloc(&chunk, cap));
                allocs_.push_back(chunk);
                stats_.device_bytes += cap;
                mid_dev_ = static_cast<char*>(chunk);
                mid_used_ = 0;
                mid_cap_ = cap;
            }
            d = reinterpret_cast<T*>(mid_dev_ + mid_used_);
            mid_used_ += need;
        } else {
            d = dalloc<T>(count);
        }
        stage_copy(d, src, bytes);  // the caller's array may die right after: the data is staged
        t_big_uploads_ += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        return d;
    }
    const size_t need = (std::max<size_t>(bytes, 1) + 255) & ~(size_t)255;  // 256-byte aligned slots
    if (arena_.used + need > arena_.cap) {
        flush_uploads();
        // the copy out of the old host image may still be running: keep the
        // image until the end of the plan (released after a stream sync)
        if (!arena_.host.empty()) arena_.retired.push_back(std::move(arena_.host));
        // chunks of 1 MiB doubling to 64 MiB: small sessions stay small
        arena_.cap = std::max(need, std::min((size_t)64 << 20, std::max((size_t)1 << 20, 2 * arena_.cap)));
        // not through dalloc: a chunk must never be released by dfree(), which
        // would take an array that happens to start the chunk for its base
        void* chunk = nullptr;
        CK(cudaMalloc(&chunk, arena_.cap));
        allocs_.push_back(chunk);
        stats_.device_bytes += arena_.cap;
        arena_.dev = static_cast<char*>(chunk);
        arena_.host.assign(arena_.cap, 0);
        arena_.used = arena_.sent = 0;
    }
    char* d = arena_.dev + arena_.used;
    if (bytes) std::memcpy(arena_.host.data() + arena_.used, src, bytes);
    arena_.used += need;
    return reinterpret_cast<T*>(d);
}

void Session::flush_uploads() {
    if (arena_.used > arena_.sent)
        stage_copy(arena_.dev + arena_.sent, arena_.host.data() + arena_.sent, arena_.used - arena_.sent);
    arena_.sent = arena_.used;
}

void Session::stage_copy(void* dst, const void* src, size_t bytes) {
    if (!stage_[0])
        for (int k = 0; k < 2; ++k) {
            CK(cudaHostAlloc((void**)&stage_[k], kStage, cudaHostAllocDefault));
            CK(cudaEventCreateWithFlags(&stage_ev_[k], cudaEventDisableTiming));
            CK(cudaEventRecord(stage_ev_[k], stream_));
        }
    for (size_t off = 0; off < bytes;) {
        const size_t n = std::min(kStage, bytes - off);
        const int k = stage_next_;
        stage_next_ ^= 1;
        const auto t0 = std::chrono::steady_clock::now();
        CK(cudaEventSynchronize(stage_ev_[k]));  // the device has read this buffer's previous contents
        const auto t1 = std::chrono::steady_clock::now();
        std::memcpy(stage_[k], static_cast<const char*>(src) + off, n);
        t_stage_wait_ += std::chrono::duration<double>(t1 - t0).count();
        t_stage_copy_ += std::chrono::duration<double>(std::chrono::steady_clock::now() - t1).count();
        ++n_stage_;
        CK(cudaMemcpyAsync(static_cast<char*>(dst) + off, stage_[k], n, cudaMemcpyHostToDevice, stream_));
        CK(cudaEventRecord(stage_ev_[k], stream_));
        off += n;
    }
}

void Session::stage_release() {
    for (int k = 0; k < 2; ++k) {
        if (stage_ev_[k]) cudaEventDestroy(stage_ev_[k]);
        if (stage_[k]) cudaFreeHost(stage_[k]);
        stage_ev_[k] = nullptr;
        stage_[k] = nullptr;
    }
}

Session::Session(const double* pos3n, int n, const SessionParams& p, const std::string& ld_path,
                 const std::string& hd_path)
    : prm_(p), npts_(n) {
    if (n <= 0) throw std::runtime_error("no points");
    auto t0 = std::chrono::steady_clock::now();
    // operator files first (Mlib3d::setup): a bad file is reported before any device work
    ld_path_ = ld_path;
    hd_path_ = hd_path;
    auto since = [](std::chrono::steady_clock::time_point a) {
        return std::chrono::duration<double>(std::chrono::steady_clock::now() - a).count();
    };
    ops_ = OperatorLib::shared(ld_path, hd_path);
    ops_->validate(p.accu);
    stats_.ops_seconds = since(t0);
    CK(cudaSetDevice(p.device));
    CK(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    pos_.assign(pos3n, pos3n + 3 * (size_t)n);
    auto t1 = std::chrono::steady_clock::now();
    tree_.build(pos_.data(), n, p.tree);
    stats_.tree_seconds = since(t1);
    t1 = std::chrono::steady_clock::now();
    build();
    CK(cudaStreamSynchronize(stream_));
    stats_.plan_seconds = since(t1);
    t1 = std::chrono::steady_clock::now();
    autotune();
    CK(cudaStreamSynchronize(stream_));
    if (overlap_) build_graph();
    stats_.tune_seconds = since(t1);
    stats_.setup_seconds = since(t0);
}

Session::~Session() {
    if (stream_) cudaStreamSynchronize(stream_);
    stage_release();
    for (cudaEvent_t e : ev_) cudaEventDestroy(e);
    for (void* p : allocs_) cudaFree(p);
    for (cudaEvent_t e : branch_ev_) cudaEventDestroy(e);
    for (cudaStream_t b : branch_) cudaStreamDestroy(b);
    if (graph_) cudaGraphExecDestroy(graph_);
    if (stream_) cudaStreamDestroy(stream_);
}

void Session::add_gemm(std::vector<GemmProblem>& probs, std::vector<std::vector<long long> >& xo,
                       std::vector<std::vector<long long> >& yo, const double2* X, double2* Y, int mode,
                       const char* label, const Digits* dg, const std::vector<char>* on_i8) {
    if (on_i8 && !on_i8->empty() && umma()) {  // all problems
        i8_target_ = dg;
        add_gemm(probs, xo, yo, X, Y, mode, label);
        i8_target_ = nullptr;
        return;
    }
    if (on_i8 && !on_i8->empty()) {  // the problems chosen for the int8 path, then the others
        std::vector<GemmProblem> big, small;
        std::vector<std::vector<long long> > bx, by, sx, sy;
        for (size_t i = 0; i < probs.size(); ++i) {
            const bool b = (*on_i8)[i];
            (b ? big : small).push_back(probs[i]);
            (b ? bx : sx).push_back(std::move(xo[i]));
            (b ? by : sy).push_back(std::move(yo[i]));
        }
        i8_target_ = dg;
        add_gemm(big, bx, by, X, Y, mode, label);
        i8_target_ = nullptr;
        add_gemm(small, sx, sy, X, Y, mode, label);
        return;
    }
    struct Clock {
        double& acc;
        std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
        ~Clock() { acc += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count(); }
    } clock{t_emit_gemm_};
    // zgemm_narrow_kernel for launches of products with up to 40 columns (operators cold:
    // 8 columns 0.44-0.6 of zgemm_kernel's time, 24 columns 0.7-0.8, 32 columns 0.8-0.95,
    // 48 columns 0.95-1.1), for launches whose 64-column tiles would not give every SM a
    // block (150 columns of 56 x 56: 18 -> 11 us), and for a launch's products of up to
    // 24 columns where they are enough for a launch of their own
    bool narrow = narrow_;
    int kmax = 0, mmax = 0;
    if (!mixed() && !i8_target_ && !narrow_) {
        size_t tiles64 = 0, few = 0, many = 0;
        for (size_t i = 0; i < probs.size(); ++i) {
            tiles64 += (size_t)((probs[i].m + GEMM_TILE_M - 1) / GEMM_TILE_M) * ((xo[i].size() + GEMM_TILE_N - 1) / GEMM_TILE_N);
            if (xo[i].size() > 40) ++many;
            if (!xo[i].empty() && xo[i].size() <= 24) ++few;
        }
        if (tiles64 < 148 || many == 0) {
            narrow = true;
        } else if (few >= 148) {  // enough for a launch of their own
            std::vector<GemmProblem> big, small;
            std::vector<std::vector<long long> > bx, by, sx, sy;
            for (size_t i = 0; i < probs.size(); ++i) {
                const bool b = xo[i].size() > 24;
                (b ? big : small).push_back(probs[i]);
                (b ? bx : sx).push_back(std::move(xo[i]));
                (b ? by : sy).push_back(std::move(yo[i]));
            }
            narrow_ = true;
            add_gemm(small, sx, sy, X, Y, mode, label);
            narrow_ = false;
            add_gemm(big, bx, by, X, Y, mode, label);
            return;
        }
    }
    for (size_t i = 0; i < probs.size(); ++i) {
        kmax = std::max(kmax, probs[i].k);
        mmax = std::max(mmax, probs[i].m);
    }
    const int tile_m = narrow && mmax > 64 ? 128 : GEMM_TILE_M, tile_n = narrow ? 8 : GEMM_TILE_N;
    double flops = 0, bytes = 0;
    std::vector<GemmProblem> P;
    std::vector<size_t> from;  // the caller's problem of each P
    std::vector<GemmTile> tiles;
    size_t ncols = 0;
    for (size_t i = 0; i < probs.size(); ++i) {
        if (xo[i].empty() || probs[i].m == 0 || probs[i].k == 0) continue;
        GemmProblem q = probs[i];
        q.col0 = (int)ncols;
        q.ncol = (int)xo[i].size();
        if (yo[i].size() != xo[i].size()) throw std::logic_error("GEMM problem with unequal column lists");
        int pid = (int)P.size();
        P.push_back(q);
        from.push_back(i);
        ncols += (size_t)q.ncol;
        for (int r0 = 0; r0 < q.m; r0 += tile_m)
            for (int c0 = 0; c0 < q.ncol; c0 += tile_n) tiles.push_back(GemmTile{pid, r0, c0, 0});
        flops += 8.0 * q.m * q.k * (double)q.ncol;
        // operator once, each input and output column once (read-modify-write for += modes)
        bytes += 16.0 * ((double)q.m * q.k + (double)q.k * q.ncol + (mode == GEMM_SET ? 1.0 : 2.0) * q.m * q.ncol);
    }
    if (ncols > (size_t)INT_MAX) throw std::runtime_error("too many GEMM columns in one launch");
    // the launch's column offsets, concatenated in problem order on all host cores
    // (pieces of at most 64k columns); the arrays are not zeroed first
    std::unique_ptr<long long[]> xs(new long long[std::max<size_t>(ncols, 1)]);
    std::unique_ptr<long long[]> ys(new long long[std::max<size_t>(ncols, 1)]);
    {
        std::vector<std::array<size_t, 3> > pieces;  // (P index, first column, end column)
        for (size_t j = 0; j < P.size(); ++j)
            for (size_t c = 0; c < (size_t)P[j].ncol; c += 65536)
                pieces.push_back({{j, c, std::min((size_t)P[j].ncol, c + 65536)}});
        host_parallel_for(pieces.size(), [&](size_t e) {
            const size_t j = pieces[e][0], c0 = pieces[e][1], n = pieces[e][2] - c0;
            std::memcpy(xs.get() + P[j].col0 + c0, xo[from[j]].data() + c0, n * sizeof(long long));
            std::memcpy(ys.get() + P[j].col0 + c0, yo[from[j]].data() + c0, n * sizeof(long long));
        });
    }
    stats_.flops_gemm += flops;
    if (tiles.empty()) return;
    Step st{};
    st.kind = 0;
    st.label = label;
    st.flops = flops;
    st.bytes = bytes;
    if (i8_target_) {
        if (umma()) {
            add_h16(P, xs.get(), ys.get(), ncols, Y, *i8_target_, st);
        } else {
            // a label of its own, so that profiles show the two kernels apart
            st.label = width_label((std::string(label).substr(0, std::string(label).rfind("_w")) + "_i8").c_str(),
                                   std::atof(label + std::string(label).rfind("_w") + 2));
            add_i8(P, xs.get(), ys.get(), ncols, Y, *i8_target_, st);
        }
        push_step(st);
        stats_.gemm_launches++;
        return;
    }
    if (umma()) {
        add_umma(P, xs.get(), ys.get(), ncols, X, Y, mode, st);
        push_step(st);
        stats_.gemm_launches++;
        return;
    }
    st.g.probs = upload(P);
    st.g.tiles = upload(tiles);
    st.g.xoff = upload_n(xs.get(), ncols);
    st.g.yoff = upload_n(ys.get(), ncols);
    st.g.ntiles = (int)tiles.size();
    st.g.X = X;
    st.g.Y = Y;
    st.g.mode = mode;
    st.g.kmax = kmax;
    st.g.rows = narrow ? tile_m : 0;
    push_step(st);
    stats_.gemm_launches++;
}

const float* Session::cached_op(const std::string& key) {
    if (opctx_.empty()) return nullptr;
    std::shared_ptr<PackedOp> e = OpCache::find(opctx_ + "|" + key);
    if (!e) return nullptr;
    held_.push_back(e);
    return e->p;
}

const float* Session::packed_operator(const GemmProblem& q, bool h16) {
    if (q.packed) return q.packed;  // shared copy from the cache
    struct Clock {
        double& acc;
        std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
        ~Clock() { acc += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count(); }
    } clock{t_pack_};
    const auto key = std::make_pair((const void*)q.A, ((long long)q.m << 32) | (long long)q.k);
    auto it = packed_.find(key);
    if (it != packed_.end()) return it->second;
    // packed operators are sub-allocated from device chunks (256-byte aligned; cp.async.bulk
    // needs 16), the unit the operator cache frees; one larger than a chunk gets its own
    const size_t nf = ((h16 ? h16_packed_floats(q.m, q.k) : umma_packed_floats(q.m, q.k)) + 63) & ~(size_t)63;
    if (nf > chunk_left_) {
        Clock ca{t_pack_alloc_};
        // chunks of 16 MiB doubling to 128 MiB: small sessions stay small, large
        // ones make few allocations
        const size_t last = chunk_ ? chunk_->bytes() / sizeof(float) : 0;
        const size_t floats = std::max(nf, std::min((size_t)32 << 20, std::max((size_t)4 << 20, 2 * last)));
        chunk_ = std::make_shared<DevChunk>(prm_.device, floats * sizeof(float));
        chunk_pos_ = chunk_->data();
        chunk_left_ = floats;
        chunk_bytes_ += floats * sizeof(float);
        stats_.device_bytes += floats * sizeof(float);
    }
    float* d = chunk_pos_;
    chunk_pos_ += nf;
    chunk_left_ -= nf;
    std::shared_ptr<PackedOp> op = std::make_shared<PackedOp>(PackedOp{chunk_, d});
    held_.push_back(op);
    auto k = opkey_.find((const void*)q.A);
    if (k != opkey_.end()) to_publish_.push_back(std::make_pair(opctx_ + "|" + k->second, op));
    if (h16)
        h16_jobs_.push_back(H16PackJob{(const float2*)q.A, d, const_cast<float*>(h16_scales(d, q.m, q.k)), q.m, q.k, q.lda,
                                       h16_tile_rows(q.m), profile_of(q)});
    else
        pack_jobs_.push_back(UmmaPackJob{(const float2*)q.A, d, umma_tile_stride(q.k), q.m, q.k, q.lda, umma_nkb(q.k)});
    return packed_[key] = d;
}

// split-TF32 tcgen05 form of one grouped GEMM launch (low-frequency passes): tiles of 128 gathered columns x
// 128 complex operator rows, the tiles of one problem adjacent so that blocks
// in flight share its packed operator in L2.
void Session::add_umma(const std::vector<GemmProblem>& P, const long long* xs, const long long* ys, size_t ncols,
                       const double2* X, double2* Y, int mode, Step& st) {
    std::vector<UmmaProblem> U;
    std::vector<UmmaTile> tiles;
    for (size_t i = 0; i < P.size(); ++i) {
        const GemmProblem& q = P[i];
        U.push_back(UmmaProblem{packed_operator(q, false), umma_tile_stride(q.k), q.m, q.k, umma_nkb(q.k), q.col0, q.ncol});
        for (int rt = 0; rt * 128 < q.m; ++rt)
            for (int c0 = 0; c0 < q.ncol; c0 += 128) {
                tiles.push_back(UmmaTile{(int)i, rt, rt * 128, std::min(128, q.m - rt * 128), c0, 0});
                st.uop.push_back(U.back().B + (size_t)rt * U.back().tile_stride);
            }
    }
    st.kind = 5;
    st.hu = UmmaSub{upload(U), upload(tiles), upload_n(xs, ncols), upload_n(ys, ncols), reinterpret_cast<const float2*>(X),
                    reinterpret_cast<float2*>(Y), (int)tiles.size(), mode, 0, 0};
    set_multi(st, st.hu, (int)tiles.size());
}

// Which problems (m, k, columns) of a plain-form launch run on the int8 path;
// empty when none.  In clocks of one SM, fitted to launches of the K = 8 .. 64
// workloads: an int8 tile (128 columns x up to 56 rows, full or not) costs 10500
// and 2700 a K block (k = 76: 24 k, k = 152: 37 k); the FP64 tensor path does 11
// complex products a clock with many columns, 8 with few.  So 128 columns of a
// 100 x 152 operator cost 75 k against 177 k, 32 columns 75 k against 61 k.  The
// launch must gain what its digits, its second launch and its last wave cost.  An eval with
// that line at 0, 20 k, 60 k and 150 k clocks an SM (us): sphere K = 8, P = 4 341, 299, 289,
// 289; P = 6 835, 833, 835, 805; P = 8 1904, 1905, 1906, 1904; K = 4, P = 8 516, 490, 487,
// 486; ellipsoid K = 16, P = 4 423, 363, 345, 346; P = 6 984, 960, 962, 988; sphere K = 16,
// P = 4 1308, 1243, 1231, 1227; P = 6 3083, 3075, 3026, 3055; exp(ir) 1446, 1404, 1402, 1434;
// cluster K = 8, P = 4 671, 659, 664, 656; P = 8 2411, 2412, 2409, 2316.
static std::vector<char> i8_choose(const std::vector<std::array<int, 3> >& shapes) {
    std::vector<char> on(shapes.size(), 0);
    double gain = 0;
    for (size_t i = 0; i < shapes.size(); ++i) {
        const double m = shapes[i][0], k = shapes[i][1], c = shapes[i][2];
        const double t8 = std::ceil(c / 128) * i8_row_tiles(shapes[i][0]) * (10500 + 2700 * std::ceil(k / 16));
        const double t64 = m * k * c / (c < 96 ? 8 : 11);
        if (t8 < t64) {
            on[i] = 1;
            gain += t64 - t8;
        }
    }
    if (gain < 148 * 60e3) on.clear();
    return on;
}

// first granule of each gathered column's vector (Digits); not zeroed first
static std::unique_ptr<int[]> granules(const long long* xs, size_t ncols, long long base, int unit, int gran) {
    std::unique_ptr<int[]> xg(new int[std::max<size_t>(ncols, 1)]);
    host_parallel_for((ncols + 65535) / 65536, [&](size_t c) {
        for (size_t j = c * 65536; j < std::min(ncols, (c + 1) * 65536); ++j) xg[j] = (int)((xs[j] - base) / unit) * gran;
    });
    return xg;
}

// int8 form of one grouped GEMM launch: the operators packed as digits (now: they
// are on the device).
void Session::add_i8(const std::vector<GemmProblem>& P, const long long* xs, const long long* ys, size_t ncols,
                     double2* Y, const Digits& dg, Step& st) {
    std::vector<I8PackJob> jobs;
    std::vector<I8Tile> tiles;
    size_t bytes = 0, rows = 0;
    int max_tiles = 1;
    for (const GemmProblem& q : P) {
        bytes += i8_packed_bytes(q.m, q.k);
        rows += q.m;
        max_tiles = std::max(max_tiles, i8_row_tiles(q.m));
    }
    char* B = dalloc<char>(bytes);
    double* ra = dalloc<double>(rows);
    for (size_t i = 0; i < P.size(); ++i) {
        const GemmProblem& q = P[i];
        jobs.push_back(I8PackJob{q.A, B, ra, q.m, q.k, q.lda, (q.k + 15) / 16, i8_tile_rows(q.m), profile_of(q)});
        i8_tiles(B, ra, q.m, q.k, q.col0, q.ncol, tiles);
        B += i8_packed_bytes(q.m, q.k);
        ra += q.m;
    }
    const std::unique_ptr<int[]> xg = granules(xs, ncols, dg.base, dg.unit, dg.gran);
    const I8PackJob* dj = upload(jobs);
    flush_uploads();
    launch_i8_pack(dj, (int)jobs.size(), max_tiles, stream_);
    CK(cudaGetLastError());
    st.kind = 8;
    st.i8 = I8Sub{upload(tiles), upload_n(xg.get(), ncols), upload_n(ys, ncols), dg.X8, (const double*)dg.cx, Y, (int)tiles.size()};
}

// FP16 form of one grouped GEMM launch of the mixed form's high-frequency passes
// (kernels_h16.cu), tiles of one problem adjacent as in add_umma.
void Session::add_h16(const std::vector<GemmProblem>& P, const long long* xs, const long long* ys, size_t ncols,
                      double2* Y, const Digits& dg, Step& st) {
    std::vector<H16Tile> tiles;
    for (const GemmProblem& q : P) h16_tiles(packed_operator(q, true), q.m, q.k, q.col0, q.ncol, tiles);
    for (const H16Tile& t : tiles) st.uop.push_back(t.B);
    st.kind = 10;
    const std::unique_ptr<int[]> xg = granules(xs, ncols, dg.base, dg.unit, dg.gran);
    st.hh = HSub{upload(tiles), upload_n(xg.get(), ncols), upload_n(ys, ncols), dg.X8,
                 (const float*)dg.cx, reinterpret_cast<float2*>(Y), (int)tiles.size(), 0};
    set_multi(st, st.hh, (int)tiles.size());
}

// The digits (mixed form: FP16 planes) of the given vectors of X, for the GEMMs that gather them.
void Session::add_digits(const I8Vec* vecs, size_t n, const double2* X, const Digits& dg, const char* label) {
    Step st{};
    st.kind = 7;
    st.label = label;
    for (size_t i = 0; i < n; ++i) st.bytes += (umma() ? 16.0 : 30.0) * vecs[i].len;
    const I8Profiles prof = n && vecs[0].profile ? profiles_ : I8Profiles{};
    if (umma()) {
        st.kind = 9;
        st.hs = HSliceSub{upload_n(vecs, n), reinterpret_cast<const float2*>(X), dg.X8, (float*)dg.cx, (int)n, 0, prof};
        set_multi(st, st.hs, st.hs.n);
        push_step(st);
        return;
    }
    st.dg.vecs = upload_n(vecs, n);
    st.dg.n = (int)n;
    st.dg.X = X;
    st.dg.X8 = dg.X8;
    st.dg.cx = (double*)dg.cx;
    st.dg.prof = prof;
    push_step(st);
}

template <class Sub>
void Session::set_multi(Step& st, const Sub& sub, int total) {
    st.msubs = upload(std::vector<Sub>(1, sub));
    st.mpre = upload(std::vector<int>{0, total});
    st.mtotal = total;
}

// Steps are emitted in blocks (phase, width): LF upward and HF upward by
// ascending width, HF downward and LF downward by descending width.
void Session::begin_block(int phase, double W) {
    cur_phase_ = phase;
    const long long w = std::lround(std::log2(W));
    cur_wkey_ = phase < 2 ? 1000 + w : 1000 - w;
    block_counts_.clear();
}

void Session::push_step(Step st) {
    // step types in the order the blocks emit them
    static const char* const order[] = {"lf_s2m",       "lf_m2m",       "lf_uc2ue", "lf_digits", "hf_m2m",
                                        "hf_digits_up", "hf_m2l",       "hf_digits_down", "hf_l2l", "lf_vlist_fft", "lf_vlist_m2l", "lf_vlist_inv",
                                        "lf_xlist",     "lf_ulist",     "lf_wlist", "lf_dc2de", "lf_l2t", "lf_l2l"};
    std::string base(st.label);
    const size_t u = base.rfind("_w");
    if (u != std::string::npos && u + 2 < base.size() && std::isdigit((unsigned char)base[u + 2]))
        base = base.substr(0, u);  // per-width label "pass_w<W>"

    long long rank = 63;
    for (size_t i = 0; i < sizeof(order) / sizeof(order[0]); ++i)
        if (base == order[i]) rank = (long long)i;
    const long long occ = block_counts_[base]++;
    st.lane = lane_;
    bounded_waits_ |= st.kind == 5 || st.kind == 8 || st.kind == 10;
    st.key = ((long long)cur_phase_ << 48) | (cur_wkey_ << 32) | (rank << 16) | occ;
    steps_.push_back(st);
}

void Session::flush_packs() {
    flush_uploads();
    if (pack_jobs_.empty() && h16_jobs_.empty()) return;
    auto to_device = [&](const void* p, size_t bytes) {
        void* d = nullptr;
        CK(cudaMalloc(&d, std::max<size_t>(bytes, 16)));
        if (bytes) CK(cudaMemcpyAsync(d, p, bytes, cudaMemcpyHostToDevice, stream_));
        return d;
    };
    void* d = to_device(pack_jobs_.data(), sizeof(UmmaPackJob) * pack_jobs_.size());
    launch_umma_pack(static_cast<const UmmaPackJob*>(d), (int)pack_jobs_.size(), stream_);
    void* dh = to_device(h16_jobs_.data(), sizeof(H16PackJob) * h16_jobs_.size());
    int max_tiles = 1;
    for (const H16PackJob& j : h16_jobs_) max_tiles = std::max(max_tiles, h16_row_tiles(j.m));
    launch_h16_pack(static_cast<const H16PackJob*>(dh), (int)h16_jobs_.size(), max_tiles, stream_);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(stream_));
    CK(cudaFree(d));
    CK(cudaFree(dh));
    pack_jobs_.clear();
    h16_jobs_.clear();
    // packed and complete: other sessions may use them from now on
    for (auto& kp : to_publish_) OpCache::publish(kp.first, kp.second);
    to_publish_.clear();
}

void Session::check_device_error() {
    if (!bounded_waits_) return;
    int h = 0;
    CK(cudaMemcpyAsync(&h, d_err_, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    if (h) throw std::runtime_error("CUDA error: a tensor-core GEMM block timed out waiting on its pipeline");
}

void Session::arm_gemm_stall(double wait_s, int kind) {
    if (std::none_of(steps_.begin(), steps_.end(), [&](const Step& st) { return st.kind == kind; }))
        throw std::invalid_argument("the session's evals do not launch this tensor-core GEMM");
    if (!(wait_s > 0 && wait_s <= 1.0)) throw std::invalid_argument("stall wait must be in (0, 1] seconds");
    stall_wait_ns_ = (unsigned long long)(wait_s * 1e9);
    stall_kind_ = kind;
}

const char* Session::width_label(const char* pass, double W) {
    char buf[64];
    snprintf(buf, sizeof buf, "%s_w%g", pass, W);
    for (const std::string& l : label_store_)
        if (l == buf) return l.c_str();
    label_store_.reserve(256);  // pointers into the store must stay valid
    if (label_store_.size() >= 256) return pass;
    label_store_.push_back(buf);
    return label_store_.back().c_str();
}

void Session::add_pt(std::vector<PtItem> items, const std::vector<PtSrc>& srcs, const char* label) {
    if (items.empty()) return;
    // An item is one warp's (or less) in every launch shape and walks its sources one
    // after the other: where a step has fewer items than the GPU has room for warps, its
    // items are split by targets, down to one target an item (K = 4, P = 4, 150 leaves of
    // 10 points: U list 35 -> 13 us, L2T 21 -> 11 us with the events around them; 80 -> 72
    // us a matvec; K = 8 cluster 643 -> 593 us, mixed ellipsoid K = 16 504 -> 481 us)
    long long targets = 0;
    for (const PtItem& it : items) targets += it.trg.n;
    if (items.size() < kPtItems && targets > (long long)items.size()) {
        const int per = (int)std::max(1ll, targets / (long long)kPtItems);
        std::vector<PtItem> split;
        for (const PtItem& it : items)
            for (int t = 0; t < it.trg.n; t += per) {
                PtItem p = it;
                p.trg.x = it.trg.x + 3 * t;
                p.trg.n = std::min(per, it.trg.n - t);
                p.out = (double2*)((char*)it.out + (size_t)t * (mixed() ? sizeof(float2) : sizeof(double2)));
                split.push_back(p);
            }
        items.swap(split);
    }
    Step st{};
    st.kind = 1;
    st.label = label;
    for (const PtItem& it : items) {
        long long ns = 0;
        for (int k = it.src_begin; k < it.src_end; ++k) ns += srcs[k].src.n;
        // one kernel evaluation (sqrt, reciprocal, sincospi) + one complex MAC per pair
        st.flops += 20.0 * it.trg.n * (double)ns;
        st.bytes += 40.0 * ns + 56.0 * it.trg.n;
    }
    st.pt.items = upload(items);
    st.pt.srcs = upload(srcs);
    st.pt.nitems = (int)items.size();
    if (mixed()) {
        st.hp = PtSub{st.pt.items, st.pt.srcs, st.pt.nitems, prm_.kernel, 0, 0};
        set_multi(st, st.hp, st.pt.nitems);
    }
    push_step(st);
}

namespace {
// Setup-time matrix products C = A * B for many small operators in one
// launch: each product is one grouped-GEMM problem whose "columns" are the
// columns of B (read from pool X) and of C (written to pool Y).
struct GemmBatch {
    std::vector<GemmProblem> probs;
    std::vector<ColumnSpan> spans;  // the columns of each problem, listed on the device
    long long ncols = 0;
    // A (m x k, lda m, device pointer), B = X[bx ..] (k x n), C = Y[cy ..] (m x n)
    void product(const double2* A, int m, int k, size_t bx, int n, size_t cy) {
        probs.push_back(GemmProblem{A, m, k, m, (int)ncols, n, nullptr});
        spans.push_back(ColumnSpan{ncols, (long long)bx, (long long)cy, k, m});
        ncols += n;
    }
    void run(const double2* X, double2* Y, cudaStream_t s) {
        if (probs.empty()) return;
        if (ncols > INT_MAX) throw std::runtime_error("too many operator columns in one setup launch");
        std::vector<GemmTile> tiles;
        for (size_t i = 0; i < probs.size(); ++i)
            for (int r0 = 0; r0 < probs[i].m; r0 += GEMM_TILE_M)
                for (int c0 = 0; c0 < probs[i].ncol; c0 += GEMM_TILE_N) tiles.push_back(GemmTile{(int)i, r0, c0, 0});
        // one allocation: a cudaFree costs as much as a small product
        auto room = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
        const size_t bp = room(sizeof(GemmProblem) * probs.size()), bt = room(sizeof(GemmTile) * tiles.size()),
                     bs = room(sizeof(ColumnSpan) * spans.size());
        char* d = nullptr;
        CK(cudaMalloc(&d, bp + bt + bs + 2 * sizeof(long long) * (size_t)ncols));
        GemmProblem* dp = reinterpret_cast<GemmProblem*>(d);
        GemmTile* dt = reinterpret_cast<GemmTile*>(d + bp);
        ColumnSpan* ds = reinterpret_cast<ColumnSpan*>(d + bp + bt);
        long long* dx = reinterpret_cast<long long*>(d + bp + bt + bs);
        CK(cudaMemcpyAsync(dp, probs.data(), sizeof(GemmProblem) * probs.size(), cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(dt, tiles.data(), sizeof(GemmTile) * tiles.size(), cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(ds, spans.data(), sizeof(ColumnSpan) * spans.size(), cudaMemcpyHostToDevice, s));
        launch_list_columns(ds, (int)spans.size(), ncols, dx, dx + ncols, s);
        launch_gemm(dp, dt, (int)tiles.size(), dx, dx + ncols, X, Y, GEMM_SET, s);
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(s));
        cudaFree(d);
    }
};

Pt3 shifted_point(int ind, double W) {  // ShiftedPoint, src/mlib3d.cpp:21-30
    int a = (ind & 4) >> 2, b = (ind & 2) >> 1, c = ind & 1;
    return Pt3{{(a - 0.5) * W / 2, (b - 0.5) * W / 2, (c - 0.5) * W / 2}};
}
// HighFetchShuffle, src/mlib3d.cpp:308-325: res(prm(d)) = tmp(d), then res(d) *= sgn(d)
std::vector<double> shuffle(const PMat& p, const Idx3& prm, const Idx3& sgn, double extra_sign) {
    std::vector<double> r((size_t)3 * p.n);
    for (int k = 0; k < p.n; ++k) {
        double t[3];
        for (int d = 0; d < 3; ++d) t[prm[d]] = p.x[3 * k + d];
        for (int d = 0; d < 3; ++d) r[3 * k + d] = extra_sign * (sgn[d] * t[d]);
    }
    return r;
}
std::vector<double2> to_d2(const CMat& m) {
    std::vector<double2> r(m.a.size());
    for (size_t i = 0; i < m.a.size(); ++i) r[i] = make_double2(m.a[i].real(), m.a[i].imag());
    return r;
}
std::vector<double2> to_d2_transpose(const CMat& m) {  // Transpose, src/mlib3d.cpp:32-42
    std::vector<double2> r(m.a.size());
    for (int i = 0; i < m.m; ++i)
        for (int j = 0; j < m.n; ++j) r[(size_t)i * m.n + j] = make_double2(m(i, j).real(), m(i, j).imag());
    return r;
}
}  // namespace

void Session::build() {
    // DDFMM_SETUP_TRACE=1: time each part of the plan (with the stream drained
    // at each mark, so device work is charged to the part that enqueued it)
    // and print the times to stderr
    const bool trace = std::getenv("DDFMM_SETUP_TRACE") != nullptr;
    auto tmark = std::chrono::steady_clock::now();
    auto phase = [&](const char* what) {
        if (!trace) return;
        CK(cudaStreamSynchronize(stream_));
        const auto t = std::chrono::steady_clock::now();
        std::fprintf(stderr, "ddfmm setup %-16s %8.3f s\n", what, std::chrono::duration<double>(t - tmark).count());
        tmark = t;
    };
    const double eps = 1e-12;
    const int P = accu_to_p(prm_.accu), G = 2 * P, G3 = G * G * G;
    const int nE = P * P * P - (P - 2) * (P - 2) * (P - 2);
    const int kern = prm_.kernel;
    if (kern != KERNEL_HELM && kern != KERNEL_EXPR) throw std::runtime_error("unknown kernel type");
    // complex state: double2 (plain FP64 form) or float2 (mixed form); plan
    // offsets are in elements, so both forms share one plan
    const bool mixed = this->mixed();
    if (umma()) opctx_ = OpCache::context(prm_.device, kern, prm_.accu, prm_.tree.npq, ld_path_, hd_path_);
    const size_t es = mixed ? sizeof(float2) : sizeof(double2);
    auto E = [&](double2* base, size_t elems) { return (double2*)((char*)base + elems * es); };
    auto salloc = [&](size_t elems) { return (double2*)dalloc<char>(elems * es); };
    // operators are built in FP64; the mixed form multiplies with FP32 copies
    std::map<const double2*, const double2*> op32;
    auto opm = [&](const double2* a, size_t n) -> const double2* {
        if (!mixed) return a;
        auto it = op32.find(a);
        if (it != op32.end()) return it->second;
        float2* b = dalloc<float2>(n);
        flush_uploads();
        launch_to_c64(a, b, (long long)n, stream_);
        CK(cudaGetLastError());
        return op32[a] = (const double2*)b;
    };
    Tree& T = tree_;
    const int nb = (int)T.boxes.size();
    stats_.n_points = npts_;
    stats_.n_boxes = nb;

    // ---------------------------------------------------------------- LF boxes, leaves, points
    std::vector<int> lfbox, lfidx(nb, -1);
    for (int b : T.order)
        if (T.boxes[b].has_pts() && T.width(T.boxes[b].level) < 1 - eps) {
            lfidx[b] = (int)lfbox.size();
            lfbox.push_back(b);
        }
    const int nLF = (int)lfbox.size();
    stats_.n_lf_boxes = nLF;
    std::vector<int> perm, leaf_off(nLF, -1), leaf_cnt(nLF, 0);
    std::vector<double> pos_sorted;
    perm.reserve(npts_);
    pos_sorted.reserve(3 * (size_t)npts_);
    for (int l = 0; l < nLF; ++l) {
        const Box& B = T.boxes[lfbox[l]];
        if (!B.terminal()) continue;
        leaf_off[l] = (int)perm.size();
        leaf_cnt[l] = (int)B.pts.size();
        for (int id : B.pts) {
            perm.push_back(id);
            for (int d = 0; d < 3; ++d) pos_sorted.push_back(pos_[3 * (size_t)id + d]);
        }
        stats_.n_leaves++;
    }
    if ((int)perm.size() != npts_) throw std::runtime_error("tree leaves do not hold every point exactly once");
    d_perm_ = upload(perm);
    d_pos_ids_ = upload(pos_);
    d_pos_sorted_ = upload(pos_sorted);
    d_den_sorted_ = salloc(npts_);
    d_den_io_ = dalloc<double2>(npts_);
    d_val_io_ = dalloc<double2>(npts_);

    phase("points");
    std::map<int, std::vector<int> > lflevels;  // level -> lf ids (key order)
    for (int l = 0; l < nLF; ++l) lflevels[T.boxes[lfbox[l]].level].push_back(l);

    double2* lf_upeq = salloc((size_t)nLF * nE);
    double2* lf_mid = salloc((size_t)nLF * nE);
    double2* lf_dneq = salloc((size_t)nLF * nE);
    spectra_elems_ = (size_t)nLF * G3;
    stats_.fft_spectra_bytes = (long long)nLF * G3 * 16;

    // per-LF-level device operators
    struct LfLevelOps {
        double W;
        const double *uep, *ucp;
        double2 *up_s, *v, *vT_s, *upT, *tns;
        int* cube_idx;
        int r;
        double2* ue2uc[8];
        double2* de2dc[8];
        bool has_children;
    };
    std::map<int, LfLevelOps> lfops;
    std::vector<KmatJob> jobs;  // kernel-matrix generation, run once below
    long long job_elems = 0;
    auto add_job = [&](const double* trg, Pt3 ts, const double* src, Pt3 ss, int m, int k, double2* out) {
        KmatJob j;
        j.trg = trg;
        j.src = src;
        j.out = out;
        for (int d = 0; d < 3; ++d) {
            j.ts[d] = ts[d];
            j.ss[d] = ss[d];
        }
        j.m = m;
        j.k = k;
        j.elem0 = job_elems;
        job_elems += (long long)m * k;
        jobs.push_back(j);
    };
    const Pt3 zero3{{0, 0, 0}};
    std::vector<double2> twf(G), twb(G);
    {
        const long double twopi = 6.283185307179586476925286766559005768L;
        for (int m = 0; m < G; ++m) {
            long double a = twopi * (long double)m / (long double)G;
            twf[m] = make_double2((double)cosl(a), -(double)sinl(a));
            twb[m] = make_double2((double)cosl(a), (double)sinl(a));
        }
    }
    const double2* d_twf = opm(upload(twf), G);
    const double2* d_twb = opm(upload(twb), G);
    vlist_init(G);
    gemm_init();
    vlist32_init(G);
    cgemm_init();
    if (umma()) {
        umma_init();
        h16_init();
    }

    for (auto& kv : lflevels) {
        int level = kv.first;
        double W = T.width(level);
        const LowFreqOp& op = ops_->low(W);
        if (op.uep.n != nE || op.ucp.n != nE)
            throw std::runtime_error("low-frequency operator size does not match ACCU");
        LfLevelOps L{};
        L.W = W;
        L.r = op.up.m;
        L.uep = upload(op.uep.x);
        L.ucp = upload(op.ucp.x);
        // fold the 1/sigma scaling into the rows of U^H (up) and of v^T.  The mixed
        // form truncates the pseudo-inverse further, at sigma < 1e-7 sigma_max: FP32
        // check values carry ~1e-7 relative noise, which the directions below that
        // would amplify into equivalent densities whose norm swamps every later FP32
        // translation (at P = 8 sigma spans 12 decades)
        double smax = 0;
        for (int i = 0; i < L.r; ++i) smax = std::max(smax, 1.0 / std::abs(op.is(i, 0)));
        std::vector<double2> up_s((size_t)L.r * nE), vT_s((size_t)L.r * nE);
        for (int i = 0; i < L.r; ++i)
            for (int j = 0; j < nE; ++j) {
                cpx s = op.is(i, 0);
                if (mixed && 1.0 / std::abs(s) < 1e-7 * smax) s = 0;
                cpx a = s * op.up(i, j), b = s * op.v(j, i);
                up_s[(size_t)j * L.r + i] = make_double2(a.real(), a.imag());
                vT_s[(size_t)j * L.r + i] = make_double2(b.real(), b.imag());
            }
        L.up_s = upload(up_s);
        L.vT_s = upload(vT_s);
        L.v = upload(to_d2(op.v));
        L.upT = upload(to_d2_transpose(op.up));
        // V-list tensors and grid positions of the uep / dcp nodes (src/wave3d_eval.cpp:607-659)
        if (op.tdim != 0 && op.tdim != G) throw std::runtime_error("ue2dc tensor size does not match ACCU");
        std::vector<double2> tns((size_t)343 * G3, make_double2(0, 0));
        for (int o = 0; o < 343; ++o) {
            const auto& t = op.ue2dc[o];
            if (t.empty()) continue;
            for (int e = 0; e < G3; ++e) tns[(size_t)o * G3 + e] = make_double2(t[e].real(), t[e].imag());
        }
        L.tns = (double2*)opm(upload(tns), tns.size());
        // (src/wave3d_eval.cpp:626-628,655-657): a = round((x + W/2)/step) + P in [P, 2P)
        std::vector<int> cidx(nE);
        double step = W / (P - 1);
        for (int k = 0; k < nE; ++k) {
            int a[3];
            for (int d = 0; d < 3; ++d) a[d] = (int)std::round((op.uep.x[3 * k + d] + W / 2) / step) + P;
            for (int d = 0; d < 3; ++d)
                if (a[d] < P || a[d] >= 2 * P) throw std::runtime_error("V-list grid index outside the corner cube");
            cidx[k] = (a[0] - P) + P * ((a[1] - P) + P * (a[2] - P));
        }
        L.cube_idx = upload(cidx);
        L.has_children = false;
        for (int l : kv.second)
            if (!T.boxes[lfbox[l]].terminal()) L.has_children = true;
        if (L.has_children) {
            const LowFreqOp& ch = ops_->low(W / 2);  // UpwardLowFetch / DownwardLowFetch
            const double* chuep = upload(ch.uep.x);
            for (int ind = 0; ind < 8; ++ind) {
                L.ue2uc[ind] = dalloc<double2>((size_t)nE * nE);
                L.de2dc[ind] = dalloc<double2>((size_t)nE * nE);
                add_job(L.ucp, zero3, chuep, shifted_point(ind, W), nE, nE, L.ue2uc[ind]);
                add_job(chuep, shifted_point(ind, W), L.ucp, zero3, nE, nE, L.de2dc[ind]);
            }
        }
        lfops[level] = L;
    }

    phase("lf_operators");
    // ---------------------------------------------------------------- HF nodes
    struct Canon {
        double W;
        Idx3 srt;
        const HighFreqOp* op;
        int r1, r2;
        double2 *E1, *E2, *E3, *E1t, *E2t, *E3t;
        double *uep, *neg_uep;
    };
    std::vector<Canon> hfcanon;
    std::map<std::pair<double, Idx3>, int> canon_id;
    auto get_canon = [&](double W, const Idx3& dir, Idx3& sgn, Idx3& prmv) -> int {
        Idx3 srt;
        index3_sort(dir, srt, sgn, prmv);
        auto key = std::make_pair(W, srt);
        auto it = canon_id.find(key);
        if (it != canon_id.end()) return it->second;
        Canon c{};
        c.W = W;
        c.srt = srt;
        c.op = &ops_->high(W, srt);
        c.r1 = c.op->uep.n;
        c.r2 = c.op->ucp.n;
        if (c.op->E1.m != c.r1 || c.op->E1.n != c.r1 || c.op->E2.m != c.r1 || c.op->E2.n != c.r2 ||
            c.op->E3.m != c.r2 || c.op->E3.n != c.r2)
            throw std::runtime_error("high-frequency operator shapes are inconsistent");
        if (c.r1 > 400 || c.r2 > 400)  // DVMAX, src/wave3d_eval.cpp:25,842-844
            throw std::runtime_error("high-frequency rank exceeds DVMAX=400");
        c.E1 = upload(to_d2(c.op->E1));
        c.E2 = upload(to_d2(c.op->E2));
        c.E3 = upload(to_d2(c.op->E3));
        c.E1t = upload(to_d2_transpose(c.op->E1));
        c.E2t = upload(to_d2_transpose(c.op->E2));
        c.E3t = upload(to_d2_transpose(c.op->E3));
        c.uep = upload(c.op->uep.x);
        std::vector<double> neg(c.op->uep.x);
        for (double& v : neg) v = -v;
        c.neg_uep = upload(neg);
        int id = (int)hfcanon.size();
        hfcanon.push_back(c);
        canon_id[key] = id;
        return id;
    };
    // per (W, dir) shuffled point sets
    struct DirPts {
        double *ucp, *dep, *uep, *dcp;  // S*ucp, -S*ucp, S*uep, -S*uep
        int r1, r2, canon;
        int did;  // dense id, in order of first use
    };
    std::map<std::pair<double, Idx3>, DirPts> dirpts;
    // dense index into dirpts (node addresses are stable): per width, the wedge's
    // components (each in [-C, C], C = npq W) address a (2C+1)^3 table
    struct DirTable {
        double W;
        int C;
        std::vector<const DirPts*> t;
    };
    std::deque<DirTable> dirtabs;
    DirTable* last_tab = nullptr;
    auto dir_slot = [&](double W, const Idx3& d) -> const DirPts** {
        if (!last_tab || last_tab->W != W) {
            last_tab = nullptr;
            for (DirTable& x : dirtabs)
                if (x.W == W) last_tab = &x;
            if (!last_tab) {
                const int C = prm_.tree.npq * (int)std::round(W);
                if (C <= 0 || C > 128) return nullptr;
                dirtabs.push_back(DirTable{W, C, std::vector<const DirPts*>((size_t)(2 * C + 1) * (2 * C + 1) * (2 * C + 1), nullptr)});
                last_tab = &dirtabs.back();
            }
        }
        const int C = last_tab->C, E = 2 * C + 1;
        for (int k = 0; k < 3; ++k)
            if (d[k] < -C || d[k] > C) return nullptr;
        return &last_tab->t[((size_t)(d[0] + C) * E + (d[1] + C)) * E + (d[2] + C)];
    };
    auto get_dir = [&](double W, const Idx3& dir) -> const DirPts& {
        const DirPts** slot = dir_slot(W, dir);
        if (slot && *slot) return **slot;
        auto key = std::make_pair(W, dir);
        auto it = dirpts.find(key);
        if (it != dirpts.end()) {
            if (slot) *slot = &it->second;
            return it->second;
        }
        Idx3 sgn, pv;
        int c = get_canon(W, dir, sgn, pv);
        const HighFreqOp& op = *hfcanon[c].op;
        DirPts d{};
        d.did = (int)dirpts.size();
        d.canon = c;
        d.r1 = hfcanon[c].r1;
        d.r2 = hfcanon[c].r2;
        d.ucp = upload(shuffle(op.ucp, pv, sgn, 1.0));
        d.dep = upload(shuffle(op.ucp, pv, sgn, -1.0));
        d.uep = upload(shuffle(op.uep, pv, sgn, 1.0));
        d.dcp = upload(shuffle(op.uep, pv, sgn, -1.0));
        DirPts& stored = dirpts[key] = d;
        if (slot) *slot = &stored;
        return stored;
    };

    std::map<int, std::vector<int> > hflevels;  // level -> tree boxes with points, width >= 1
    for (int b : T.order)
        if (T.boxes[b].has_pts() && T.width(T.boxes[b].level) > 1 - eps) hflevels[T.boxes[b].level].push_back(b);

    // node vectors start at multiples of 16 complex numbers: the granules of the
    // int8 GEMM's digits, and aligned 128-byte (64-byte) pieces for the others
    auto node_stride = [](int r) { return (long long)((r + 15) & ~15); };
    // nodes of a box are contiguous and in its (sorted) wedge order, so a
    // (box, wedge) node is found by binary search in the box's range (HfNodes::find)
    HfNodes up, dn;
    up.first.assign(nb, 0);
    up.cnt.assign(nb, 0);
    dn.first.assign(nb, 0);
    dn.cnt.assign(nb, 0);
    {
        size_t nu = 0, nd = 0;
        for (auto& kv : hflevels)
            for (int b : kv.second) {
                nu += T.boxes[b].outdirs.size();
                nd += T.boxes[b].incdirs.size();
            }
        up.v.reserve(nu);
        dn.v.reserve(nd);
    }
    long long upeq_total = 0, dnchk_total = 0;
    for (auto& kv : hflevels) {
        const double W = T.width(kv.first);
        const std::vector<int>& bx = kv.second;
        const size_t nbx = bx.size();
        // the level's wedges, created in first-use order (their dense ids follow it):
        // a box's outgoing wedges, then its incoming ones, box by box
        for (int b : bx) {
            for (const Idx3& d : T.boxes[b].outdirs) get_dir(W, d);
            for (const Idx3& d : T.boxes[b].incdirs) get_dir(W, d);
        }
        // every wedge of the level now has its point sets: the nodes are filled on
        // all host cores from per-box prefix sums (a box's nodes are contiguous, in
        // its sorted wedge order), read-only lookups through the level's table
        const DirPts** tab = dir_slot(W, Idx3{{0, 0, 0}}) ? last_tab->t.data() : nullptr;
        const int C = last_tab ? last_tab->C : 0, E = 2 * C + 1;
        auto lookup = [&](const Idx3& d) -> const DirPts& {
            if (tab && d[0] >= -C && d[0] <= C && d[1] >= -C && d[1] <= C && d[2] >= -C && d[2] <= C) {
                const DirPts* q = tab[((size_t)(d[0] + C) * E + (d[1] + C)) * E + (d[2] + C)];
                if (q) return *q;
            }
            return dirpts.at(std::make_pair(W, d));
        };
        std::vector<long long> uo(nbx + 1, 0), dof(nbx + 1, 0);
        std::vector<int> un(nbx + 1, 0), dnn(nbx + 1, 0);
        host_parallel_for(nbx, [&](size_t i) {
            const Box& B = T.boxes[bx[i]];
            long long a = 0, c = 0;
            for (const Idx3& d : B.outdirs) a += node_stride(lookup(d).r1);
            for (const Idx3& d : B.incdirs) c += node_stride(lookup(d).r1);
            uo[i + 1] = a;
            dof[i + 1] = c;
            un[i + 1] = (int)B.outdirs.size();
            dnn[i + 1] = (int)B.incdirs.size();
        });
        const int u0 = (int)up.v.size(), d0 = (int)dn.v.size();
        uo[0] = upeq_total;
        dof[0] = dnchk_total;
        un[0] = u0;
        dnn[0] = d0;
        for (size_t i = 0; i < nbx; ++i) {
            uo[i + 1] += uo[i];
            dof[i + 1] += dof[i];
            un[i + 1] += un[i];
            dnn[i + 1] += dnn[i];
        }
        up.v.resize((size_t)un[nbx]);
        dn.v.resize((size_t)dnn[nbx]);
        host_parallel_for(nbx, [&](size_t i) {
            const int b = bx[i];
            const Box& B = T.boxes[b];
            up.first[b] = un[i];
            up.cnt[b] = un[i + 1] - un[i];
            long long o = uo[i];
            int k = un[i];
            for (const Idx3& d : B.outdirs) {
                const DirPts& dp = lookup(d);
                up.v[k++] = HfNode{b, d, dp.canon, o, o, dp.did};  // M2M adds straight into the vector
                o += node_stride(dp.r1);
            }
            dn.first[b] = dnn[i];
            dn.cnt[b] = dnn[i + 1] - dnn[i];
            o = dof[i];
            k = dnn[i];
            for (const Idx3& d : B.incdirs) {
                const DirPts& dp = lookup(d);
                dn.v[k++] = HfNode{b, d, dp.canon, o, o, dp.did};  // L2L reads the vector itself
                o += node_stride(dp.r1);
            }
        });
        upeq_total = uo[nbx];
        dnchk_total = dof[nbx];
        up.range[kv.first] = std::make_pair(u0, (int)up.v.size());
        dn.range[kv.first] = std::make_pair(d0, (int)dn.v.size());
    }
    phase("hf_nodes");
    stats_.hf_up_nodes = (long long)up.v.size();
    stats_.hf_down_nodes = (long long)dn.v.size();
    // every accumulator of an eval in one allocation, zeroed by one memset at its start,
    // and with them the flag of GEMMs that gave up: an eval reports its own failure only
    const size_t acc_elems[5] = {(size_t)npts_, (size_t)nLF * nE, (size_t)nLF * nE, (size_t)upeq_total,
                                 (size_t)dnchk_total};
    size_t acc_off[6] = {0};
    for (int i = 0; i < 5; ++i) acc_off[i + 1] = acc_off[i] + ((acc_elems[i] + 31) & ~(size_t)31);
    double2* acc = salloc(acc_off[5] + 1);
    zero_at_start_.push_back(Memset{acc, es * (acc_off[5] + 1)});
    d_err_ = (int*)E(acc, acc_off[5]);
    d_val_sorted_ = acc;
    double2* lf_upchk = E(acc, acc_off[1]);
    double2* lf_dnchk = E(acc, acc_off[2]);
    double2* hf_upeq = E(acc, acc_off[3]);
    double2* hf_dnchk = E(acc, acc_off[4]);

    // ---------------------------------------------------------------- HF operators
    // Raw kernel matrices -- M2M ue2uc and L2L de2dc per (W, wedge, child), M2L per
    // (W, canonical wedge, canonical offset) -- are generated once, then folded
    // with the skeleton factors of uc2ue = {E1, E2, E3} (src/mlib3d.cpp:204-207,
    // :246-250) so that the eval applies one dense operator per translation plus
    // nothing else:
    //   upward   w   += [E2 * (E3 * ue2uc_c * E1(child))] w_c           (upeqnden = E1 w)
    //   M2L      u_t += [E1^T * M(o) * E1] w_s                          (u = E1^T dnchkval)
    //   downward u_c += [(E1(child)^T * de2dc_c * E3^T) * E2^T] u       (dneqnden = E3^T E2^T u)
    // At W = 1 the children are low-frequency boxes and carry no E1 factor.
    // E1 = inv(R1) and E3 = inv(R2^H) are ill-conditioned (~1e7), so they are
    // only ever multiplied into the smooth kernel matrices, never into each other;
    // E2 joins last.  Applied per node instead, E2 and E2^T were 14% of the HF
    // products and four of the ten HF launches of a width, and their inputs and
    // outputs another pass over the node vectors; folded, the rounding of a
    // translation is the same in FP64 (2e-15 against a long-double product, within
    // 15% of the two-step form) and 2-4 times smaller in FP32.
    auto take = [](size_t& pool, size_t n) {
        size_t o = pool;
        pool += (n + 15) & ~(size_t)15;
        return o;
    };
    size_t scr = 0;
    // place of a folded operator: kInt8 | offset in the pool of int8 products' operators, or an
    // offset in the other pool, or kNone (no box has a child there)
    constexpr size_t kInt8 = (size_t)1 << 62, kNone = ~(size_t)0;
    // cache keys of the shared operators: (kind, width, wedge, child or offset)
    auto opk = [](const char* kind, double W, const Idx3& d, int a, int b = 0, int c = 0) {
        char buf[128];
        snprintf(buf, sizeof buf, "%s|%.17g|%d,%d,%d|%d,%d,%d", kind, W, d[0], d[1], d[2], a, b, c);
        return std::string(buf);
    };
    struct DirMats {
        size_t raw[8], tmp[8], fin[8];
        int mrows, mcols, rmid, canon, ccanon;  // rmid: the wedge's r2, between the factors
        bool cached;            // all eight come from the shared cache
        const float* pk[8];     // their packed copies
    };
    std::map<std::pair<double, Idx3>, DirMats> m2m_mats, l2l_mats;
    const double* lf_half_uep = nullptr;
    if (!hflevels.empty()) {
        const LowFreqOp& lf_half = ops_->low(0.5);
        if (lf_half.uep.n != nE) throw std::runtime_error("width-1/2 operators do not match ACCU");
        lf_half_uep = upload(lf_half.uep.x);
    }
    auto child_pts = [&](double W, const Idx3& dir, bool upward, int& rc, int& ccanon) -> const double* {
        if (W == 1.0) {
            rc = nE;
            ccanon = -1;
            return lf_half_uep;  // LF uep at W/2 for both directions (src/mlib3d.cpp:199-202,254-257)
        }
        const DirPts& cp = get_dir(W / 2, predir(dir));
        rc = cp.r1;
        ccanon = cp.canon;
        return upward ? cp.uep : cp.dcp;
    };
    std::vector<DirMats*> m2m_of(dirpts.size(), nullptr), l2l_of(dirpts.size(), nullptr);  // by dense wedge id
    for (auto& kv : hflevels) {
        double W = T.width(kv.first);
        auto ur = up.range[kv.first], dr = dn.range[kv.first];
        for (int i = ur.first; i < ur.second; ++i) {
            if (m2m_of[up.v[i].did]) continue;
            auto key = std::make_pair(W, up.v[i].dir);
            const DirPts& dp = get_dir(W, up.v[i].dir);
            DirMats M{};
            child_pts(W, up.v[i].dir, true, M.mcols, M.ccanon);
            M.mrows = dp.r1;
            M.rmid = dp.r2;
            M.canon = dp.canon;
            M.cached = !opctx_.empty();
            for (int ind = 0; ind < 8 && M.cached; ++ind)
                M.cached = (M.pk[ind] = cached_op(opk("m2m", W, up.v[i].dir, ind))) != nullptr;
            for (int ind = 0; ind < 8 && !M.cached; ++ind) {
                M.raw[ind] = take(scr, (size_t)M.rmid * M.mcols);
                M.tmp[ind] = take(scr, (size_t)M.rmid * M.mcols);
                M.fin[ind] = kNone;
            }
            m2m_of[up.v[i].did] = &(m2m_mats[key] = M);
        }
        for (int i = dr.first; i < dr.second; ++i) {
            if (l2l_of[dn.v[i].did]) continue;
            auto key = std::make_pair(W, dn.v[i].dir);
            const DirPts& dp = get_dir(W, dn.v[i].dir);
            DirMats M{};
            child_pts(W, dn.v[i].dir, false, M.mrows, M.ccanon);
            M.mcols = dp.r1;
            M.rmid = dp.r2;
            M.canon = dp.canon;
            M.cached = !opctx_.empty();
            for (int ind = 0; ind < 8 && M.cached; ++ind)
                M.cached = (M.pk[ind] = cached_op(opk("l2l", W, dn.v[i].dir, ind))) != nullptr;
            for (int ind = 0; ind < 8 && !M.cached; ++ind) {
                M.raw[ind] = take(scr, (size_t)M.mrows * M.rmid);
                M.tmp[ind] = take(scr, (size_t)M.mrows * M.rmid);
                M.fin[ind] = kNone;
            }
            l2l_of[dn.v[i].did] = &(l2l_mats[key] = M);
        }
    }
    phase("m2m_l2l_plan");
    // M2L: canonical offset o_c = S^-1 (c_t - c_s), so M(dir, o) = M(canon, o_c)
    std::unordered_map<uint64_t, int> m2l_id;  // (canon, ox, oy, oz) packed -> matrix
    struct M2LMat {
        size_t raw, tmp, fin;
        int canon, r1;
        Pt3 shift;
        const float* pk;  // packed copy from the shared cache, or null
        std::string key;
    };
    std::vector<M2LMat> m2l_mats;
    std::map<int, std::vector<std::vector<long long> > > m2l_x, m2l_y;  // level -> per problem columns
    std::map<int, std::vector<int> > m2l_probs;                         // level -> matrix ids
    {
        // far pairs listed on all host cores (plan.cpp), merged here in chunk order:
        // matrix ids, problem order and column order as one pass in node order
        std::vector<M2LChunk> chunks = m2l_pairs(T, up, dn);
        std::vector<int> local;  // matrix id -> problem index within its level (-1: none yet)
        int cur_level = INT_MIN;
        for (M2LChunk& C : chunks) {
            if (C.level != cur_level) {
                cur_level = C.level;
                local.assign(m2l_mats.size(), -1);
            }
            const double W = T.width(C.level);
            auto& X = m2l_x[C.level];
            auto& Y = m2l_y[C.level];
            auto& Pids = m2l_probs[C.level];
            for (size_t k = 0; k < C.keys.size(); ++k) {
                auto mit = m2l_id.find(C.keys[k]);
                int gid;
                if (mit == m2l_id.end()) {
                    const Canon& c = hfcanon[C.kcanon[k]];
                    const std::array<int, 3>& oc = C.koc[k];
                    gid = (int)m2l_mats.size();
                    size_t n = (size_t)c.r1 * c.r1;
                    const std::string key = opk("m2l", W, c.srt, oc[0], oc[1], oc[2]);
                    const float* pk = cached_op(key);
                    M2LMat M{0, 0, 0, C.kcanon[k], c.r1, Pt3{{oc[0] * W, oc[1] * W, oc[2] * W}}, pk, key};
                    if (!pk) {
                        M.raw = take(scr, n);
                        M.tmp = take(scr, n);
                    }
                    m2l_mats.push_back(M);
                    m2l_id[C.keys[k]] = gid;
                } else {
                    gid = mit->second;
                }
                if ((size_t)gid >= local.size()) local.resize(m2l_mats.size(), -1);
                int li = local[gid];
                if (li < 0) {
                    li = (int)Pids.size();
                    local[gid] = li;
                    Pids.push_back(gid);
                    X.emplace_back();
                    Y.emplace_back();
                }
                X[li].insert(X[li].end(), C.X[k].begin(), C.X[k].end());
                Y[li].insert(Y[li].end(), C.Y[k].begin(), C.Y[k].end());
            }
            stats_.hf_far_pairs += C.pairs;
            std::vector<std::vector<long long> >().swap(C.X);
            std::vector<std::vector<long long> >().swap(C.Y);
        }
    }
    phase("m2l_plan");
    stats_.m2l_matrices = (long long)m2l_mats.size();
    // children with points of every high-frequency box (-1: none)
    std::vector<int> kids((size_t)nb * 8, -1);
    for (auto& kv : hflevels)
        for (int b : kv.second)
            for (int ind = 0; ind < 8; ++ind) {
                const int c = T.child(b, ind);
                if (c >= 0 && T.boxes[c].has_pts()) kids[(size_t)b * 8 + ind] = c;
            }
    // the column lists of every level's M2M and L2L launches, built on all host cores (plan.cpp)
    std::vector<std::pair<double, Idx3> > did_wedge(dirpts.size());
    for (auto& kv : dirpts) did_wedge[kv.second.did] = kv.first;
    std::vector<long long> lf_off(nb, -1);
    for (int l = 0; l < nLF; ++l) lf_off[lfbox[l]] = (long long)l * nE;
    HfColumns cols = hf_columns(T, up, dn, kids, lf_off, dirpts.size(), hfcanon.size(), false);
    phase("hf_columns");
    // ---------------------------------------------------------------- routes of the HF products
    // plain form: the int8 path for problems large enough; tcgen05 form: FP16 planes for all
    std::map<int, std::vector<char> > m2m_i8, m2l_i8, l2l_i8;  // level -> problems on the int8 path
    std::set<int> up_i8, dn_i8;  // levels whose outgoing / incoming vectors are written as digits
    bool lf_i8 = false;
    const bool profiled = hfcanon.size() < 65535;  // I8Vec::profile has 16 bits
    if (!mixed || umma()) {
        auto choose = [&](const std::vector<std::array<int, 3> >& shapes) {
            if (umma()) return std::vector<char>(shapes.size(), 1);
            if (!profiled) return std::vector<char>();
            if (prm_.int8_rule == INT8_BY_SIZE) return i8_choose(shapes);
            std::vector<char> on(prm_.int8_rule == INT8_ALTERNATE ? shapes.size() : 0);
            for (size_t i = 0; i < on.size(); i += 2) on[i] = 1;
            return on;
        };
        for (auto& kv : hflevels) {
            const int level = kv.first;
            const double W = T.width(level);
            auto shapes = [&](const ColLists& L, const std::vector<DirMats*>& of) {
                std::vector<std::array<int, 3> > v;
                if (umma()) v.resize(L.key.size());  // all of them
                for (size_t i = v.size(); i < L.key.size(); ++i) {
                    const DirMats& M = *of[L.key[i] / 8];
                    v.push_back({{M.mrows, M.mcols, (int)L.x[i].size()}});
                }
                return v;
            };
            std::vector<std::array<int, 3> > far;
            for (size_t i = 0; i < m2l_probs[level].size(); ++i) {
                const int r1 = m2l_mats[m2l_probs[level][i]].r1;
                far.push_back({{r1, r1, (int)m2l_x[level][i].size()}});
            }
            m2m_i8[level] = choose(shapes(cols.m2m.at(level), m2m_of));
            m2l_i8[level] = choose(far);
            l2l_i8[level] = choose(shapes(cols.l2l.at(level), l2l_of));
            if (!m2m_i8[level].empty()) {
                if (W == 1.0)
                    lf_i8 = true;
                else
                    up_i8.insert(level + 1);
            }
            if (!m2l_i8[level].empty()) up_i8.insert(level);
            if (!l2l_i8[level].empty()) dn_i8.insert(level);
        }
    }
    // The folded operators.  i8_pack_kernel alone reads those of int8 products, so theirs is a
    // pool that is released once they are packed: FP64 operators kept beside their digits,
    // digits with memory of their own each way and spectra beside them took 26.6 GB for a
    // sphere of K = 64 at P = 6, released and shared they take 19.9 (24.0 while it is set up)
    size_t keep = 0, keep8 = 0;
    auto lay_out = [&](size_t& fin, size_t n, const std::vector<char>& on, size_t i) {
        fin = !mixed && !on.empty() && on[i] ? kInt8 | take(keep8, n) : take(keep, n);
    };
    for (auto& kv : hflevels) {
        const int level = kv.first;
        auto lay_out_all = [&](const ColLists& L, const std::vector<DirMats*>& of, const std::vector<char>& on) {
            for (size_t i = 0; i < L.key.size(); ++i) {
                DirMats& M = *of[L.key[i] / 8];
                if (!M.cached) lay_out(M.fin[L.key[i] % 8], (size_t)M.mrows * M.mcols, on, i);
            }
        };
        lay_out_all(cols.m2m.at(level), m2m_of, m2m_i8[level]);
        for (size_t i = 0; i < m2l_probs[level].size(); ++i) {
            M2LMat& M = m2l_mats[m2l_probs[level][i]];
            if (!M.pk) lay_out(M.fin, (size_t)M.r1 * M.r1, m2l_i8[level], i);
        }
        lay_out_all(cols.l2l.at(level), l2l_of, l2l_i8[level]);
    }
    phase("routes");
    // right factors E1, E2^T and E3^T as gatherable columns in the scratch pool
    std::vector<size_t> scr_E1(hfcanon.size()), scr_E2t(hfcanon.size()), scr_E3t(hfcanon.size());
    for (size_t c = 0; c < hfcanon.size(); ++c) {
        scr_E1[c] = take(scr, (size_t)hfcanon[c].r1 * hfcanon[c].r1);
        scr_E2t[c] = take(scr, (size_t)hfcanon[c].r1 * hfcanon[c].r2);
        scr_E3t[c] = take(scr, (size_t)hfcanon[c].r2 * hfcanon[c].r2);
    }
    double2* dkeep = dalloc<double2>(keep);
    double2* dkeep8 = keep8 ? dalloc<double2>(keep8) : nullptr;
    double2* dscr = nullptr;
    if (scr) CK(cudaMalloc(&dscr, sizeof(double2) * scr));
    flush_uploads();
    for (size_t c = 0; c < hfcanon.size(); ++c) {
        CK(cudaMemcpyAsync(dscr + scr_E1[c], hfcanon[c].E1, sizeof(double2) * hfcanon[c].r1 * hfcanon[c].r1,
                           cudaMemcpyDeviceToDevice, stream_));
        CK(cudaMemcpyAsync(dscr + scr_E2t[c], hfcanon[c].E2t, sizeof(double2) * hfcanon[c].r1 * hfcanon[c].r2,
                           cudaMemcpyDeviceToDevice, stream_));
        CK(cudaMemcpyAsync(dscr + scr_E3t[c], hfcanon[c].E3t, sizeof(double2) * hfcanon[c].r2 * hfcanon[c].r2,
                           cudaMemcpyDeviceToDevice, stream_));
    }
    for (auto& kv : m2m_mats) {
        if (kv.second.cached) continue;
        double W = kv.first.first;
        const DirPts& dp = get_dir(W, kv.first.second);
        int rc, cc;
        const double* cp = child_pts(W, kv.first.second, true, rc, cc);
        for (int ind = 0; ind < 8; ++ind)
            add_job(dp.ucp, zero3, cp, shifted_point(ind, W), dp.r2, rc, dscr + kv.second.raw[ind]);
    }
    for (auto& kv : l2l_mats) {
        if (kv.second.cached) continue;
        double W = kv.first.first;
        const DirPts& dp = get_dir(W, kv.first.second);
        int rc, cc;
        const double* cp = child_pts(W, kv.first.second, false, rc, cc);
        for (int ind = 0; ind < 8; ++ind)
            add_job(cp, shifted_point(ind, W), dp.dep, zero3, rc, dp.r2, dscr + kv.second.raw[ind]);
    }
    for (const M2LMat& M : m2l_mats)
        if (!M.pk) add_job(hfcanon[M.canon].neg_uep, M.shift, hfcanon[M.canon].uep, zero3, M.r1, M.r1, dscr + M.raw);

    phase("job_list");
    // generate every kernel matrix now
    if (!jobs.empty()) {
        KmatJob* d_jobs = upload(jobs);
        flush_uploads();
        launch_kmat(d_jobs, (int)jobs.size(), job_elems, kern, stream_);
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(stream_));
    }

    phase("kmat");
    // fold, in three rounds of products (raw doubles as scratch once read):
    //   M2M  tmp = ue2uc E1(child);  mid = E3 tmp (or E3 raw);  fin = E2 mid
    //   L2L  tmp = de2dc E3^T;       mid = E1(child)^T tmp;     fin = mid E2^T
    //   M2L  tmp = M E1;                                        fin = E1^T tmp
    if (scr) {
        GemmBatch right, left, last, last8;
        auto fold = [&](const double2* A, int m, int k, size_t bx, int n, size_t fin) {
            (fin & kInt8 ? last8 : last).product(A, m, k, bx, n, fin & ~kInt8);
        };
        for (auto& kv : m2m_mats) {
            const DirMats& M = kv.second;
            for (int ind = 0; ind < 8 && !M.cached; ++ind) {
                if (M.fin[ind] == kNone) continue;
                const bool hf = M.ccanon >= 0;  // else the children are low-frequency boxes
                const size_t in = hf ? M.tmp[ind] : M.raw[ind], mid = hf ? M.raw[ind] : M.tmp[ind];
                if (hf) right.product(dscr + M.raw[ind], M.rmid, M.mcols, scr_E1[M.ccanon], M.mcols, M.tmp[ind]);
                left.product(hfcanon[M.canon].E3, M.rmid, M.rmid, in, M.mcols, mid);
                fold(hfcanon[M.canon].E2, M.mrows, M.rmid, mid, M.mcols, M.fin[ind]);
            }
        }
        for (auto& kv : l2l_mats) {
            const DirMats& M = kv.second;
            for (int ind = 0; ind < 8 && !M.cached; ++ind) {
                if (M.fin[ind] == kNone) continue;
                const bool hf = M.ccanon >= 0;
                const size_t mid = hf ? M.raw[ind] : M.tmp[ind];
                right.product(dscr + M.raw[ind], M.mrows, M.rmid, scr_E3t[M.canon], M.rmid, M.tmp[ind]);
                if (hf) left.product(hfcanon[M.ccanon].E1t, M.mrows, M.mrows, M.tmp[ind], M.rmid, mid);
                fold(dscr + mid, M.mrows, M.rmid, scr_E2t[M.canon], M.mcols, M.fin[ind]);
            }
        }
        for (const M2LMat& M : m2l_mats) {
            if (M.pk) continue;
            right.product(dscr + M.raw, M.r1, M.r1, scr_E1[M.canon], M.r1, M.tmp);
            fold(hfcanon[M.canon].E1t, M.r1, M.r1, M.tmp, M.r1, M.fin);
        }
        right.run(dscr, dscr, stream_);
        left.run(dscr, dscr, stream_);
        last.run(dscr, dkeep, stream_);
        last8.run(dscr, dkeep8, stream_);
        CK(cudaStreamSynchronize(stream_));
        CK(cudaFree(dscr));
    }
    phase("fold");
    const double2* dkeepm = opm(dkeep, keep);
    auto KP = [&](size_t fin) { return fin & kInt8 ? dkeep8 + (fin & ~kInt8) : E((double2*)dkeepm, fin); };

    // ---------------------------------------------------------------- steps: LF upward
    auto lf_set = [&](const double* x, int n, Pt3 shift, double scale) {
        PtSet s;
        s.x = x;
        s.n = n;
        for (int d = 0; d < 3; ++d) s.shift[d] = shift[d];
        s.scale = scale;
        return s;
    };
    auto leaf_set = [&](int l) { return lf_set(d_pos_sorted_ + 3 * (size_t)leaf_off[l], leaf_cnt[l], zero3, 1.0); };
    auto single = [&](const GemmProblem& p, const std::vector<long long>& x, const std::vector<long long>& y,
                      const double2* X, double2* Y, int mode, const char* label) {
        std::vector<GemmProblem> ps(1, p);
        std::vector<std::vector<long long> > xo(1, x), yo(1, y);
        add_gemm(ps, xo, yo, X, Y, mode, label);
    };
    // y = B (A x) on the boxes at the given offsets: one launch where both operators fit
    // zgemm_pair_kernel and its 8-column blocks leave SMs free as zgemm_narrow_kernel's
    // would (K = 4, P = 4: two launches of 10.8 us event to event, one of 14.7; K = 16: 26.4
    // and 17.4 us), else two, whose wider tiles read the operators less often
    auto twice = [&](const double2* A, const double2* B, int r, const std::vector<long long>& at, const double2* X, double2* Y,
                     const char* label) {
        if (mixed || nE > GEMM_PAIR_MAX || r > GEMM_PAIR_MAX || at.empty() || (at.size() + 63) / 64 >= 148) {
            single(GemmProblem{opm(A, (size_t)r * nE), r, nE, r, 0, 0}, at, at, X, lf_mid, GEMM_SET, label);
            single(GemmProblem{opm(B, (size_t)r * nE), nE, r, nE, 0, 0}, at, at, lf_mid, Y, GEMM_SET, label);
            return;
        }
        Step st{};
        st.kind = 11;
        st.label = label;
        st.flops = 16.0 * r * nE * (double)at.size();
        st.bytes = 16.0 * (2.0 * r * nE + 2.0 * nE * (double)at.size());
        st.gp = GemmPair{A, B, nE, r, (int)at.size(), upload(at), X, Y};
        stats_.flops_gemm += st.flops;
        stats_.gemm_launches++;
        push_step(st);
    };
    for (auto it = lflevels.rbegin(); it != lflevels.rend(); ++it) {
        const LfLevelOps& L = lfops[it->first];
        const auto& ids = it->second;
        begin_block(0, L.W);
        // S2M at leaves (src/wave3d_eval.cpp:441-451)
        std::vector<PtItem> items;
        std::vector<PtSrc> srcs;
        for (int l : ids) {
            const Box& B = T.boxes[lfbox[l]];
            if (!B.terminal()) continue;
            PtItem itm;
            itm.trg = lf_set(L.ucp, nE, T.center(B), 1.0);
            itm.out = E(lf_upchk, (size_t)l * nE);
            itm.src_begin = (int)srcs.size();
            srcs.push_back(PtSrc{leaf_set(l), E(d_den_sorted_, leaf_off[l])});
            itm.src_end = (int)srcs.size();
            items.push_back(itm);
        }
        add_pt(items, srcs, "lf_s2m");
        // M2M from children (src/wave3d_eval.cpp:452-463) and, further down, L2L to them:
        // one launch for the 8 child positions, a problem each (an adaptive tree has many
        // levels of few boxes: 8 launches a level were half of such an eval's)
        if (L.has_children) {
            std::vector<GemmProblem> probs;
            std::vector<std::vector<long long> > x(8), y(8);
            for (int ind = 0; ind < 8; ++ind) {
                probs.push_back(GemmProblem{opm(L.ue2uc[ind], (size_t)nE * nE), nE, nE, nE, 0, 0});
                for (int l : ids) {
                    int b = lfbox[l];
                    if (T.boxes[b].terminal()) continue;
                    int c = T.child(b, ind);
                    if (c < 0 || !T.boxes[c].has_pts()) continue;
                    x[ind].push_back((long long)lfidx[c] * nE);
                    y[ind].push_back((long long)l * nE);
                }
            }
            if (!up.v.empty() || !dn.v.empty()) {
                add_gemm(probs, x, y, lf_upeq, lf_upchk, GEMM_ATOMIC, "lf_m2m");  // siblings add into one parent
            } else {
                // no high-frequency passes (K = 1, 2): nothing else of an eval adds in an order
                // of its own, so without atomics here a matvec repeats bit for bit
                for (int ind = 0; ind < 8; ++ind) single(probs[ind], x[ind], y[ind], lf_upeq, lf_upchk, GEMM_ADD, "lf_m2m");
            }
        }
        // upeqnden = v * (1/sigma .* (U^H * upchk))   (src/wave3d_eval.cpp:466-478)
        std::vector<long long> a;
        for (int l : ids) a.push_back((long long)l * nE);
        twice(L.up_s, L.v, L.r, a, lf_upchk, lf_upeq, "lf_uc2ue");
    }

    phase("steps_lf_up");
    // ---------------------------------------------------------------- digits of the HF inputs
    // (mixed form: FP16 planes) of the vectors that the products on those routes gather
    Digits lf_dg;
    std::map<int, Digits> up_dg, dn_dg;  // by level
    char* dg_X8 = nullptr;               // of the high-frequency levels
    size_t dg_bytes = 0;
    {
        const size_t gb = umma() ? H16_GRANULE : I8_GRANULE, cb = umma() ? sizeof(float) : sizeof(double);
        lf_dg.unit = nE;
        lf_dg.gran = (nE + 15) / 16;
        if (lf_i8) {
            lf_dg.X8 = dalloc<char>((size_t)nLF * lf_dg.gran * gb);
            lf_dg.cx = dalloc<char>((size_t)nLF * lf_dg.gran * cb);
        }
        // Outgoing digits of a level are read by the M2M above it and last by its M2L, then
        // its incoming ones are written and read by its L2L: one place for both.
        auto place = [&](const HfNodes& N, int level, long long total, Digits& d) {  // base; granules of the level
            const auto r = N.range.at(level);
            if (r.first == r.second) return (size_t)0;
            d.base = N.v[r.first].off;
            return (size_t)((r.second == (int)N.v.size() ? total : N.v[r.second].off) - d.base) / 16;
        };
        size_t granules = 0;
        std::map<int, size_t> at;
        for (auto& kv : hflevels) {
            const int level = kv.first;
            at[level] = granules;
            const size_t u = up_i8.count(level) ? place(up, level, upeq_total, up_dg[level]) : 0;
            const size_t d = dn_i8.count(level) ? place(dn, level, dnchk_total, dn_dg[level]) : 0;
            granules += std::max(u, d);
        }
        if (granules) {
            dg_bytes = granules * gb;
            dg_X8 = dalloc<char>(dg_bytes);
            char* cx = dalloc<char>(granules * cb);
            for (std::map<int, Digits>* m : {&up_dg, &dn_dg})
                for (auto& kv : *m) {
                    kv.second.X8 = dg_X8 + at[kv.first] * gb;
                    kv.second.cx = cx + at[kv.first] * cb;
                }
        }
        if (!mixed && (lf_i8 || granules)) i8_init();
    }
    phase("digit_buffers");
    // Profiles of the outgoing vectors (kernels_i8.cu).  Incoming vectors are flat as they are.
    if (profiled && !up_i8.empty()) {
        int stride = 0;
        for (const Canon& c : hfcanon) stride = std::max(stride, (c.r1 + 15) & ~15);
        std::vector<unsigned char> prof;
        for (const Canon& c : hfcanon) {
            std::vector<double> size(c.r1, 0.0);
            for (int j = 0; j < c.r1; ++j) {
                for (int i = 0; i < c.r1; ++i) {
                    const cpx& e = c.op->E1(i, j);
                    size[j] = std::max(size[j], std::max(std::fabs(e.real()), std::fabs(e.imag())));
                }
                size[j] = 1.0 / size[j];
            }
            const std::vector<unsigned char> row = i8_profile(size.data(), c.r1, stride);
            prof.insert(prof.end(), row.begin(), row.end());
        }
        profiles_ = I8Profiles{upload(prof), stride};
    }
    auto add_node_digits = [&](const HfNodes& N, int level, const double2* X, const Digits& d, const char* label) {
        const bool profile = profiled && &N == &up;
        const auto r = N.range.at(level);
        const size_t n = (size_t)(r.second - r.first);
        std::unique_ptr<I8Vec[]> v(new I8Vec[n]);  // not zeroed first
        host_parallel_for((n + 16383) / 16384, [&](size_t c) {
            for (size_t i = c * 16384; i < std::min(n, (c + 1) * 16384); ++i) {
                const HfNode& u = N.v[r.first + i];
                v[i] = I8Vec{u.off, (int)((u.off - d.base) / 16), (unsigned short)hfcanon[u.canon].r1,
                             (unsigned short)(profile ? u.canon + 1 : 0)};
            }
        });
        add_digits(v.get(), n, X, d, label);
    };
    // ---------------------------------------------------------------- steps: HF upward
    // widths ascending = levels descending; hf_upeq holds w (upeqnden = E1 w)
    for (auto hit = hflevels.rbegin(); hit != hflevels.rend(); ++hit) {
        int level = hit->first;
        double W = T.width(level);
        auto ur = up.range[level];
        if (ur.first == ur.second) continue;
        begin_block(1, W);
        if (W == 1.0 && lf_i8) {
            std::vector<I8Vec> v;
            for (int l : lflevels[level + 1]) v.push_back(I8Vec{(long long)l * nE, l * lf_dg.gran, (unsigned short)nE, 0});
            add_digits(v.data(), v.size(), lf_upeq, lf_dg, "lf_digits");
        }
        // M2M: w = sum_children [E2 E3 ue2uc E1(child)] w_child (src/wave3d_eval.cpp:796-849),
        // one launch for the 8 child positions: a problem per (wedge, child), all adding into
        // the parents' vectors
        {
            ColLists& L = cols.m2m.at(level);
            std::vector<GemmProblem> probs;
            for (int k : L.key) {
                const Idx3& dir = did_wedge[k / 8].second;
                const int ind = k % 8;
                const DirMats& M = m2m_mats.at(std::make_pair(W, dir));
                if (M.cached) {
                    probs.push_back(GemmProblem{nullptr, M.mrows, M.mcols, M.mrows, 0, 0, M.pk[ind]});
                } else {
                    probs.push_back(GemmProblem{KP(M.fin[ind]), M.mrows, M.mcols, M.mrows, 0, 0, nullptr, profiled ? M.ccanon + 1 : 0});
                    if (!opctx_.empty()) opkey_[KP(M.fin[ind])] = opk("m2m", W, dir, ind);
                }
            }
            add_gemm(probs, L.x, L.y, W == 1.0 ? lf_upeq : hf_upeq, hf_upeq, GEMM_ATOMIC, width_label("hf_m2m", W),
                     W == 1.0 ? &lf_dg : &up_dg[level + 1], &m2m_i8[level]);
        }
        if (up_i8.count(level)) add_node_digits(up, level, hf_upeq, up_dg[level], "hf_digits_up");
    }

    phase("steps_hf_up");
    // ---------------------------------------------------------------- steps: HF downward
    // widths descending = levels ascending; hf_dnchk holds u = E1^T dnchkval
    for (auto it = hflevels.begin(); it != hflevels.end(); ++it) {
        int level = it->first;
        double W = T.width(level);
        auto dr = dn.range[level];
        if (dr.first == dr.second) continue;
        begin_block(2, W);
        // M2L (src/wave3d_eval.cpp:876-928)
        {
            std::vector<GemmProblem> probs;
            for (int gid : m2l_probs[level]) {
                const M2LMat& M = m2l_mats[gid];
                if (M.pk) {
                    probs.push_back(GemmProblem{nullptr, M.r1, M.r1, M.r1, 0, 0, M.pk});
                } else {
                    probs.push_back(GemmProblem{KP(M.fin), M.r1, M.r1, M.r1, 0, 0, nullptr, profiled ? M.canon + 1 : 0});
                    if (!opctx_.empty()) opkey_[KP(M.fin)] = M.key;
                }
            }
            add_gemm(probs, m2l_x[level], m2l_y[level], hf_upeq, hf_dnchk, GEMM_ATOMIC, width_label("hf_m2l", W),
                     &up_dg[level], &m2l_i8[level]);
        }
        if (dn_i8.count(level)) add_node_digits(dn, level, hf_dnchk, dn_dg[level], "hf_digits_down");
        // L2L into the children's (pdir) u, or LF dnchkval at W=1 (src/wave3d_eval.cpp:938-991),
        // one launch for the 8 child positions: a problem per (wedge, child)
        {
            ColLists& L = cols.l2l.at(level);
            std::vector<GemmProblem> probs;
            for (int k : L.key) {
                const Idx3& dir = did_wedge[k / 8].second;
                const int ind = k % 8;
                const DirMats& M = l2l_mats.at(std::make_pair(W, dir));
                if (M.cached) {
                    probs.push_back(GemmProblem{nullptr, M.mrows, M.mcols, M.mrows, 0, 0, M.pk[ind]});
                } else {
                    probs.push_back(GemmProblem{KP(M.fin[ind]), M.mrows, M.mcols, M.mrows, 0, 0});
                    if (!opctx_.empty()) opkey_[KP(M.fin[ind])] = opk("l2l", W, dir, ind);
                }
            }
            add_gemm(probs, L.x, L.y, hf_dnchk, W == 1.0 ? lf_dnchk : hf_dnchk, GEMM_ATOMIC, width_label("hf_l2l", W),
                     &dn_dg[level], &l2l_i8[level]);
        }
    }

    phase("steps_hf_down");
    // Small instances do not fill the GPU in any pass: their V-list sums and near field
    // run beside the high-frequency passes (run_steps).  The line is the size of the
    // summed target spectra, which then need memory of their own.  One stream / with branches,
    // by that size: plain 8 MB 325 / 287 us, 31 MB 1284 / 1237, 105 MB 3098 / 3024, a cluster
    // with 36 MB 1111 / 663; mixed 53 MB 1206 / 1145, 67 MB 1535 / 1422.  At the line it is even
    // (plain K = 32: 123 MB 5313 / 5440, 133 MB 3726 / 3588), above it nothing (mixed 207 MB
    // 4508 / 4461 us, 832 MB 17.54 / 17.58 ms).
    overlap_ = !hflevels.empty() && !lflevels.empty() && (size_t)nLF * G3 * es <= ((size_t)128 << 20);
    if (overlap_) {
        branch_.resize(std::min<size_t>(lflevels.size(), kBranches));
        for (cudaStream_t& b : branch_) CK(cudaStreamCreateWithFlags(&b, cudaStreamNonBlocking));
        branch_ev_.resize(2 + 2 * branch_.size() + 2 * lflevels.size());
        for (cudaEvent_t& e : branch_ev_) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    // Source spectra: each eval writes every one it reads.  Where no pass overlaps another the
    // high-frequency passes are over by then, and their digits' memory will do.
    const size_t spec_bytes = (size_t)nLF * G3 * es;
    double2* lf_spec = !overlap_ && spec_bytes <= dg_bytes ? (double2*)dg_X8 : salloc((size_t)nLF * G3);
    // ---------------------------------------------------------------- steps: LF downward
    for (auto& kv : lflevels) {  // levels ascending = widths descending
        int level = kv.first;
        const LfLevelOps& L = lfops[level];
        const auto& ids = kv.second;
        double W = L.W;
        // the widest level's check values also receive the high-frequency L2L, atomically:
        // what adds to them otherwise waits for it on the main stream
        const Step::Lane below = kv.first == lflevels.begin()->first ? Step::MAIN : Step::SIDE_LATE;
        begin_block(3, W);
        // V list: FFT M2L (src/wave3d_eval.cpp:602-661).  The pointwise sums run by
        // target parent (kernels.cuh, VlistGroups): the targets of a parent share one
        // pass over the union of their V-list sources; then one inverse transform
        // per target.
        {
            const auto tv = std::chrono::steady_clock::now();
            VlistGroupPlan vg = vlist_groups(T, lfbox, lfidx, ids);
            t_emit_vgroups_ += std::chrono::duration<double>(std::chrono::steady_clock::now() - tv).count();
            stats_.v_pairs += vg.pairs;
            const std::vector<int>& trg = vg.trg;
            if (!trg.empty()) {
                const std::vector<int>& srcb = vg.src;
                VlistLevel VL{G, P, nE, L.cube_idx, L.tns, d_twf, d_twb};  // FP32 data in the mixed form
                Step f{};
                f.kind = 2;
                f.label = "lf_vlist_fft";
                f.flops = 8.0 * 3 * (double)G3 * G * srcb.size();
                f.bytes = 16.0 * ((double)nE + G3) * srcb.size();
                f.v.L = VL;
                f.v.src_boxes = upload(srcb);
                f.v.nsrc = (int)srcb.size();
                f.v.upeq = lf_upeq;
                f.v.spec = lf_spec;
                if (mixed) {
                    f.hvf = VfSub{VL, f.v.src_boxes, reinterpret_cast<const float2*>(lf_upeq),
                                  reinterpret_cast<float2*>(lf_spec), f.v.nsrc, 0};
                    set_multi(f, f.hvf, f.v.nsrc);
                }
                lane_ = Step::SIDE_LATE;
                push_step(f);
                // summed target spectra, of their own where the sums may overlap the
                // high-frequency passes; else a high-frequency buffer when one is large enough
                // (every high-frequency pass has run before this low-frequency downward
                // step, so the outgoing densities and the incoming check values are free
                // by then), else a buffer of their own
                const size_t tsp_elems = trg.size() * (size_t)G3;
                double2* tsp = overlap_                           ? salloc(tsp_elems)
                               : tsp_elems <= (size_t)upeq_total  ? hf_upeq
                               : tsp_elems <= (size_t)dnchk_total ? hf_dnchk
                                                                  : salloc(tsp_elems);
                const int ngroups = (int)vg.gptr.size() - 1;
                const long long npairs = vg.pairs;
                Step a{};
                a.kind = 3;
                a.label = "lf_vlist_m2l";
                a.flops = 8.0 * (double)G3 * npairs;
                // compulsory: each source spectrum, the 316 tensors, each target's summed spectrum
                a.bytes = 16.0 * ((double)G3 * srcb.size() + 316.0 * G3 + (double)G3 * trg.size());
                a.v.L = VL;
                a.v.grp = VlistGroups{upload(vg.gptr), reinterpret_cast<const int2*>(upload(vg.gsrc)), upload(vg.gtrg),
                                      ngroups};
                a.v.spec = lf_spec;
                a.v.tsp = tsp;
                if (mixed) {
                    a.hva = VaSub{VL, a.v.grp.gptr, a.v.grp.gsrc, a.v.grp.gtrg, reinterpret_cast<const float2*>(lf_spec),
                                  reinterpret_cast<float2*>(tsp), ngroups, 0};
                    set_multi(a, a.hva, ngroups);
                }
                push_step(a);
                lane_ = below;
                Step iv{};
                iv.kind = 6;
                iv.label = "lf_vlist_inv";
                iv.flops = 8.0 * (double)G * ((double)G * G * P + G * P * P + P * P * P) * trg.size();
                iv.bytes = 16.0 * ((double)G3 + 2.0 * nE) * trg.size();
                iv.v.L = VL;
                iv.v.trg = upload(trg);
                iv.v.ntrg = (int)trg.size();
                iv.v.tsp = tsp;
                iv.v.dnchk = lf_dnchk;
                if (mixed) {
                    iv.hvi = ViSub{VL, iv.v.trg, reinterpret_cast<const float2*>(tsp), reinterpret_cast<float2*>(lf_dnchk),
                                   iv.v.ntrg, 0};
                    set_multi(iv, iv.hvi, iv.v.ntrg);
                }
                push_step(iv);
                lane_ = Step::MAIN;
            }
        }
        // X list (src/wave3d_eval.cpp:663-686), into dnchk or, for small leaves, into extval
        {
            std::vector<PtItem> itemsA, itemsB;
            std::vector<PtSrc> srcsA, srcsB;
            for (int l : ids) {
                const Box& B = T.boxes[lfbox[l]];
                if (B.xlist.empty()) continue;
                bool direct = B.terminal() && leaf_cnt[l] < nE;
                PtItem itm;
                itm.trg = direct ? leaf_set(l) : lf_set(L.uep, nE, T.center(B), 1.0);
                itm.out = direct ? E(d_val_sorted_, leaf_off[l]) : E(lf_dnchk, (size_t)l * nE);
                auto& S = direct ? srcsA : srcsB;
                itm.src_begin = (int)S.size();
                for (int s : B.xlist) {
                    int ls = lfidx[s];
                    S.push_back(PtSrc{leaf_set(ls), E(d_den_sorted_, leaf_off[ls])});
                    stats_.x_pairs++;
                }
                itm.src_end = (int)S.size();
                (direct ? itemsA : itemsB).push_back(itm);
            }
            lane_ = Step::SIDE_EARLY;
            add_pt(itemsA, srcsA, "lf_xlist");
            lane_ = below;
            add_pt(itemsB, srcsB, "lf_xlist");
            lane_ = Step::MAIN;
        }
        // U list (src/wave3d_eval.cpp:585-600) and W list (:688-718) into extval
        {
            std::vector<PtItem> items, witems;
            std::vector<PtSrc> srcs, wsrcs;
            for (int l : ids) {
                const Box& B = T.boxes[lfbox[l]];
                if (!B.ulist.empty()) {
                    PtItem itm;
                    itm.trg = leaf_set(l);
                    itm.out = E(d_val_sorted_, leaf_off[l]);
                    itm.src_begin = (int)srcs.size();
                    for (int s : B.ulist) {
                        int ls = lfidx[s];
                        srcs.push_back(PtSrc{leaf_set(ls), E(d_den_sorted_, leaf_off[ls])});
                        stats_.u_pairs++;
                        stats_.u_interactions += (long long)leaf_cnt[l] * leaf_cnt[ls];
                    }
                    itm.src_end = (int)srcs.size();
                    items.push_back(itm);
                }
                if (!B.wlist.empty()) {
                    PtItem itm;
                    itm.trg = leaf_set(l);
                    itm.out = E(d_val_sorted_, leaf_off[l]);
                    itm.src_begin = (int)wsrcs.size();
                    for (int s : B.wlist) {
                        int ls = lfidx[s];
                        const Box& SB = T.boxes[s];
                        if (SB.terminal() && leaf_cnt[ls] < nE) {
                            wsrcs.push_back(PtSrc{leaf_set(ls), E(d_den_sorted_, leaf_off[ls])});
                        } else {
                            double coef = T.width(SB.level) / W;
                            wsrcs.push_back(PtSrc{lf_set(L.uep, nE, T.center(SB), coef), E(lf_upeq, (size_t)ls * nE)});
                        }
                        stats_.w_pairs++;
                    }
                    itm.src_end = (int)wsrcs.size();
                    witems.push_back(itm);
                }
            }
            lane_ = Step::SIDE_EARLY;
            add_pt(items, srcs, "lf_ulist");
            lane_ = Step::SIDE_LATE;
            add_pt(witems, wsrcs, "lf_wlist");
            lane_ = Step::MAIN;
        }
        // dneqnden = up^T (1/sigma .* (v^T dnchk))   (src/wave3d_eval.cpp:536-547, src/mlib3d.cpp:147-152)
        std::vector<long long> a;
        for (int l : ids) a.push_back((long long)l * nE);
        twice(L.vT_s, L.upT, L.r, a, lf_dnchk, lf_dneq, "lf_dc2de");
        // L2T at leaves (src/wave3d_eval.cpp:550-560)
        {
            std::vector<PtItem> items;
            std::vector<PtSrc> srcs;
            for (int l : ids) {
                const Box& B = T.boxes[lfbox[l]];
                if (!B.terminal()) continue;
                PtItem itm;
                itm.trg = leaf_set(l);
                itm.out = E(d_val_sorted_, leaf_off[l]);
                itm.src_begin = (int)srcs.size();
                srcs.push_back(PtSrc{lf_set(L.ucp, nE, T.center(B), 1.0), E(lf_dneq, (size_t)l * nE)});
                itm.src_end = (int)srcs.size();
                items.push_back(itm);
            }
            add_pt(items, srcs, "lf_l2t");
        }
        // L2L to the children (src/wave3d_eval.cpp:562-579)
        if (L.has_children) {
            std::vector<GemmProblem> probs;
            std::vector<std::vector<long long> > x(8), y(8);
            for (int ind = 0; ind < 8; ++ind) {
                probs.push_back(GemmProblem{opm(L.de2dc[ind], (size_t)nE * nE), nE, nE, nE, 0, 0});
                for (int l : ids) {
                    int b = lfbox[l];
                    if (T.boxes[b].terminal()) continue;
                    int c = T.child(b, ind);
                    if (c < 0 || !T.boxes[c].has_pts()) continue;
                    x[ind].push_back((long long)l * nE);
                    y[ind].push_back((long long)lfidx[c] * nE);
                }
            }
            add_gemm(probs, x, y, lf_dneq, lf_dnchk, GEMM_ADD, "lf_l2l");  // every child has one parent
        }
    }
    phase("steps_lf_down");
    if (trace)
        std::fprintf(stderr,
                     "ddfmm setup   (host seconds in GEMM step emission %.3f, V-list grouping %.3f, uploads above "
                     "64 KB %.3f, operator packing %.3f of which chunk allocation %.3f; %lld device allocations "
                     "%.3f, %lld staged copies: waits %.3f, host copies %.3f)\n",
                     t_emit_gemm_, t_emit_vgroups_, t_big_uploads_, t_pack_, t_pack_alloc_, n_malloc_, t_malloc_,
                     n_stage_, t_stage_wait_, t_stage_copy_);
    flush_packs();
    if (dkeep8) {  // packed as digits by now
        CK(cudaStreamSynchronize(stream_));
        dfree(dkeep8);
    }
    if (mixed) {
        // the mixed eval reads only the FP32 copies (and, on tcgen05, only the packed
        // GEMM operators): release the FP64 operators and the unpacked GEMM copies
        CK(cudaStreamSynchronize(stream_));
        std::set<const void*> vlist32{d_twf, d_twb};
        for (auto& kv : lfops) vlist32.insert(kv.second.tns);
        for (auto& kv : op32) {
            dfree(kv.first);
            if (umma() && !vlist32.count(kv.second)) dfree(kv.second);
        }
    }
    flush_uploads();
    CK(cudaStreamSynchronize(stream_));
    stage_release();
    std::vector<char>().swap(arena_.host);  // every chunk is on the device now
    arena_.retired.clear();
    arena_.used = arena_.sent = arena_.cap;
    phase("packs_release");
    stats_.kernel_launches = (long long)steps_.size() + 2;
}

static const char* kernel_name(int kind, int tpi, bool narrow) {
    switch (kind) {
        case 0: return narrow ? "zgemm_narrow_kernel" : "zgemm_kernel";
        case 1:
            switch (tpi) {  // the launch shape the autotuner chose
                case 4: return "pt_kernel<4>";
                case 8: return "pt_kernel<8>";
                case 16: return "pt_kernel<16>";
                case PT_WARP_TARGETS: return "ptw_kernel<targets,4>";
                case PT_WARP_TARGETS2: return "ptw_kernel<targets,2>";
                case PT_WARP_SOURCES: return "ptw_kernel<sources,8>";
                case PT_WARP_SOURCES4: return "ptw_kernel<sources,4>";
                default: return "pt_kernel<32>";
            }
        case 2: return "vlist_forward_kernel";
        case 3: return "vlist_group_kernel";
        case 6: return "vlist_inverse_kernel";
        case 7: return "i8_slice_kernel";
        case 8: return "i8_gemm_kernel";
        case 9: return "h16_slice_kernel";
        case 10: return "h16_gemm_kernel";
        case 11: return "zgemm_pair_kernel";
        default: return "umma_cgemm_kernel";
    }
}

void Session::launch_step(const Step& st, cudaStream_t s, double2* spec) {
    const bool m = mixed();
    unsigned long long stall_ns = 0;  // failure-path hook: one launch only
    if (stall_wait_ns_ && st.kind == stall_kind_) std::swap(stall_ns, stall_wait_ns_);
    switch (st.kind) {
        case 0:
            if (m)
                launch_cgemm(st.g.probs, st.g.tiles, st.g.ntiles, st.g.xoff, st.g.yoff, st.g.X, st.g.Y, st.g.mode, s);
            else if (st.g.rows)
                launch_gemm_narrow(st.g.probs, st.g.tiles, st.g.ntiles, st.g.xoff, st.g.yoff, st.g.X, st.g.Y, st.g.mode,
                                   st.g.kmax, st.g.rows, s);
            else
                launch_gemm(st.g.probs, st.g.tiles, st.g.ntiles, st.g.xoff, st.g.yoff, st.g.X, st.g.Y, st.g.mode, s);
            break;
        case 1:
            if (m)
                launch_pt32(static_cast<const PtSub*>(st.msubs), st.mpre, 1, st.mtotal, nullptr, s, st.tpi ? st.tpi : 32);
            else
                launch_pt(st.pt.items, st.pt.nitems, st.pt.srcs, prm_.kernel, s, st.tpi ? st.tpi : 32);
            break;
        case 2:
            if (m)
                launch_vlist_forward32(static_cast<const VfSub*>(st.msubs), st.mpre, 1, st.mtotal, st.v.L.G, nullptr,
                                       spec != st.v.spec ? spec : nullptr, s, &st.hvf);
            else
                launch_vlist_forward(st.v.L, st.v.src_boxes, st.v.nsrc, st.v.upeq, spec, s);
            break;
        case 3:
            if (m)
                launch_vlist_group32(static_cast<const VaSub*>(st.msubs), st.mpre, 1, st.mtotal, st.v.L.G, nullptr,
                                     spec != st.v.spec ? spec : nullptr, s, &st.hva);
            else
                launch_vlist_group(st.v.L, st.v.grp, spec, st.v.tsp, s);
            break;
        case 6:
            if (m)
                launch_vlist_inverse32(static_cast<const ViSub*>(st.msubs), st.mpre, 1, st.mtotal, st.v.L.G, nullptr, s,
                                       &st.hvi);
            else
                launch_vlist_inverse(st.v.L, st.v.trg, st.v.ntrg, st.v.tsp, st.v.dnchk, s);
            break;
        case 7: launch_i8_slice(st.dg.vecs, st.dg.n, st.dg.X, st.dg.X8, st.dg.cx, st.dg.prof, s); break;
        case 8: launch_i8_gemm(st.i8, d_err_, s, stall_ns, stall_ns > 0); break;
        case 11: launch_gemm_pair(st.gp, s); break;
        case 9:
            launch_h16_slice(static_cast<const HSliceSub*>(st.msubs), st.mpre, 1, st.mtotal, nullptr, s, st.hs);
            break;
        case 10:
            launch_h16_gemm(static_cast<const HSub*>(st.msubs), st.mpre, 1, st.mtotal, nullptr, d_err_, s, st.hh,
                            nullptr, stall_ns, stall_ns > 0);
            break;
        case 5:
            launch_umma_cgemm(static_cast<const UmmaSub*>(st.msubs), st.mpre, 1, st.mtotal, nullptr, d_err_, s, &st.hu,
                              stall_ns, stall_ns > 0);
            break;
    }
}

// The accumulators a point-interaction step writes are zeroed at the start of
// every eval, so running it here on setup-time contents is harmless.
void Session::autotune() {
    cudaEvent_t a = nullptr, b = nullptr;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    for (Step& st : steps_) {
        if (st.kind != 1) continue;
        static const std::vector<int> shapes{32, 16, 8, 4, PT_WARP_TARGETS, PT_WARP_TARGETS2, PT_WARP_SOURCES,
                                             PT_WARP_SOURCES4};
        float best = 0.f;
        int best_tpi = shapes[0];
        // per-launch time of one shape over `reps` launches after a warm-up
        auto time_shape = [&](int reps) {
            launch_step(st, stream_, st.v.spec);
            CK(cudaEventRecord(a, stream_));
            for (int r = 0; r < reps; ++r) launch_step(st, stream_, st.v.spec);
            CK(cudaEventRecord(b, stream_));
            CK(cudaEventSynchronize(b));
            float ms = 0.f;
            CK(cudaEventElapsedTime(&ms, a, b));
            return ms / reps;
        };
        for (int tpi : shapes) {
            st.tpi = tpi;
            float ms = time_shape(3);
            // short steps: time over ~0.5 ms of launches, or three launches read mostly noise
            if (ms * 3 < 0.5f) ms = time_shape(std::min(50, (int)(0.5f / std::max(ms, 1e-3f)) + 1));
            if (tpi == shapes[0] || ms < best) {
                best = ms;
                best_tpi = tpi;
            }
        }
        st.tpi = best_tpi;
        stats_.tuned_steps++;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    CK(cudaGetLastError());
}

void Session::run_steps(cudaStream_t s) {
    if (graph_ && !profiling_ && !stall_wait_ns_) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        CK(cudaStreamIsCapturing(s, &cap));
        if (cap == cudaStreamCaptureStatusNone) {
            CK(cudaGraphLaunch(graph_, s));
            return;
        }
    }
    for (const Memset& m : zero_at_start_) CK(cudaMemsetAsync(m.p, 0, m.bytes, s));
    if (profiling_ && ev_.size() < 2 * steps_.size()) {
        size_t have = ev_.size();
        ev_.resize(2 * steps_.size());
        for (size_t i = have; i < ev_.size(); ++i) CK(cudaEventCreate(&ev_[i]));
    }
    if (profiling_ && !ev_pending_.empty()) profile_read();  // keep one eval of events in flight at most
    if (overlap_ && !profiling_) {
        run_overlapped(s);
        return;
    }
    for (size_t i = 0; i < steps_.size(); ++i) {
        const Step& st = steps_[i];
        if (profiling_) CK(cudaEventRecord(ev_[2 * i], s));
        launch_step(st, s, st.v.spec);
        if (profiling_) {
            CK(cudaEventRecord(ev_[2 * i + 1], s));
            ev_pending_.push_back(std::make_pair((int)i, (int)(2 * i)));
        }
    }
}

// The steps with a branch (stream) per low-frequency level beside the caller's
// stream.  A level's branch runs, in the serial order, its S2M (the finest level's
// stays on the main stream, which starts with it), its U and direct X lists, and once
// the upward low-frequency passes are done its V-list transforms and sums, W list and,
// below the widest level, what adds into its check values; then its L2T, once the main
// stream has the level's densities.  Every one of them writes values, check values or
// spectra of its own level's boxes, and before the join nothing on the main stream
// touches those.  Works on a capturing stream: the branches join the capture at the
// fork and leave it at the last join.  An adaptive tree of five levels (cluster, K = 8)
// takes 530 us with one side stream for all levels, 496 with a branch each (a first,
// cold eval 907 and 728).
void Session::run_overlapped(cudaStream_t s) {
    const size_t nb = branch_.size();
    auto level = [](const Step& st) {  // 0 for the widest
        const int w = (int)((st.key >> 32) & 0xffff);
        return (st.key >> 48) < 2 ? 999 - w : w - 1001;
    };
    auto branch = [&](const Step& st) { return branch_[(size_t)level(st) % nb]; };
    size_t used = 0;
    auto after = [&](cudaStream_t to, cudaStream_t from) {  // `to` goes on once `from` has come here
        CK(cudaEventRecord(branch_ev_[used], from));
        CK(cudaStreamWaitEvent(to, branch_ev_[used], 0));
        ++used;
    };
    auto all_after = [&]() {
        CK(cudaEventRecord(branch_ev_[used], s));
        for (cudaStream_t b : branch_) CK(cudaStreamWaitEvent(b, branch_ev_[used], 0));
        ++used;
    };
    const int finest = level(steps_[0]);
    auto apart = [&](const Step& st) {  // S2M of the levels that others come before, L2T of those that others follow
        const int pass = (int)(st.key >> 48);
        return st.kind == 1 && level(st) != finest && (pass == 0 || (pass == 3 && !std::strcmp(st.label, "lf_l2t")));
    };
    all_after();
    std::map<int, size_t> s2m;  // level -> event
    for (const Step& st : steps_)
        if ((st.key >> 48) == 0 && apart(st)) {
            launch_step(st, branch(st), st.v.spec);
            CK(cudaEventRecord(branch_ev_[used], branch(st)));
            s2m[level(st)] = used++;
        }
    for (const Step& st : steps_)
        if (st.lane == Step::SIDE_EARLY) launch_step(st, branch(st), st.v.spec);
    size_t i = 0;
    for (; i < steps_.size() && (steps_[i].key >> 48) == 0; ++i) {
        auto e = s2m.find(level(steps_[i]));
        if (e != s2m.end()) {
            CK(cudaStreamWaitEvent(s, branch_ev_[e->second], 0));
            s2m.erase(e);
        }
        if (!apart(steps_[i])) launch_step(steps_[i], s, steps_[i].v.spec);
    }
    all_after();
    for (const Step& st : steps_)
        if (st.lane == Step::SIDE_LATE) launch_step(st, branch(st), st.v.spec);
    for (; i < steps_.size() && (steps_[i].key >> 48) < 3; ++i) launch_step(steps_[i], s, steps_[i].v.spec);
    for (cudaStream_t b : branch_) after(s, b);
    std::set<cudaStream_t> open;  // branches with an L2T on them
    for (; i < steps_.size(); ++i) {
        const Step& st = steps_[i];
        if (st.lane != Step::MAIN) continue;
        if (!apart(st)) {
            launch_step(st, s, st.v.spec);
            continue;
        }
        after(branch(st), s);
        launch_step(st, branch(st), st.v.spec);
        open.insert(branch(st));
    }
    for (cudaStream_t b : open) after(s, b);
}

// Everything between the densities' gather and the values' scatter (whose arrays are
// the caller's) as one graph: a small instance's eval otherwise spends as long on
// its 25 to 100 runtime calls as the GPU does on their work (K = 4, P = 4: 64 -> 59 us a
// matvec, a K = 8 cluster 565 -> 534 us).
void Session::build_graph() {
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
    try {
        run_steps(stream_);
    } catch (...) {
        cudaStreamEndCapture(stream_, &g);
        if (g) cudaGraphDestroy(g);
        throw;
    }
    CK(cudaStreamEndCapture(stream_, &g));
    const cudaError_t e = cudaGraphInstantiate(&graph_, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) graph_ = nullptr;
    CK(e);
    CK(cudaGraphUpload(graph_, stream_));  // the first eval should not pay for it
}

void Session::profile_enable(bool on) {
    if (!on && !ev_pending_.empty()) profile_read();
    profiling_ = on;
}

std::vector<Session::ProfileEntry> Session::profile_read() {
    for (auto& pe : ev_pending_) {
        CK(cudaEventSynchronize(ev_[pe.second + 1]));
        float ms = 0;
        CK(cudaEventElapsedTime(&ms, ev_[pe.second], ev_[pe.second + 1]));
        const Step& st = steps_[pe.first];
        ProfileEntry& e = prof_[st.label];
        e.label = st.label;
        e.kernel = kernel_name(st.kind, st.tpi, st.g.rows > 0);
        e.launches += 1;
        e.ms += ms;
        e.flops += st.flops;
        e.bytes += st.bytes;
    }
    ev_pending_.clear();
    // in launch order: by the first step of each label
    std::vector<ProfileEntry> out;
    std::set<std::string> seen;
    for (const Step& st : steps_) {
        auto it = prof_.find(st.label);
        if (it != prof_.end() && seen.insert(st.label).second) out.push_back(it->second);
    }
    return out;
}

void Session::eval_device(const double2* den, double2* val, cudaStream_t s) {
    if (mixed())
        launch_gather32(den, d_perm_, d_den_sorted_, npts_, 0, s);
    else
        launch_gather_den(den, d_perm_, d_den_sorted_, npts_, s);
    run_steps(s);
    if (mixed())
        launch_scatter32(d_val_sorted_, d_perm_, val, npts_, 0, d_err_, s);
    else
        launch_scatter_val(d_val_sorted_, d_perm_, val, npts_, d_err_, s);
    CK(cudaGetLastError());
}

void Session::eval_device_c64(const float2* den, float2* val, cudaStream_t s) {
    if (!mixed()) throw std::invalid_argument("complex64 evaluation needs a mixed-precision session");
    launch_gather32(den, d_perm_, d_den_sorted_, npts_, 1, s);
    run_steps(s);
    launch_scatter32(d_val_sorted_, d_perm_, val, npts_, 1, d_err_, s);
    CK(cudaGetLastError());
}

void Session::eval_host_c64(const std::complex<float>* den, std::complex<float>* val) {
    if (!mixed()) throw std::invalid_argument("complex64 evaluation needs a mixed-precision session");
    CK(cudaMemcpyAsync(d_den_io_, den, sizeof(float2) * npts_, cudaMemcpyHostToDevice, stream_));
    eval_device_c64((const float2*)d_den_io_, (float2*)d_val_io_, stream_);
    CK(cudaMemcpyAsync(val, d_val_io_, sizeof(float2) * npts_, cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    check_device_error();
}

// run_steps with the V-list launches on `spec` for the spectra, no profiling.
void Session::run_steps_spec(cudaStream_t s, double2* spec) {
    for (const Memset& m : zero_at_start_) CK(cudaMemsetAsync(m.p, 0, m.bytes, s));
    for (const Step& st : steps_) launch_step(st, s, spec);
}

void Session::eval_device_scratch(const double2* den, double2* val, cudaStream_t s, double2* spec, size_t capacity) {
    const size_t es = mixed() ? sizeof(float2) : sizeof(double2);
    if (spectra_elems_ * es > capacity * sizeof(double2)) {
        char msg[200];
        snprintf(msg, sizeof msg,
                 "the session's V-list spectra need %.1f MiB, more than the %.1f MiB of fixed scratch",
                 spectra_elems_ * es / 1048576.0, capacity * sizeof(double2) / 1048576.0);
        throw std::invalid_argument(msg);
    }
    if (mixed())
        launch_gather32(den, d_perm_, d_den_sorted_, npts_, 0, s);
    else
        launch_gather_den(den, d_perm_, d_den_sorted_, npts_, s);
    run_steps_spec(s, spec);
    if (mixed())
        launch_scatter32(d_val_sorted_, d_perm_, val, npts_, 0, d_err_, s);
    else
        launch_scatter_val(d_val_sorted_, d_perm_, val, npts_, d_err_, s);
    CK(cudaGetLastError());
}

void Session::eval_host(const std::complex<double>* den, std::complex<double>* val) {
    CK(cudaMemcpyAsync(d_den_io_, den, sizeof(double2) * npts_, cudaMemcpyHostToDevice, stream_));
    eval_device(d_den_io_, d_val_io_, stream_);
    CK(cudaMemcpyAsync(val, d_val_io_, sizeof(double2) * npts_, cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    check_device_error();
}

void Session::direct_host(const std::complex<double>* den, const int* ids, int nids, std::complex<double>* out) {
    if (nids <= 0) return;
    for (int i = 0; i < nids; ++i)
        if (ids[i] < 0 || ids[i] >= npts_) throw std::runtime_error("check id out of range");
    int* d_ids = nullptr;
    double2* d_out = nullptr;
    CK(cudaMalloc(&d_ids, sizeof(int) * nids));
    CK(cudaMalloc(&d_out, sizeof(double2) * nids));
    CK(cudaMemcpyAsync(d_den_io_, den, sizeof(double2) * npts_, cudaMemcpyHostToDevice, stream_));
    CK(cudaMemcpyAsync(d_ids, ids, sizeof(int) * nids, cudaMemcpyHostToDevice, stream_));
    launch_direct(d_pos_ids_, d_den_io_, npts_, d_ids, nids, d_out, prm_.kernel, stream_);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(out, d_out, sizeof(double2) * nids, cudaMemcpyDeviceToHost, stream_));
    CK(cudaStreamSynchronize(stream_));
    cudaFree(d_ids);
    cudaFree(d_out);
}

}  // namespace ddfmm
