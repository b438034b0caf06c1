// One complex product through a session's GEMM kernels (test entry point
// ddfmm_test_gemm): what a translation of an eval runs, on the caller's matrices.
#include <cuda_runtime.h>

#include <cmath>
#include <stdexcept>
#include <string>
#include <vector>

#include "kernels.cuh"

namespace ddfmm {

namespace {
void ck(cudaError_t e) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error: ") + cudaGetErrorString(e));
}
struct Pool {  // device copies, freed together
    std::vector<void*> p;
    ~Pool() {
        for (void* q : p) cudaFree(q);
    }
    template <class T>
    T* put(const std::vector<T>& v) {
        T* d = nullptr;
        ck(cudaMalloc(&d, sizeof(T) * (v.empty() ? 1 : v.size())));
        p.push_back(d);
        if (!v.empty()) ck(cudaMemcpy(d, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice));
        return d;
    }
};
}  // namespace

// Y (m x ncol) += A (m x k) X (k x ncol), all column-major complex; the columns
// are gathered from and scattered to padded vectors in reverse order.
void test_gemm(const double2* A, int m, int k, const double2* X, int ncol, int path, double2* Y) {
    Pool P;
    const int kx = path == 8 ? m : k;  // length of an input vector
    const int sx = (kx + 15) / 16 * 16, sy = (m + 15) / 16 * 16;
    std::vector<double2> hx((size_t)sx * ncol, make_double2(0, 0)), hy((size_t)sy * ncol, make_double2(0, 0));
    std::vector<long long> xo(ncol), yo(ncol);
    std::vector<int> xg(ncol);
    std::vector<I8Vec> vecs(ncol);
    for (int c = 0; c < ncol; ++c) {
        const int at = ncol - 1 - c;
        xo[c] = (long long)at * sx;
        yo[c] = (long long)at * sy;
        xg[c] = at * (sx / 16);
        vecs[c] = I8Vec{xo[c], xg[c], (unsigned short)k, (unsigned short)(path >= 6)};
        for (int i = 0; i < kx; ++i) hx[xo[c] + i] = X[(size_t)c * kx + i];
        for (int i = 0; i < m; ++i) hy[yo[c] + i] = Y[(size_t)c * m + i];
    }
    const double2* dA = P.put(std::vector<double2>(A, A + (size_t)m * k));
    const double2* dX = P.put(hx);
    double2* dY = P.put(hy);
    const long long* dyo = P.put(yo);
    I8Profiles prof{nullptr, sx};
    if (path == 6 || path == 7) {  // the columns as one class of vectors
        std::vector<double> size(k, 0.0);
        for (size_t e = 0; e < (size_t)k * ncol; ++e)
            size[e % k] = std::fmax(size[e % k], std::fmax(std::fabs(X[e].x), std::fabs(X[e].y)));
        prof.prof = P.put(i8_profile(size.data(), k, sx));
    }
    if (path == 0) {
        std::vector<GemmTile> tiles;
        for (int r = 0; r < m; r += GEMM_TILE_M)
            for (int c = 0; c < ncol; c += GEMM_TILE_N) tiles.push_back(GemmTile{0, r, c, 0});
        gemm_init();
        launch_gemm(P.put(std::vector<GemmProblem>(1, GemmProblem{dA, m, k, m, 0, ncol, nullptr})), P.put(tiles),
                    (int)tiles.size(), P.put(xo), dyo, dX, dY, GEMM_ATOMIC, nullptr);
    } else if (path == 2) {
        const int rows = m > 64 ? 128 : 64;
        std::vector<GemmTile> tiles;
        for (int r = 0; r < m; r += rows)
            for (int c = 0; c < ncol; c += 8) tiles.push_back(GemmTile{0, r, c, 0});
        gemm_init();
        launch_gemm_narrow(P.put(std::vector<GemmProblem>(1, GemmProblem{dA, m, k, m, 0, ncol, nullptr})), P.put(tiles),
                           (int)tiles.size(), P.put(xo), dyo, dX, dY, GEMM_ATOMIC, k, rows, nullptr);
    } else if (path == 5) {  // the identity, then A, at the offsets of both
        if (m != k || m > GEMM_PAIR_MAX) throw std::invalid_argument("the pair kernel takes square operators of up to 64 rows");
        std::vector<double2> one((size_t)m * m, make_double2(0, 0));
        for (int i = 0; i < m; ++i) one[(size_t)i * m + i] = make_double2(1, 0);
        launch_gemm_pair(GemmPair{P.put(one), dA, m, m, ncol, P.put(xo), dX, dY}, nullptr);
    } else if (path == 8) {  // the transpose of A, then A
        if (m > GEMM_PAIR_MAX || k > GEMM_PAIR_MAX) throw std::invalid_argument("the pair kernel takes up to 64 rows and columns");
        std::vector<double2> t((size_t)m * k);
        for (int i = 0; i < m; ++i)
            for (int j = 0; j < k; ++j) t[(size_t)i * k + j] = A[(size_t)j * m + i];
        launch_gemm_pair(GemmPair{P.put(t), dA, m, k, ncol, P.put(xo), dX, dY}, nullptr);
    } else if (path == 3 || path == 4 || path == 7) {  // mixed form, on FP32 copies: 3 FP16 planes, 4 split TF32
        auto narrow = [](const std::vector<double2>& v) {
            std::vector<float2> r;
            for (const double2& a : v) r.push_back(make_float2((float)a.x, (float)a.y));
            return r;
        };
        const float2* fA = P.put(narrow(std::vector<double2>(A, A + (size_t)m * k)));
        const float2* fX = P.put(narrow(hx));
        std::vector<float2> fy = narrow(hy);
        float2* fY = P.put(fy);
        int* err = P.put(std::vector<int>(1, 0));
        if (path != 4) {
            float* B = P.put(std::vector<float>(h16_packed_floats(m, k)));
            char* X16 = P.put(std::vector<char>((size_t)ncol * (sx / 16) * H16_GRANULE));
            float* cx = P.put(std::vector<float>((size_t)ncol * (sx / 16)));
            std::vector<H16Tile> tiles;
            h16_tiles(B, m, k, 0, ncol, tiles);
            h16_init();
            launch_h16_pack(P.put(std::vector<H16PackJob>(1, H16PackJob{fA, B, const_cast<float*>(h16_scales(B, m, k)), m, k,
                                                                        m, h16_tile_rows(m), prof.prof})),
                            1, h16_row_tiles(m), nullptr);
            launch_h16_slice(nullptr, nullptr, 1, ncol, nullptr, nullptr, HSliceSub{P.put(vecs), fX, X16, cx, ncol, 0, prof});
            launch_h16_gemm(nullptr, nullptr, 1, (int)tiles.size(), nullptr, err, nullptr,
                            HSub{P.put(tiles), P.put(xg), dyo, X16, cx, fY, (int)tiles.size(), 0});
        } else {
            float* B = P.put(std::vector<float>(umma_packed_floats(m, k)));
            std::vector<UmmaTile> tiles;
            for (int r = 0; r * 128 < m; ++r)
                for (int c = 0; c < ncol; c += 128) tiles.push_back(UmmaTile{0, r, r * 128, m - r * 128 < 128 ? m - r * 128 : 128, c, 0});
            umma_init();
            launch_umma_pack(P.put(std::vector<UmmaPackJob>(1, UmmaPackJob{fA, B, umma_tile_stride(k), m, k, m, umma_nkb(k)})),
                             1, nullptr);
            const UmmaSub one{P.put(std::vector<UmmaProblem>(1, UmmaProblem{B, umma_tile_stride(k), m, k, umma_nkb(k), 0, ncol})),
                              P.put(tiles), P.put(xo), dyo, fX, fY, (int)tiles.size(), GEMM_ATOMIC, 0, 0};
            launch_umma_cgemm(nullptr, nullptr, 1, (int)tiles.size(), nullptr, err, nullptr, &one);
        }
        int h = 0;
        ck(cudaMemcpy(&h, err, sizeof(int), cudaMemcpyDeviceToHost));
        if (h) throw std::runtime_error("CUDA error: a tensor-core GEMM timed out waiting on its pipeline");
        ck(cudaGetLastError());
        ck(cudaMemcpy(fy.data(), fY, sizeof(float2) * fy.size(), cudaMemcpyDeviceToHost));
        for (int c = 0; c < ncol; ++c)
            for (int i = 0; i < m; ++i) Y[(size_t)c * m + i] = make_double2(fy[yo[c] + i].x, fy[yo[c] + i].y);
        return;
    } else {
        const int nkb = (k + 15) / 16;
        char* B = P.put(std::vector<char>(i8_packed_bytes(m, k)));
        double* ra = P.put(std::vector<double>(m));
        char* X8 = P.put(std::vector<char>((size_t)ncol * (sx / 16) * I8_GRANULE));
        double* cx = P.put(std::vector<double>((size_t)ncol * (sx / 16)));
        std::vector<I8Tile> tiles;
        i8_tiles(B, ra, m, k, 0, ncol, tiles);
        int* err = P.put(std::vector<int>(1, 0));
        i8_init();
        launch_i8_pack(P.put(std::vector<I8PackJob>(1, I8PackJob{dA, B, ra, m, k, m, nkb, i8_tile_rows(m), prof.prof})), 1,
                       i8_row_tiles(m), nullptr);
        launch_i8_slice(P.put(vecs), ncol, dX, X8, cx, prof, nullptr);
        launch_i8_gemm(I8Sub{P.put(tiles), P.put(xg), dyo, X8, cx, dY, (int)tiles.size()}, err, nullptr);
        int h = 0;
        ck(cudaMemcpy(&h, err, sizeof(int), cudaMemcpyDeviceToHost));
        if (h) throw std::runtime_error("CUDA error: the int8 GEMM timed out waiting on its pipeline");
    }
    ck(cudaGetLastError());
    ck(cudaMemcpy(hy.data(), dY, sizeof(double2) * hy.size(), cudaMemcpyDeviceToHost));
    for (int c = 0; c < ncol; ++c)
        for (int i = 0; i < m; ++i) Y[(size_t)c * m + i] = hy[yo[c] + i];
}

}  // namespace ddfmm
