// Driver of the grid-wide conjugate gradient (built and run by
// tests/test_gpu_cg_grid.py): one system solved by the kernel that keeps R
// rows per thread in registers and by the one that keeps none, on the same
// blocks, so that each thread owns the same rows and every sum is formed in
// the same order. Prints the iterations and the number of entries of the
// solution whose bits differ.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

namespace {
#include "cg_grid.cuh"
}

#define TRY(x)                                                             \
    do {                                                                   \
        const cudaError_t e = (x);                                         \
        if (e != cudaSuccess) {                                            \
            std::printf("error %s: %s\n", #x, cudaGetErrorString(e));      \
            return 2;                                                      \
        }                                                                  \
    } while (0)

template <typename T>
T *upload(const std::vector<T> &v) {
    T *p = nullptr;
    if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess) return nullptr;
    if (cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) return nullptr;
    return p;
}

int main(int argc, char **argv) {
    if (argc != 4) return 2;
    const int w = std::atoi(argv[1]), h = std::atoi(argv[2]), R = std::atoi(argv[3]);
    int n = w * h, sms = 0;
    TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0));
    const int blocks = (n + kGridCgThreads * R - 1) / (kGridCgThreads * R);
    if (R < 1 || R > 4 || w < 2 || h < 2 || blocks > sms || blocks > kGridCgBlocks) return 2;
    // five-point Laplacian of a w x h grid with uneven couplings, in ELL form
    std::vector<int> col((size_t)kEll * n);
    std::vector<double> val((size_t)kEll * n, 0.0), dinv(n), b(n), x0(n, 0.0);
    auto coupling = [](int i, int j) { return 1.0 + 0.37 * ((i < j ? i * 31 + j : j * 31 + i) % 17) / 17.0; };
    for (int i = 0; i < n; i++) {
        const int cx = i % w, cy = i / w;
        int e = 1;
        double diag = 1e-3;
        auto add = [&](int j) {
            col[(size_t)e * n + i] = j;
            val[(size_t)e * n + i] = -coupling(i, j);
            diag += coupling(i, j);
            e++;
        };
        if (cx > 0) add(i - 1);
        if (cx + 1 < w) add(i + 1);
        if (cy > 0) add(i - w);
        if (cy + 1 < h) add(i + w);
        for (; e < kEll; e++) col[(size_t)e * n + i] = i;
        col[i] = i;
        val[i] = diag;
        dinv[i] = 1.0 / diag;
        b[i] = ((i * 7919LL) % 1013) / 1013.0 - 0.4;
    }
    const int *dcol = upload(col);
    const double *dval = upload(val), *ddinv = upload(dinv), *db = upload(b);
    double *x = upload(x0), *r = upload(x0), *z = upload(x0), *p0 = upload(x0), *p1 = upload(x0);
    double *scal = upload(std::vector<double>(kGridCgDoubles, 0.0));
    if (!dcol || !dval || !ddinv || !db || !x || !r || !z || !p0 || !p1 || !scal) return 2;
    std::vector<double> got[2] = {x0, x0};
    double out[2][2];
    for (int k = 0; k < 2; k++) {
        TRY(cudaMemcpy(x, x0.data(), n * sizeof(double), cudaMemcpyHostToDevice));
        TRY(cudaMemset(scal, 0, kGridCgDoubles * sizeof(double)));
        unsigned *cnt = (unsigned *)(scal + 16);
        double2 *sums = (double2 *)(scal + 32);
        double rtol = 1e-10, eta = 0.0;
        int maxit = 400;
        const double *t1 = nullptr;
        void *args[] = {&n, &dcol, &dval, &ddinv, &db, &x, &r, &z, &p0, &p1, &scal, &cnt, &sums, &rtol, &eta, &maxit, &t1};
        const void *fn = k == 0   ? (const void *)k_cg_grid<0>
                         : R == 1 ? (const void *)k_cg_grid<1>
                         : R == 2 ? (const void *)k_cg_grid<2>
                         : R == 3 ? (const void *)k_cg_grid<3>
                                  : (const void *)k_cg_grid<4>;
        TRY(cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kGridCgThreads), args, 0, 0));
        TRY(cudaDeviceSynchronize());
        TRY(cudaMemcpy(got[k].data(), x, n * sizeof(double), cudaMemcpyDeviceToHost));
        TRY(cudaMemcpy(out[k], scal, sizeof(out[k]), cudaMemcpyDeviceToHost));
    }
    int differ = 0;
    for (int i = 0; i < n; i++) differ += std::memcmp(&got[0][i], &got[1][i], sizeof(double)) != 0;
    std::printf("blocks %d iterations %.0f %.0f differ %d\n", blocks, out[0][1], out[1][1], differ);
    return 0;
}
