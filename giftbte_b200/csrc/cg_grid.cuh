// The grid-wide conjugate gradient of the macro systems. Included by solver.cu
// inside its anonymous namespace.
#pragma once

// Jacobi-preconditioned CG of a system too large for one cluster, one
// cooperative launch for the whole solve. The rows are held in ELL form
// (kEll columns, padding: value 0 on the row itself) and spread over the
// grid's threads, row i0 + k * (threads) for k < R.
//
// What bounds it is the latency of the grid-wide sums (about 2,400 clocks of
// barrier and 500 of reads and adds each), so an iteration has two of them
// and nothing else that waits: a thread forms the new search
// direction p = z + beta p_old for itself and, in the product A p, for its
// neighbours too (p alternates between two buffers), so p needs no barrier
// of its own. With R > 0 a thread's matrix rows and its entries of x, r, p and A p
// stay in registers for the whole solve and only z and p go through L2; R = 0
// serves more rows than registers hold (p is then updated in place, behind a
// third barrier). x, r, z and p get the same values either way: z = D^-1 r is
// rounded before p = z + beta p_old, which is one fused step, for a thread's
// own rows as for its neighbours' (left to the compiler, a thread's own p took
// the product unrounded, so x moved along another p than A was applied to).
// Per iteration 8.06 -> 5.63 us on 48,000 cells, 17.0 -> 7.52 us on 196,608,
// against a CSR loop with three barriers and atomic sums (whose order, and
// bits, varied).
constexpr int kEll = 5;             // a tetrahedron's or quadrilateral's row: itself and four neighbours
constexpr int kGridCgThreads = 512;
constexpr int kGridCgBlocks = 1024;  // most blocks (entries of one exchange)
constexpr int kGridCgTries = 1 << 22;
// device memory of the exchanges: {sum of (x - t1)^2, iterations}, the
// arrival counter, then two sets of kGridCgBlocks pairs of sums
constexpr size_t kGridCgDoubles = 32 + 2 * (size_t)kGridCgBlocks * 2;

// Sums v1, v2 over the grid, the same bits on every thread: every block
// stores its pair of sums and counts itself in; past the last arrival each
// block reads all pairs and adds them in block order. Epochs alternate
// between two sets of pairs: a block stores epoch e + 2 only after every
// block has arrived at e + 1, that is after every block has read epoch e.
// One thread per block polls the counter (every thread polling its own
// block's flag took twice to three times as long on 94 to 148 blocks). Data
// written before the call is visible to loads that bypass L1 (__ldcg) after
// it. False when a block did not arrive within kGridCgTries polls; the
// caller then stops (uniformly over the block).
__device__ __forceinline__ bool grid_sum2(double &v1, double &v2, unsigned epoch, unsigned *cnt, double2 *sums) {
    __shared__ double sw[2][32];
    __shared__ double2 sb[kGridCgBlocks];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5, G = gridDim.x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v1 += __shfl_xor_sync(0xffffffffu, v1, o);
        v2 += __shfl_xor_sync(0xffffffffu, v2, o);
    }
    if (lane == 0) sw[0][warp] = v1, sw[1][warp] = v2;
    __syncthreads();
    double2 *set = sums + (epoch & 1) * kGridCgBlocks;
    bool lost = false;
    if (warp == 0) {
        v1 = lane < nw ? sw[0][lane] : 0.0;
        v2 = lane < nw ? sw[1][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v1 += __shfl_xor_sync(0xffffffffu, v1, o);
            v2 += __shfl_xor_sync(0xffffffffu, v2, o);
        }
        if (lane == 0) {
            __stcg(set + blockIdx.x, make_double2(v1, v2));
            __threadfence();
            atomicAdd(cnt, 1u);
            const unsigned want = epoch * (unsigned)G;
            unsigned got = 0;
            for (int t = 0; t < kGridCgTries; t++) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(cnt) : "memory");
                if (got >= want) break;
            }
            lost = got < want;
        }
    }
    if (__syncthreads_or(lost)) return false;
    for (int k = tid; k < G; k += blockDim.x) sb[k] = __ldcg(set + k);
    __syncthreads();
    v1 = v2 = 0;
    for (int k = lane; k < G; k += 32) v1 += sb[k].x, v2 += sb[k].y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v1 += __shfl_xor_sync(0xffffffffu, v1, o);
        v2 += __shfl_xor_sync(0xffffffffu, v2, o);
    }
    return true;
}

// Stops when |r| <= max(rtol |b|, eta |r0|): rtol is the absolute floor,
// eta bounds the reduction needed from a warm start. out[0] = the sum of
// (x - t1)^2 (t1 may be null), out[1] = iterations, -1 if an exchange was lost.
template <int R>
__global__ void __launch_bounds__(kGridCgThreads, 1)
    k_cg_grid(int n, const int *__restrict__ col, const double *__restrict__ val, const double *__restrict__ dinv,
              const double *__restrict__ b, double *__restrict__ x, double *r_, double *z, double *p0, double *p1,
              double *out, unsigned *cnt, double2 *sums, double rtol, double eta, int maxit,
              const double *__restrict__ t1) {
    constexpr int RR = R > 0 ? R : 1;
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x, st = gridDim.x * blockDim.x;
    unsigned epoch = 0;
    int jc[RR][kEll];
    double av[RR][kEll], xr[RR], rr_[RR], di[RR], pr[RR], Ap[RR];
    bool ok = true;
    double rz = 0, bb = 0, rr = 0, zero = 0;
    // r = b - A x, z = D^-1 r
    auto start = [&](int i, double &r) {
        double ax = 0;
#pragma unroll
        for (int e = 0; e < kEll; e++) ax += val[(size_t)e * n + i] * x[col[(size_t)e * n + i]];
        r = b[i] - ax;
        const double zi = dinv[i] * r;
        z[i] = zi;
        rz += r * zi;
        bb += b[i] * b[i];
        rr += r * r;
        return zi;
    };
    if constexpr (R > 0) {
#pragma unroll
        for (int k = 0; k < R; k++) {
            const int i = i0 + k * st;
            rr_[k] = xr[k] = di[k] = pr[k] = Ap[k] = 0;
            if (i >= n) continue;
#pragma unroll
            for (int e = 0; e < kEll; e++) jc[k][e] = col[(size_t)e * n + i], av[k][e] = val[(size_t)e * n + i];
            xr[k] = x[i];
            di[k] = dinv[i];
            start(i, rr_[k]);
        }
    } else {
        for (int i = i0; i < n; i += st) {
            double r;
            p0[i] = start(i, r);
            r_[i] = r;
        }
    }
    ok = grid_sum2(rz, bb, ++epoch, cnt, sums);
    if (ok) ok = grid_sum2(rr, zero, ++epoch, cnt, sums);
    const double thr = fmax(rtol * rtol * bb, eta * eta * rr);
    double beta = 0;
    int it = 0;
    while (ok && it < maxit && rr > thr) {
        double pap = 0, rzn = 0, rrn = 0;
        zero = 0;
        if constexpr (R > 0) {
            const double *po = it & 1 ? p1 : p0;
            double *pn = it & 1 ? p0 : p1;
#pragma unroll
            for (int k = 0; k < R; k++) {
                const int i = i0 + k * st;
                if (i >= n) continue;
                double zj[kEll], pj[kEll], s = 0;
#pragma unroll
                for (int e = 0; e < kEll; e++) {
                    zj[e] = __ldcg(z + jc[k][e]);
                    pj[e] = it ? __ldcg(po + jc[k][e]) : 0.0;
                }
#pragma unroll
                for (int e = 0; e < kEll; e++) s = __fma_rn(av[k][e], __fma_rn(beta, pj[e], zj[e]), s);
                pr[k] = __fma_rn(beta, pr[k], __dmul_rn(di[k], rr_[k]));
                __stcg(pn + i, pr[k]);
                Ap[k] = s;
                pap += pr[k] * s;
            }
        } else {
            for (int i = i0; i < n; i += st) {
                double s = 0;
#pragma unroll
                for (int e = 0; e < kEll; e++)
                    s = __fma_rn(val[(size_t)e * n + i], __ldcg(p0 + col[(size_t)e * n + i]), s);
                p1[i] = s;  // A p, read back by this thread only
                pap += __ldcg(p0 + i) * s;
            }
        }
        ok = grid_sum2(pap, zero, ++epoch, cnt, sums);
        if (!ok) break;
        const double alpha = rz / pap;
        if constexpr (R > 0) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                const int i = i0 + k * st;
                if (i >= n) continue;
                xr[k] += alpha * pr[k];
                const double ri = rr_[k] - alpha * Ap[k];
                rr_[k] = ri;
                const double zi = __dmul_rn(di[k], ri);
                __stcg(z + i, zi);
                rzn += ri * zi;
                rrn += ri * ri;
            }
        } else {
            for (int i = i0; i < n; i += st) {
                x[i] += alpha * __ldcg(p0 + i);
                const double ri = r_[i] - alpha * p1[i];
                r_[i] = ri;
                const double zi = dinv[i] * ri;
                z[i] = zi;
                rzn += ri * zi;
                rrn += ri * ri;
            }
        }
        ok = grid_sum2(rzn, rrn, ++epoch, cnt, sums);
        if (!ok) break;
        beta = rzn / rz;
        rz = rzn;
        rr = rrn;
        if constexpr (R == 0) {
            for (int i = i0; i < n; i += st) __stcg(p0 + i, __fma_rn(beta, __ldcg(p0 + i), z[i]));
            double d1 = 0, d2 = 0;
            ok = grid_sum2(d1, d2, ++epoch, cnt, sums);
        }
        it++;
    }
    double sq = 0;
    zero = 0;
    if constexpr (R > 0) {
#pragma unroll
        for (int k = 0; k < R; k++) {
            const int i = i0 + k * st;
            if (i >= n) continue;
            x[i] = xr[k];
            if (t1) sq += (xr[k] - t1[i]) * (xr[k] - t1[i]);
        }
    } else if (t1) {
        for (int i = i0; i < n; i += st) sq += (x[i] - t1[i]) * (x[i] - t1[i]);
    }
    if (ok && t1) ok = grid_sum2(sq, zero, ++epoch, cnt, sums);
    if (i0 == 0) {
        out[0] = sq;
        out[1] = ok ? (double)it : -1.0;
    }
}
