// Second-order transport through face values: the gradient kernel writes one
// upwind value per face instead of DIM gradient components per cell, and the
// residual reads four rows instead of a gather of neighbours' values and
// gradients. Included by solver.cu inside its anonymous namespace.
#pragma once

// 16-byte pieces of a band row: 4 FP32 or 2 FP64 bands
template <typename S>
constexpr int kPieceBands = 16 / (int)sizeof(S);

template <typename S, int N>
__device__ __forceinline__ void ld_piece(const S *p, S (&v)[N]) {
    static_assert(N * sizeof(S) == 16, "one 16-byte piece");
    if constexpr (sizeof(S) == 4) {
        const float4 a = *reinterpret_cast<const float4 *>(p);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    } else {
        const double2 a = *reinterpret_cast<const double2 *>(p);
        v[0] = a.x, v[1] = a.y;
    }
}
template <typename S, int N>
__device__ __forceinline__ void st_piece(S *p, const S (&v)[N]) {
    static_assert(N * sizeof(S) == 16, "one 16-byte piece");
    if constexpr (sizeof(S) == 4)
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else
        *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
}

// A stencil entry and a face of the block, as the kernel stages them: the
// weights (or the offset from the cell centre to the face centre) in the
// storage precision with, in the last word, the byte offset of the
// neighbour's row in the tile (or the face's slot).
template <typename S, int DIM> struct FaceW;
template <int DIM> struct alignas(16) FaceW<float, DIM> { float x, y, z; int at; };
template <> struct alignas(16) FaceW<double, 3> { double x, y, z; int at, pad; };
template <> struct alignas(16) FaceW<double, 2> { double x, y; int at, pad[3]; };
static_assert(sizeof(FaceW<float, 2>) == face_entry_bytes(4) && sizeof(FaceW<float, 3>) == face_entry_bytes(4) &&
                  sizeof(FaceW<double, 2>) == face_entry_bytes(8) && sizeof(FaceW<double, 3>) == face_entry_bytes(8),
              "the host sizes the tiles");

// Which side of every face its upwind value comes from: bit j of
// mask[d][c] is set when cell c writes the value of its face j in direction
// d. On an interior face the side-0 cell decides by the sign of s.n on its
// own normal, so exactly one of the two cells writes; on a wall face the
// cell writes where the direction leaves it (s.n >= 0).
template <int DIM>
__global__ void __launch_bounds__(256) k_face_mask(DMesh m, DPhys p, unsigned char *__restrict__ mask) {
    const int nc = m.nc;
    const size_t total = (size_t)p.nd * nc;
    for (size_t t = gtid(); t < total; t += gstride()) {
        const int c = (int)(t % nc);
        const size_t d = t / nc;
        const double sx = p.sx[d], sy = p.sy[d], sz = p.sz[d];
        const int k0 = m.cf_ptr[c], k1 = m.cf_ptr[c + 1];
        unsigned bits = 0;
        for (int k = k0; k < k1; k++) {
            const int ks = m.cf_bound[k] < 0 ? m.f_cf0[m.cf_face[k]] : k;
            const double sn = sx * m.cf_nx[ks] + sy * m.cf_ny[ks] + (DIM == 3 ? sz * m.cf_nz[ks] : 0.0);
            if ((sn >= 0) == (ks == k)) bits |= 1u << (k - k0);
        }
        mask[t] = (unsigned char)bits;
    }
}

// loads from a shared-memory address (32-bit); what they read was written by
// ordinary stores and by cp.async, hence the clobber
__device__ __forceinline__ void lds(unsigned a, float (&v)[4]) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "r"(a)
                 : "memory");
}
__device__ __forceinline__ void lds(unsigned a, double (&v)[2]) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void lds(unsigned a, FaceW<float, 2> &t) {
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=r"(t.at)
                 : "r"(a)
                 : "memory");
}
__device__ __forceinline__ void lds(unsigned a, FaceW<float, 3> &t) {
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=r"(t.at)
                 : "r"(a)
                 : "memory");
}
__device__ __forceinline__ void lds(unsigned a, FaceW<double, 2> &t) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(t.x), "=d"(t.y) : "r"(a) : "memory");
    asm volatile("ld.shared.b32 %0, [%1+16];" : "=r"(t.at) : "r"(a) : "memory");
}
__device__ __forceinline__ void lds(unsigned a, FaceW<double, 3> &t) {
    double w;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(t.x), "=d"(t.y) : "r"(a) : "memory");
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2+16];" : "=d"(t.z), "=d"(w) : "r"(a) : "memory");
    t.at = __double2loint(w);
}

// LSQ gradient and upwind face values of a block of B consecutive cells.
//
// The batch's rows are cut into slabs of W * NP 16-byte pieces that run
// across directions (piece P of the batch is piece P % ppd of direction
// P / ppd, ppd = nb * sizeof(S) / 16), so a slab is full whatever the band
// count. One CTA walks `per` slabs of one block. The block's stencil entries
// and faces are staged in shared memory once; the rows of the block's union
// (its cells and every stencil neighbour) follow slab by slab with 16-byte
// cp.async. W lanes share a cell, each with NP pieces of its row.
//
// Per band and direction the gradient is k_gradient8's, entry by entry in
// the same order, and the face value y = e + g . r is k_residual8's; a cell
// writes the faces its mask names to F[batch direction][face][band], and,
// for the outgoing wall values that follow the sweep, its gradient to
// gw[batch direction][wall slot][DIM][band] for each of its wall faces.
//
// What bounds it are the shared loads and the staging: a row load serves 128
// bands of a stencil entry in four wavefronts, the entry itself costs about two
// and a half however few cells share it. Several pieces per lane (NP) share the
// entry; in 3D the slab they need would leave one CTA per SM, so NP = 1 there.
// In 3D the pipe is 64% busy and a quarter of the warps are there to cover the
// loads' latency and the next slab's copies; in 2D it is 70% busy.
// Writing face values instead of gradients leaves its time where the tiled
// gradient's was (17,939 triangles x 40 x 64 FP32: 0.23 -> 0.25 ms; 48,000
// tetrahedra x 40 x 128 FP32: 4.85 -> 4.85 ms; 12,000 FP64: 3.18 -> 2.85 ms);
// the gain is the residual's.
template <typename S, int DIM, int W, int NP>
__global__ void __launch_bounds__(256, DIM == 2 ? 4 : 2)
    k_grad_face(DMesh m, int nb, const float4 *__restrict__ pk,
                const int *__restrict__ tile_ptr, const int *__restrict__ tile_cells,
                const unsigned short *__restrict__ tile_loc, int B, int qmax, int umax,
                const unsigned char *__restrict__ mask, const int *__restrict__ cf_gw, int nws,
                const S *__restrict__ eps, S *__restrict__ F, S *__restrict__ gw, int d0, int ndb, int per) {
    constexpr int VE = kPieceBands<S>, SW = W * NP, RB = SW * 16;  // pieces and bytes of a staged row
    constexpr int U = NP == 1 ? 4 : 2;                             // stencil entries in flight
    using FW = FaceW<S, DIM>;
    extern __shared__ __align__(16) unsigned char fsm[];
    FW *wq = reinterpret_cast<FW *>(fsm);
    FW *fq = wq + qmax;                                    // [B][4] faces
    unsigned char *rows = reinterpret_cast<unsigned char *>(fq + 4 * B);  // [umax][SW] pieces
    int *uoff = reinterpret_cast<int *>(rows + (size_t)umax * RB);
    const unsigned wq_s = (unsigned)__cvta_generic_to_shared(wq), rows_s = (unsigned)__cvta_generic_to_shared(rows);
    const int nc = m.nc, nf = m.nf, blk = blockIdx.x;
    const int c0 = blk * B, c1 = min(c0 + B, nc), ncell = c1 - c0;
    const int qb0 = m.nbr_ptr[c0], qb1 = m.nbr_ptr[c1];
    const int u0 = tile_ptr[blk], nu = tile_ptr[blk + 1] - u0;
    const int tid = threadIdx.x, bd = blockDim.x;
    for (int q = qb0 + tid; q < qb1; q += bd) {
        FW t;
        if constexpr (sizeof(S) == 4) {
            const float4 a = pk[q];
            t.x = a.x, t.y = a.y, t.z = a.z;
        } else {
            t.x = m.lsq_w[3 * q], t.y = m.lsq_w[3 * q + 1];
            if constexpr (DIM == 3) t.z = m.lsq_w[3 * q + 2];
        }
        t.at = (int)tile_loc[q] * RB;
        wq[q - qb0] = t;
    }
    const int i = tid / W, l = tid % W;  // cell of the block, lane of the cell
    const bool active = i < ncell;
    const int c = c0 + (active ? i : 0);
    const int k0 = m.cf_ptr[c], nface = active ? m.cf_ptr[c + 1] - k0 : 0;
    bool wall = false;
    for (int j = 0; j < nface; j++) {
        const int k = k0 + j;
        wall |= m.cf_bound[k] >= 0;
        if (l == 0) {
            FW t;
            S rx, ry, rz;
            face_off<S, DIM>(m, k, c, true, rx, ry, rz);
            t.x = rx, t.y = ry;
            if constexpr (DIM == 3 || sizeof(S) == 4) t.z = rz;
            t.at = m.cf_face[k] * nb;
            fq[4 * i + j] = t;
        }
    }
    for (int u = tid; u < nu; u += bd) uoff[u] = tile_cells[u0 + u] * nb;
    const unsigned wa = wq_s + (unsigned)(m.nbr_ptr[c] - qb0) * (unsigned)sizeof(FW);
    const int nq = active ? m.nbr_ptr[c + 1] - m.nbr_ptr[c] : 0;
    // the lane's pieces of the row: with W < 8 the cells of a quarter warp
    // take them in different orders, so that its eight 16-byte loads fall
    // into distinct bank groups whatever rows the cells name
    int pc[NP];
#pragma unroll
    for (int n = 0; n < NP; n++) pc[n] = l + W * (n ^ (i & (NP - 1)));
    const int ppd = nb / VE, npc = ndb * ppd;
    const int s0 = blockIdx.y * per, s1 = min(s0 + per, (npc + SW - 1) / SW);
    // (batch direction, piece of its rows) of batch piece P, then P + SW at
    // a time: the division only where a direction is shorter than a slab
    struct At {
        int dl, b;
    };
    auto locate = [&](int P) {
        At a;
        a.dl = P / ppd;
        a.b = P - a.dl * ppd;
        return a;
    };
    auto step = [&](At &a) {
        a.b += SW;
        if (a.b >= ppd) {
            const int k = ppd < SW ? a.b / ppd : 1;
            a.dl += k;
            a.b -= k * ppd;
        }
    };
    // a thread copies piece cp_l of every (bd / SW)-th row of the union
    const int cp_l = tid % SW, cp_u = tid / SW, cp_d = bd / SW;
    At ca = locate(s0 * SW + cp_l), pa[NP];
#pragma unroll
    for (int n = 0; n < NP; n++) pa[n] = locate(s0 * SW + pc[n]);
    __syncthreads();
    auto stage = [&]() {
        if (ca.dl < ndb) {
            const S *src = eps + (size_t)(d0 + ca.dl) * nc * nb + ca.b * VE;
            unsigned dst = rows_s + (unsigned)(cp_l * 16 + cp_u * RB);
            for (int u = cp_u; u < nu; u += cp_d, dst += cp_d * RB)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src + uoff[u]));
        }
        step(ca);
        cp_async_commit();
        cp_async_wait<0>();
    };
    for (int s = s0; s < s1; s++) {
        At at[NP];
        unsigned mk[NP];
#pragma unroll
        for (int n = 0; n < NP; n++) {
            at[n] = pa[n];
            step(pa[n]);
            mk[n] = active && at[n].dl < ndb ? mask[(size_t)(d0 + at[n].dl) * nc + c] : 0;
        }
        __syncthreads();  // the previous slab's reads are done
        stage();
        __syncthreads();
        if (!active) continue;
        unsigned row[NP];
#pragma unroll
        for (int n = 0; n < NP; n++) row[n] = rows_s + (unsigned)(pc[n] * 16);
        S ec[NP][VE], gx[NP][VE], gy[NP][VE], gz[NP][VE];
#pragma unroll
        for (int n = 0; n < NP; n++) {
            lds(row[n] + i * RB, ec[n]);
#pragma unroll
            for (int v = 0; v < VE; v++) gx[n][v] = gy[n][v] = gz[n][v] = 0;
        }
        auto entry = [&](const FW &t, const S (&e)[NP][VE]) {
#pragma unroll
            for (int n = 0; n < NP; n++)
#pragma unroll
                for (int v = 0; v < VE; v++) {
                    const S de = nbr_term(e[n][v], ec[n][v]);
                    gx[n][v] += t.x * de;
                    gy[n][v] += t.y * de;
                    if constexpr (DIM == 3) gz[n][v] += t.z * de;
                }
        };
        int q = 0;
        unsigned wc = wa;
        for (; q + U <= nq; q += U, wc += U * (unsigned)sizeof(FW)) {
            FW t[U];
            S e[U][NP][VE];
#pragma unroll
            for (int u = 0; u < U; u++) lds(wc + u * (unsigned)sizeof(FW), t[u]);
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int n = 0; n < NP; n++) lds(row[n] + t[u].at, e[u][n]);
#pragma unroll
            for (int u = 0; u < U; u++) entry(t[u], e[u]);
        }
        for (; q < nq; q++, wc += (unsigned)sizeof(FW)) {
            FW t;
            S e[NP][VE];
            lds(wc, t);
#pragma unroll
            for (int n = 0; n < NP; n++) lds(row[n] + t.at, e[n]);
            entry(t, e);
        }
#pragma unroll
        for (int n = 0; n < NP; n++) {
            if (at[n].dl >= ndb) continue;
            centre_term<VE>(m, c, ec[n], gx[n], gy[n], gz[n]);
            S *Fd = F + (size_t)at[n].dl * nf * nb + at[n].b * VE;
            for (int j = 0; j < nface; j++) {
                if (!(mk[n] >> j & 1)) continue;
                const FW t = fq[4 * i + j];
                S y[VE];
#pragma unroll
                for (int v = 0; v < VE; v++) {
                    y[v] = ec[n][v] + gx[n][v] * t.x + gy[n][v] * t.y;
                    if constexpr (DIM == 3) y[v] += gz[n][v] * t.z;
                }
                st_piece(Fd + t.at, y);
            }
            if (wall)
                for (int j = 0; j < nface; j++) {
                    const int slot = cf_gw[k0 + j];
                    if (slot < 0) continue;
                    S *gp = gw + ((size_t)at[n].dl * nws + slot) * DIM * nb + at[n].b * VE;
                    st_piece(gp, gx[n]);
                    st_piece(gp + nb, gy[n]);
                    if constexpr (DIM == 3) st_piece(gp + 2 * nb, gz[n]);
                }
        }
    }
}

// Second-order residual from the face values (k_residual8's formula, face by
// face in the same order):
//   R = C_b (T_old - T_base - tau|v| B) + Q hr tau / s_c
//       - eps_c - tau|v| / s_c sum_f A_f/V (s.n_f) y_f
// A thread owns one 16-byte piece of one cell and walks kResDirs directions.
// The coefficients A_f/V (s.n_f) of the CTA's cells and directions are
// formed once in shared memory (in FP64, rounded once), so the band threads
// of a cell do no FP64 geometry; the band constants are staged beside them.
//
// Bound by HBM latency and bandwidth: it reads e once and every face value
// once from HBM (its second reader finds it in L2) and writes R. At three
// CTAs per SM (80 registers; at four they spill, at two too few loads are in
// flight: 0.26 ms each on the first size below): 17,939 triangles x 40 bands
// x 64 directions FP32 0.45 ms with neighbour gradients, 0.23 ms here (2.8
// TB/s), FP64 0.74 -> 0.34 ms; 48,000 tetrahedra x 40 x 128 FP32 3.22 ->
// 1.28 ms (3.4 TB/s), 12,000 FP64 1.15 -> 0.50 ms.
// The face sum's term: the FP32 form rounds the product before the sum, as
// the compiler does in the branches of k_residual8, so every residual form
// gives the same bits.
__device__ __forceinline__ float add_face(float acc, float a, float y) { return __fadd_rn(acc, __fmul_rn(a, y)); }
__device__ __forceinline__ double add_face(double acc, double a, double y) { return acc + a * y; }
template <typename S, int DIM>
__global__ void __launch_bounds__(256, 3) k_resid_face(DMesh m, DPhys p, int cpb, const S *__restrict__ eps,
                                                       const S *__restrict__ F,
                                                       const unsigned char *__restrict__ mask,
                                                       const double *__restrict__ Tb, const double *__restrict__ Bf,
                                                       const double *__restrict__ Told,
                                                       const double *__restrict__ eb, const int *__restrict__ pos_of,
                                                       S *__restrict__ Rlo, int d0, int ndb) {
    constexpr int VE = kPieceBands<S>;
    extern __shared__ __align__(16) unsigned char rfm[];
    const int nb = p.nb, nc = m.nc, nf = m.nf, ppd = nb / VE, nbm = nb * p.nmat;
    double2 *cst = reinterpret_cast<double2 *>(rfm);  // [nmat][nb] {C, tau |v|}
    S *tvs = reinterpret_cast<S *>(cst + nbm);        // [nmat][nb] tau |v| in the storage precision
    S *coef = tvs + nbm;                              // [kResDirs][cpb][4]
    const int cb = blockIdx.x * cpb, ncell = min(cpb, nc - cb);
    const int da = blockIdx.y * kResDirs, nd = min(kResDirs, ndb - da);
    const int tid = threadIdx.x;
    for (int b = tid; b < nbm; b += blockDim.x) {
        const double tv = p.tau[b] * p.vmag[b];
        cst[b] = make_double2(p.C[b], tv);
        tvs[b] = (S)tv;
    }
    for (int t = tid; t < kResDirs * cpb * 4; t += blockDim.x) {
        const int j = t & 3, ci = (t >> 2) % cpb, dd = (t >> 2) / cpb;
        S a = 0;
        if (ci < ncell && dd < nd) {
            const int c = cb + ci, k = m.cf_ptr[c] + j;
            if (k < m.cf_ptr[c + 1]) {
                const size_t d = d0 + da + dd;
                const double sn = p.sx[d] * m.cf_nx[k] + p.sy[d] * m.cf_ny[k] + (DIM == 3 ? p.sz[d] * m.cf_nz[k] : 0.0);
                a = (S)(m.cf_area[k] * (m.tsc[c] / m.vol[c]) * sn);
            }
        }
        coef[t] = a;
    }
    __syncthreads();
    const int ci = tid / ppd, b0 = (tid - ci * ppd) * VE;
    if (ci >= ncell) return;
    const int c = cb + ci, mo = mat_off(p, c), k0 = m.cf_ptr[c], nface = m.cf_ptr[c + 1] - k0;
    const double tb = Tb[c], dT = Told[c] - tb, hc = m.heat[c] * m.tsc[c];
    int at[4];
    unsigned walls = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        at[j] = j < nface ? m.cf_face[k0 + j] * nb : 0;
        if (j < nface && m.cf_bound[k0 + j] >= 0) walls |= 1u << j;
    }
    const S *ep = eps + ((size_t)(d0 + da) * nc + c) * nb + b0;
    const S *Fp = F + (size_t)da * nf * nb + b0;
    size_t dc = (size_t)(d0 + da) * nc + c;
    for (int dd = 0; dd < nd; dd++, dc += nc, ep += (size_t)nc * nb, Fp += (size_t)nf * nb) {
        S ec[VE], y[4][VE], acc[VE];
        ld_piece(ep, ec);
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (j < nface) ld_piece(Fp + at[j], y[j]);
        const int pos = pos_of[dc];
        const double B = Bf[dc];
        if (walls) {
            // inflow wall faces take the wall value
            const unsigned in = walls & ~(unsigned)mask[dc];
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (in >> j & 1) {
                    const double *e = eb + ((size_t)(d0 + da + dd) * m.nbs + m.cf_bside[k0 + j]) * nb + b0;
#pragma unroll
                    for (int v = 0; v < VE; v++) y[j][v] = (S)(e[v] - cst[mo + b0 + v].x * tb);
                }
        }
#pragma unroll
        for (int v = 0; v < VE; v++) acc[v] = (S)0;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (j < nface) {
                const S a = coef[(dd * cpb + ci) * 4 + j];
#pragma unroll
                for (int v = 0; v < VE; v++) acc[v] = add_face(acc[v], a, y[j][v]);
            }
        S out[VE];
#pragma unroll
        for (int v = 0; v < VE; v++) {
            const double2 k = cst[mo + b0 + v];
            double fx = k.x * (dT - k.y * B);
            if (hc != 0) fx += hc * p.hr[mo + b0 + v] * p.tau[mo + b0 + v];
            out[v] = (S)fx - ec[v] - tvs[mo + b0 + v] * acc[v];
        }
        st_piece(Rlo + ((size_t)(da + dd) * nc + pos) * nb + b0, out);
    }
}

// The explicit time step (FP64, base 0) from the face values, in place:
// e <- e (1 - dt/tau) - dt (sum_f A/V (v.n) x_f - C Told/tau). A thread keeps
// a 16-byte piece of a cell's bands over `dirs` directions (kResDirs, as
// k_resid_face does, or fewer where that leaves SMs without a block); only the
// thread that writes a value reads it, so the new field needs no second array
// and no copy back. Bound by the face rows it streams.
// 4,608 triangles x 20 bands x 32 directions (FP64): 27 us, and a whole step
// 287 -> 153 us against gradient arrays, a thread per value and a copy back.
// 288 triangles x 2 bands x 256 directions: 27.6 us with eight directions each,
// 16.6 us with four.
template <int DIM>
__global__ void __launch_bounds__(256, 3) k_tr_step_face(DMesh m, DPhys p, int cpb, int dirs, double *eps,
                                                         const double *__restrict__ F,
                                                         const unsigned char *__restrict__ mask,
                                                         const double *__restrict__ Told,
                                                         const double *__restrict__ eb, double dt, int d0, int ndb) {
    constexpr int VE = kPieceBands<double>;
    extern __shared__ __align__(16) unsigned char rfm[];
    double *coef = reinterpret_cast<double *>(rfm);  // [dirs][cpb][4]
    const int nb = p.nb, nc = m.nc, nf = m.nf, ppd = nb / VE;
    const int cb = blockIdx.x * cpb, ncell = min(cpb, nc - cb);
    const int da = blockIdx.y * dirs, nd = min(dirs, ndb - da);
    const int tid = threadIdx.x;
    for (int t = tid; t < dirs * cpb * 4; t += blockDim.x) {
        const int j = t & 3, ci = (t >> 2) % cpb, dd = (t >> 2) / cpb;
        double a = 0;
        if (ci < ncell && dd < nd) {
            const int c = cb + ci, k = m.cf_ptr[c] + j;
            if (k < m.cf_ptr[c + 1]) {
                const size_t d = d0 + da + dd;
                const double sn = p.sx[d] * m.cf_nx[k] + p.sy[d] * m.cf_ny[k] + (DIM == 3 ? p.sz[d] * m.cf_nz[k] : 0.0);
                a = m.cf_area[k] / m.vol[c] * sn;
            }
        }
        coef[t] = a;
    }
    __syncthreads();
    const int ci = tid / ppd, b0 = (tid - ci * ppd) * VE;
    if (ci >= ncell) return;
    const int c = cb + ci, mo = mat_off(p, c), k0 = m.cf_ptr[c], nface = m.cf_ptr[c + 1] - k0;
    double keep[VE], src[VE], vm[VE];
#pragma unroll
    for (int v = 0; v < VE; v++) {
        const double tau = p.tau[mo + b0 + v] * m.tsc[c];
        keep[v] = 1 - dt / tau;
        src[v] = Told[c] * p.C[mo + b0 + v] / tau;
        vm[v] = p.vmag[mo + b0 + v];
    }
    int at[4];
    unsigned walls = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        at[j] = j < nface ? m.cf_face[k0 + j] * nb : 0;
        if (j < nface && m.cf_bound[k0 + j] >= 0) walls |= 1u << j;
    }
    double *ep = eps + ((size_t)(d0 + da) * nc + c) * nb + b0;
    const double *Fp = F + (size_t)da * nf * nb + b0;
    size_t dc = (size_t)(d0 + da) * nc + c;
    for (int dd = 0; dd < nd; dd++, dc += nc, ep += (size_t)nc * nb, Fp += (size_t)nf * nb) {
        double ec[VE], y[4][VE], acc[VE];
        ld_piece(ep, ec);
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (j < nface) ld_piece(Fp + at[j], y[j]);
        if (walls) {
            // inflow wall faces take the wall value
            const unsigned in = walls & ~(unsigned)mask[dc];
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (in >> j & 1)
                    ld_piece(eb + ((size_t)(d0 + da + dd) * m.nbs + m.cf_bside[k0 + j]) * nb + b0, y[j]);
        }
#pragma unroll
        for (int v = 0; v < VE; v++) acc[v] = 0;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (j < nface) {
                const double a = coef[(dd * cpb + ci) * 4 + j];
#pragma unroll
                for (int v = 0; v < VE; v++) acc[v] += a * y[j][v];
            }
#pragma unroll
        for (int v = 0; v < VE; v++) ec[v] = ec[v] * keep[v] - dt * (vm[v] * acc[v] - src[v]);
        st_piece(ep, ec);
    }
}

// k_bound_out with the gradients of the wall cells only (gw of k_grad_face):
// e_c(new) + g_c(pre-sweep) . (x_f - x_c) on the walls a direction leaves. A
// thread per (wall side, band) walks its block's share of the directions
// (dir_grid): 0.30 -> 0.14 ms against a thread per value (4,800 wall faces x
// 40 bands x 128 directions).
template <typename S, int DIM>
__global__ void __launch_bounds__(256) k_bound_out_w(DMesh m, DPhys p, const S *__restrict__ eps,
                                                     const S *__restrict__ gw, int nws, int nw,
                                                     const int *__restrict__ wall_side,
                                                     const int *__restrict__ wall_slot,
                                                     const double *__restrict__ Tb, const double *__restrict__ gTb,
                                                     double *__restrict__ eb, int d0, int ndb) {
    const int nb = p.nb, t = (int)gtid();
    if (t >= nw * nb) return;
    const int w = t / nb, b = t - w * nb, s = wall_side[w], c = m.bs_cell[s], k = m.bs_cf[s], mo = mat_off(p, c);
    const int slot = wall_slot[w];
    const double vm = p.vmag[mo + b], Cb = p.C[mo + b], Tc = Tb[c];
    const double nx = m.cf_nx[k], ny = m.cf_ny[k], nz = m.cf_nz[k];
    const double rx = m.cf_fx[k] - m.cx[c], ry = m.cf_fy[k] - m.cy[c], rz = m.cf_fz[k] - m.cz[c];
    const double gx = gTb[3 * c], gy = gTb[3 * c + 1], gz = gTb[3 * c + 2];
    const DirRange r = dir_share(ndb);
#pragma unroll 4
    for (int dl = r.first; dl < r.end; dl++) {
        const int d = d0 + dl;
        const double vn = vm * p.sx[d] * nx + vm * p.sy[d] * ny + vm * p.sz[d] * nz;
        if (!(vn >= 0)) continue;
        const S *gp = gw + ((size_t)dl * nws + slot) * DIM * nb + b;
        double v = ((double)gp[0] + Cb * gx) * rx + ((double)gp[nb] + Cb * gy) * ry;
        if (DIM == 3) v += ((double)gp[2 * nb] + Cb * gz) * rz;
        eb[((size_t)d * m.nbs + s) * nb + b] = Cb * Tc + (double)eps[((size_t)d * m.nc + c) * nb + b] + v;
    }
}
