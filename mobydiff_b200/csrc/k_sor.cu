// k_sor.cu -- red-black SOR velocity-pressure projection,
// src/modules/pressure/pressure_redblack.f90:27-254.
//
// One launch per colour sweep, one thread per cell of that colour.  Cells of
// one colour share no face and each owns its p, so the parallel sweep is
// bit-for-bit the reference's sequential loop (compiled with -fmad=false and
// the reference's expression order).  The reference iterates a fixed nIter;
// with tol > 0 the sweeps continue until ||div u||_2 <= max(tol*||div u*||_2,
// atol), checked every `check_every` iterations by a deterministic reduction.
//
// HBM: the IBM factors mu = 1/(1+dt_gamma*coef) are computed once per
// projection (the reference recomputes six per cell per sweep, :117-122);
// when the coefficients do not vary along z -- both the reference geometry
// and the wavy channel depend on x and y only -- mu is one (nx+2)(ny+2)
// plane per component that stays in L2, otherwise a padded array.  The same
// formula gives the same bits.  Successive sweeps walk the z planes in
// opposite directions, so each starts on the planes the previous one left
// in the 126 MB L2.
#include "mdx_cell.cuh"
#include "mdx_resident.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

// mu = 1/(1 + dt_gamma*coef) over n elements of each component.
__global__ void k_mu_tables(long long n, double dg, const double* __restrict__ cu, const double* __restrict__ cv,
                            const double* __restrict__ cw, double* __restrict__ mu) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        mu[t] = 1.0 / (1.0 + dg * __ldg(cu + t));
        mu[n + t] = 1.0 / (1.0 + dg * __ldg(cv + t));
        mu[2 * n + t] = 1.0 / (1.0 + dg * __ldg(cw + t));
    }
}


template <int MU>
__global__ void __launch_bounds__(256)
k_sor_sweep(mdx_dims d, mdx_bc_dev bc, mdx_sor_params p, int parity, int reverse, double* __restrict__ un,
            double* __restrict__ vn, double* __restrict__ wn, double* __restrict__ pn,
            const double* __restrict__ mu) {
    const int ni = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int kk = blockIdx.z * blockDim.z + threadIdx.z + 1;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    if (ni > nx / 2 || j > ny || kk > nz) return;
    const int k = reverse ? nz + 1 - kk : kk;
    const bool perx = bc.per[0] != 0, pery = bc.per[1] != 0, perz = bc.per[2] != 0;
    int jp = j + 1;
    if (pery && jp > ny) jp = 1;
    int kp = k + 1;
    if (perz && kp > nz) kp = 1;
    const int iLo = 1 + ((j + k + parity) & 1);
    const int i = iLo + 2 * (ni - 1);
    int ip = i + 1;
    if (perx && ip > nx) ip = 1;
    const long long c = pidx(d, i, j, k);
    const long long cip = pidx(d, ip, j, k), cjp = pidx(d, i, jp, k), ckp = pidx(d, i, j, kp);
    double mu_u_i = 1.0, mu_u_ip = 1.0, mu_v_j = 1.0, mu_v_jp = 1.0, mu_w_k = 1.0, mu_w_kp = 1.0;
    if (MU == MU_PLANE) {  // :117-122, z-invariant coefficients
        const long long np = (long long)d.nxp * d.nyp;
        const long long q = i + (long long)d.nxp * j;
        mu_u_i = __ldg(mu + q);
        mu_u_ip = __ldg(mu + ip + (long long)d.nxp * j);
        mu_v_j = __ldg(mu + np + q);
        mu_v_jp = __ldg(mu + np + i + (long long)d.nxp * jp);
        mu_w_k = __ldg(mu + 2 * np + q);
        mu_w_kp = mu_w_k;
    } else if (MU == MU_FULL) {
        const long long np = d.npad;
        mu_u_i = __ldg(mu + c);
        mu_u_ip = __ldg(mu + cip);
        mu_v_j = __ldg(mu + np + c);
        mu_v_jp = __ldg(mu + np + cjp);
        mu_w_k = __ldg(mu + 2 * np + c);
        mu_w_kp = __ldg(mu + 2 * np + ckp);
    }
    double u_i = un[c], u_ip = un[cip], v_j = vn[c], v_jp = vn[cjp], w_k = wn[c], w_kp = wn[ckp], pc = pn[c];
    sor_cell(u_i, u_ip, v_j, v_jp, w_k, w_kp, pc, mu_u_i, mu_u_ip, mu_v_j, mu_v_jp, mu_w_k, mu_w_kp, p, bc, i, j, k,
             nx, ny, nz);
    un[c] = u_i;
    un[cip] = u_ip;
    vn[c] = v_j;
    vn[cjp] = v_jp;
    wn[c] = w_k;
    wn[ckp] = w_kp;
    pn[c] = pc;
}

// ---------------------------------------------------------------------------
// One full red+black iteration in one pass (periodic x and z).
//
// A block owns 60 x (RY-3) columns of cells and a chunk of KZ planes and
// walks it in z.  u, v, w are read from one state and written to another, so
// blocks never see each other's updates; a block recomputes its halo (two
// cells below, one above, in every direction) from the values their owners
// use, so every face ends with the value of a red sweep followed by a black
// one, bit for bit.  p belongs to one cell and is updated in place.
//
// A warp is one row of 64 cells, a lane two neighbouring ones.  The red cells
// of plane m+2 and the black cells of plane m do not depend on each other and
// lie in different columns of a lane's two: a phase updates both, with one
// barrier.  u and v, which neighbours share, are in a ring of six planes in
// shared memory (m-1 on its way out, m .. m+2 in work, m+3 and m+4 in flight,
// cp.async); w and p stay with their columns, in registers, read and written
// 16 bytes a lane.  Rows store even cells, then odd cells: one colour of a
// row is contiguous, and so is a fetch.
//
// A colour sweep each moves u, v, w, p twice through HBM: 78 us an iteration
// of 180x150x140, at 6.2 TB/s.  A pass moves them once: 59 us (DRAM at 43 %,
// shared-memory pipe at 52 %; the chain of a phase, shared memory - 12 FP64
// operations - shared memory - barrier, is what is left).  On the way: slots
// and plane numbers by remainders 90, 20 registers' worth of values moved
// along each phase 88, w and p a lane at a time and selected as soon as read
// 97, selected a phase later 62.  Its predecessor, u, v, w, p in shared
// memory and four barriers a plane, took 254.
// RY: 20 rows where the factors are 1 (94 registers), 16 with factors per
// column (20 would spill: 111 against 63 us); 8 for MDX_SORV_FUSED8.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

constexpr int PASS_TX = 60, PASS_SLOTS = 6;
constexpr int PASS_H = 40, PASS_R = 72;   // a row: even cells from 0, odd cells from PASS_H (other banks)
template <int RY> struct pass_geom {
    static constexpr int TY = RY - 3;
    static constexpr int NU = RY * PASS_R, NV = (RY + 1) * PASS_R, SLOT = NU + NV;
    static constexpr size_t SMEM = sizeof(double) * PASS_SLOTS * SLOT;
};

template <int MU, int PY, int RY>
__global__ void __launch_bounds__(32 * RY, RY == 8 ? 2 : 1)
k_sor_pass(mdx_dims d, mdx_bc_dev bc, mdx_sor_params P, int KZ, const double* __restrict__ u0,
           const double* __restrict__ v0, const double* __restrict__ w0, double* __restrict__ u1,
           double* __restrict__ v1, double* __restrict__ w1, double* __restrict__ pn,
           const double* __restrict__ mu) {
    using G = pass_geom<RY>;
    extern __shared__ double sm[];
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const int l = threadIdx.x & 31, r = threadIdx.x >> 5;
    const int x0 = blockIdx.x * PASS_TX + 1, y0 = blockIdx.y * G::TY + 1, k0 = blockIdx.z * KZ + 1;
    const int k1 = min(k0 + KZ - 1, nz);
    const unsigned plane = (unsigned)(d.nxp * d.nyp);   // offsets into an array: 32 bits (pass_fits)
    auto wrapx = [&](int c) { return ((x0 - 4 + c) % nx + nx) % nx + 1; };          // cell c of the row
    auto rowy = [&](int q) {                                                         // row q of the tile
        const int g = y0 - 2 + q;
        return PY ? ((g - 1) % ny + ny) % ny + 1 : min(max(g, 0), ny + 1);
    };
    const int j = y0 - 2 + r, gj = rowy(r);
    const bool row_in = PY || (j >= 1 && j <= ny);

    // fetched and written as cells l and l + 32 of a row, which are contiguous
    const unsigned f0 = wrapx(l) + d.nxp * gj, f1 = wrapx(l + 32) + d.nxp * gj;
    const unsigned fx = wrapx(64) + d.nxp * gj;             // the face right of the last cell
    const unsigned h = d.nxp * (rowy(RY) - gj);             // from row 0 of the tile to row RY
    const int t0 = r * PASS_R + (l & 1) * PASS_H + (l >> 1), t1 = t0 + 16;   // their places in a plane
    auto fetch = [&](int slot, unsigned o) {
        double* s = sm + slot * G::SLOT;
        cp_async8(s + t0, u0 + (o + f0));
        cp_async8(s + t1, u0 + (o + f1));
        if (l == 0) cp_async8(s + r * PASS_R + 32, u0 + (o + fx));
        cp_async8(s + G::NU + t0, v0 + (o + f0));
        cp_async8(s + G::NU + t1, v0 + (o + f1));
        if (r == 0) {
            cp_async8(s + G::NU + RY * PASS_R + t0, v0 + (o + f0 + h));
            cp_async8(s + G::NU + RY * PASS_R + t1, v0 + (o + f1 + h));
        }
    };

    // The lane's cells are 2l and 2l + 1, x = x0-3+2l even: 16 bytes together
    // but where the period ends between them.  Column A is red on planes of
    // k0's parity, column B on the others; a: A is the second cell.
    const int a = (j + k0 + 1) & 1, cA = 2 * l + a, cB = 2 * l + 1 - a;
    const int xe = x0 - 3 + 2 * l;
    const bool ends = wrapx(2 * l) == nx;
    const unsigned ge = (xe >= 0 && xe <= nx ? xe : wrapx(2 * l)) + d.nxp * gj;
    const unsigned g0 = wrapx(2 * l) + d.nxp * gj, g1 = wrapx(2 * l + 1) + d.nxp * gj;
    const bool own_row = row_in && r >= 2 && r <= RY - 2 && j <= ny;
    auto owned = [&](int c) { return own_row && c >= 3 && c <= 62 && x0 - 3 + c <= nx; };
    const bool o0 = owned(2 * l), o1 = owned(2 * l + 1), own = o0 || o1;
    const bool full = o0 && o1;
    auto put2 = [&](double* q, unsigned o, double x, double y, auto FULL) {
        if (FULL) *reinterpret_cast<double2*>(q + (o + ge)) = make_double2(x, y);
        else if (o0) q[o + ge] = x;
        else q[o + ge + 1] = y;
    };
    auto get_w = [&](unsigned o) {
        if (!ends) return __ldg(reinterpret_cast<const double2*>(w0 + (o + ge)));
        return make_double2(__ldg(w0 + (o + g0)), __ldg(w0 + (o + g1)));
    };
    auto get_p = [&](unsigned o) { return *reinterpret_cast<const double2*>(pn + (o + ge)); };
    auto to_cols = [&](double2 t, double& A, double& B) {
        A = a ? t.y : t.x;
        B = a ? t.x : t.y;
    };
    const bool wall = !PY && j == ny;
    struct factors { double u_i, u_ip, v_j, v_jp, w, fac; };
    auto column = [&](int c) {
        factors m{1.0, 1.0, 1.0, 1.0, 1.0, 0.0};
        const unsigned g = wrapx(c) + d.nxp * gj;
        if (MU == MU_PLANE) {
            m.u_i = __ldg(mu + g);
            m.u_ip = __ldg(mu + wrapx(c + 1) + d.nxp * gj);
            m.v_j = __ldg(mu + plane + g);
            m.v_jp = __ldg(mu + plane + wrapx(c) + d.nxp * rowy(r + 1));
            m.w = __ldg(mu + 2 * plane + g);
        }
        m.fac = sor_factor(m.u_i, m.u_ip, m.v_j, m.v_jp, m.w, m.w, P);
        return m;
    };
    const factors FA = column(cA), FB = column(cB);
    // places in a plane of the columns' faces and of cell c + 1's
    const int sA = r * PASS_R + a * PASS_H + l, sB = r * PASS_R + (1 - a) * PASS_H + l;
    const int nA = a ? r * PASS_R + l + 1 : sB, nB = a ? sA : r * PASS_R + l + 1;
    struct faces { double u_i, u_ip, v_j, v_jp; };
    auto get = [&](int slot, int s0, int s1) {
        const double *su = sm + slot * G::SLOT, *sv = su + G::NU;
        return faces{su[s0], su[s1], sv[s0], sv[s0 + PASS_R]};
    };
    auto put = [&](int slot, int s0, int s1, const faces& f) {
        double *su = sm + slot * G::SLOT, *sv = su + G::NU;
        su[s0] = f.u_i;
        su[s1] = f.u_ip;
        sv[s0] = f.v_j;
        sv[s0 + PASS_R] = f.v_jp;
    };
    auto update = [&](faces& f, const factors& m, double& wk, double& wkp, double& pc) {
        sor_cell_fac<1, PY, 1>(f.u_i, f.u_ip, f.v_j, f.v_jp, wk, wkp, pc, m.u_i, m.u_ip, m.v_j, m.v_jp, m.w, m.w,
                               m.fac, P, bc, 0, j, 0, nx, ny, nz);
    };
    auto cell = [&](int slot, int s0, int s1, const factors& m, double& wk, double& wkp, double& pc) {
        faces f = get(slot, s0, s1);
        update(f, m, wk, wkp, pc);
        put(slot, s0, s1, f);
    };
    auto put_uv = [&](int slot, unsigned o, auto FULL) {
        const double* su = sm + slot * G::SLOT + r * PASS_R + l;
        const double* sv = su + G::NU;
        put2(u1, o, su[0], su[PASS_H], FULL);
        put2(v1, o, sv[0], sv[PASS_H], FULL);
        if (wall) put2(v1, o + d.nxp, sv[PASS_R], sv[PASS_R + PASS_H], FULL);
    };
    // Plane k is in slot (k - k0 + 2) mod 6 and its w and p in entry (k - k0 + 1)
    // mod 6: the loop is unrolled by 6 so that both are constants.
    const unsigned top = (unsigned)nz * plane;
    auto next = [&](unsigned o) { return o == top ? plane : o + plane; };
    unsigned o = (unsigned)(((k0 - 3) % nz + nz) % nz + 1) * plane;   // plane k0-2
    double wA[6], wB[6], pA[6], pB[6], wl, none = 0.0;
    double2 wq[5], wnext, pnext = make_double2(0.0, 0.0), p0 = pnext;
#pragma unroll
    for (int q = 0; q < 5; ++q) {   // planes k0-2 .. k0+2
        if (k0 - 2 + q <= k1 + 1) fetch(q, o);
        cp_async_commit();
        wq[q] = get_w(o);
        o = next(o);
    }
    unsigned om = (unsigned)k0 * plane - plane;   // plane k0-1
    if (own) {
        p0 = get_p(om + plane);
        if (k0 + 1 <= k1) pnext = get_p(om + 2 * plane);
    }
    to_cols(wq[0], wl, none);
    none = 0.0;
    to_cols(wq[1], wA[0], wB[0]);
    to_cols(wq[2], wA[1], wB[1]);
    to_cols(wq[3], wA[2], wB[2]);
    wnext = wq[4];
    pA[0] = pB[0] = 0.0;
    to_cols(p0, pA[1], pB[1]);
    cp_async_wait<1>();   // planes up to k0 + 1
    __syncthreads();
    if (row_in) {   // red cells of planes k0-2, k0-1, k0
        cell(0, sA, nA, FA, wl, wA[0], none);
        cell(1, sB, nB, FB, wB[0], wB[1], none);
        cell(2, sA, nA, FA, wA[1], wA[2], pA[1]);
    }
    __syncthreads();

    // Plane m = k0-1+U (mod 6): red cells of m+2 in column R, black ones of m
    // in column K.  o: plane m+4 in the periodic array, om: plane m.
    // Both cells are updated by every lane, their chains side by side: what
    // the tile's outermost cells and, at the end, plane k1+2 get is wrong and
    // reaches no owned face.
    auto phase = [&](auto UC, int m, int sR, int sK, int nR, int nK, const factors& FR, const factors& FK,
                     double (&wR)[6], double (&wK)[6], double (&pR)[6], double (&pK)[6]) {
        constexpr int U = decltype(UC)::value;
        // what the last plane read, a barrier ago; nothing waits for a read of its own plane
        to_cols(wnext, wA[(U + 3) % 6], wB[(U + 3) % 6]);
        to_cols(pnext, pA[(U + 2) % 6], pB[(U + 2) % 6]);
        if (m + 4 <= k1 + 2) {
            if (m + 4 <= k1 + 1) fetch((U + 5) % 6, o);
            wnext = get_w(o);
            o = next(o);
        }
        cp_async_commit();
        if (own && m + 3 <= k1) pnext = get_p(om + 3 * plane);
        if (row_in) {
            faces fK = get((U + 1) % 6, sK, nK), fR = get((U + 3) % 6, sR, nR);
            update(fK, FK, wK[U], wK[(U + 1) % 6], pK[U]);
            update(fR, FR, wR[(U + 2) % 6], wR[(U + 3) % 6], pR[(U + 2) % 6]);
            put((U + 1) % 6, sK, nK, fK);
            put((U + 3) % 6, sR, nR, fR);
        }
        auto store = [&](auto FULL) {
            put2(w1, om, a ? wB[U] : wA[U], a ? wA[U] : wB[U], FULL);
            put2(pn, om, a ? pB[U] : pA[U], a ? pA[U] : pB[U], FULL);
            if (m > k0) put_uv(U, om - plane, FULL);
        };
        if (m >= k0) {
            if (full) store(std::true_type{});
            else if (own) store(std::false_type{});
        }
        om += plane;
        cp_async_wait<1>();   // plane m + 3
        __syncthreads();
    };
    auto odd = [&](auto UC, int m) { phase(UC, m, sB, sA, nB, nA, FB, FA, wB, wA, pB, pA); };
    auto even = [&](auto UC, int m) { phase(UC, m, sA, sB, nA, nB, FA, FB, wA, wB, pA, pB); };
    for (int m = k0 - 1;; m += 6) {
        odd(std::integral_constant<int, 0>{}, m);
        if (m + 1 > k1) break;
        even(std::integral_constant<int, 1>{}, m + 1);
        if (m + 2 > k1) break;
        odd(std::integral_constant<int, 2>{}, m + 2);
        if (m + 3 > k1) break;
        even(std::integral_constant<int, 3>{}, m + 3);
        if (m + 4 > k1) break;
        odd(std::integral_constant<int, 4>{}, m + 4);
        if (m + 5 > k1) break;
        even(std::integral_constant<int, 5>{}, m + 5);
        if (m + 6 > k1) break;
    }
    if (full) put_uv((k1 - k0 + 2) % 6, om - plane, std::true_type{});
    else if (own) put_uv((k1 - k0 + 2) % 6, om - plane, std::false_type{});
}

double mdx_div_floor(const mdx_ctx_t* ctx, double umax) {
    const double eps = 2.220446049250313e-16;
    const mdx_grid_t& g = ctx->g;
    return eps * std::sqrt((double)ctx->d.nint) * umax * (1.0 / g.dx + 1.0 / g.dy + 1.0 / g.dz);
}

// One colour sweep for periodic x and z (the configurations of every run
// here): boundary flags are compile-time constants, in-plane offsets are
// 32-bit, and registers are bounded for occupancy.
// FIRST: the faces are read from u*, v*, w* and written to u, v, w, in place
// of the copy that starts a projection: a sweep of one colour touches every
// face between two cells, and k_shell_copy sets the rest before it.
template <int MU, int PY, bool FIRST>
__global__ void __launch_bounds__(256, 4)
k_sor_sweep_pxz(mdx_dims d, mdx_bc_dev bc, mdx_sor_params p, int parity, int reverse, double* __restrict__ un,
                double* __restrict__ vn, double* __restrict__ wn, double* __restrict__ pn,
                const double* __restrict__ mu, const double* __restrict__ us, const double* __restrict__ vs,
                const double* __restrict__ ws) {
    const int ni = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int kk = blockIdx.z * blockDim.z + threadIdx.z + 1;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    if (ni > nx / 2 || j > ny || kk > nz) return;
    const int k = reverse ? nz + 1 - kk : kk;
    const int jp = (PY && j == ny) ? 1 : j + 1;
    const int kp = (k == nz) ? 1 : k + 1;
    const int i = 1 + ((j + k + parity) & 1) + 2 * (ni - 1);
    const int ip = (i == nx) ? 1 : i + 1;
    const long long plane = (long long)d.nxp * d.nyp;
    const int q = i + d.nxp * j, qip = ip + d.nxp * j, qjp = i + d.nxp * jp;
    double* U = un + k * plane;
    double* Vv = vn + k * plane;
    double* W = wn + k * plane;
    double* Wn = wn + kp * plane;
    double* Pp = pn + k * plane;
    double mu_u_i = 1.0, mu_u_ip = 1.0, mu_v_j = 1.0, mu_v_jp = 1.0, mu_w = 1.0;
    if (MU == MU_PLANE) {
        mu_u_i = __ldg(mu + q);
        mu_u_ip = __ldg(mu + qip);
        mu_v_j = __ldg(mu + plane + q);
        mu_v_jp = __ldg(mu + plane + qjp);
        mu_w = __ldg(mu + 2 * plane + q);
    }
    double u_i, u_ip, v_j, v_jp, w_k, w_kp, pc = Pp[q];
    if (FIRST) {
        u_i = __ldg(us + k * plane + q);
        u_ip = __ldg(us + k * plane + qip);
        v_j = __ldg(vs + k * plane + q);
        v_jp = __ldg(vs + k * plane + qjp);
        w_k = __ldg(ws + k * plane + q);
        w_kp = __ldg(ws + kp * plane + q);
    } else {
        u_i = U[q];
        u_ip = U[qip];
        v_j = Vv[q];
        v_jp = Vv[qjp];
        w_k = W[q];
        w_kp = Wn[q];
    }
    const double fac = sor_factor(mu_u_i, mu_u_ip, mu_v_j, mu_v_jp, mu_w, mu_w, p);
    sor_cell_fac<1, PY, 1>(u_i, u_ip, v_j, v_jp, w_k, w_kp, pc, mu_u_i, mu_u_ip, mu_v_j, mu_v_jp, mu_w, mu_w, fac, p,
                           bc, i, j, k, nx, ny, nz);
    U[q] = u_i;
    U[qip] = u_ip;
    Vv[q] = v_j;
    Vv[qjp] = v_jp;
    W[q] = w_k;
    Wn[q] = w_kp;
    Pp[q] = pc;
}

// u, v, w <- u*, v*, w* where no cell pair's face lies: the ghost layers and
// the wall rows v(1), v(ny+1).  Faces of the box as in k_bc_fft.
__global__ void k_shell_copy(mdx_dims d, double* __restrict__ un, double* __restrict__ vn, double* __restrict__ wn,
                             const double* __restrict__ us, const double* __restrict__ vs,
                             const double* __restrict__ ws) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y * blockDim.y + threadIdx.y;
    auto put = [&](int i, int j, int k) {
        const long long c = pidx(d, i, j, k);
        un[c] = us[c];
        vn[c] = vs[c];
        wn[c] = ws[c];
    };
    if (blockIdx.z == 0) {
        if (a > d.nx + 1 || b > d.ny + 1) return;
        put(a, b, 0);
        put(a, b, d.nz + 1);
    } else if (blockIdx.z == 1) {
        if (a > d.nx + 1 || b >= d.nz) return;
        put(a, 0, b + 1);
        put(a, d.ny + 1, b + 1);
        const long long c = pidx(d, a, 1, b + 1);
        vn[c] = vs[c];
    } else {
        if (a >= d.ny || b >= d.nz) return;
        put(0, a + 1, b + 1);
        put(d.nx + 1, a + 1, b + 1);
    }
}

// ---------------------------------------------------------------------------
// The same colour sweep on colour-split copies of u, v, w, p (cidx): the
// cells of one colour in a row and every face they touch are consecutive, so
// a warp's loads and stores fill whole 32-byte sectors instead of every other
// element of them.  Same per-cell arithmetic as k_sor_sweep_pxz, so the
// same bits; the copies are made once per projection (k_split_copy).
// ---------------------------------------------------------------------------
template <int MU, int PY>
__global__ void __launch_bounds__(256, 4)
k_sor_sweep_split(mdx_dims d, mdx_bc_dev bc, mdx_sor_params p, int parity, int reverse, double* __restrict__ un,
                  double* __restrict__ vn, double* __restrict__ wn, double* __restrict__ pn,
                  const double* __restrict__ mu) {
    const int ni = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int kk = blockIdx.z * blockDim.z + threadIdx.z + 1;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    if (ni > nx / 2 || j > ny || kk > nz) return;
    const int k = reverse ? nz + 1 - kk : kk;
    const int jp = (PY && j == ny) ? 1 : j + 1;
    const int kp = (k == nz) ? 1 : k + 1;
    const int i = 1 + ((j + k + parity) & 1) + 2 * (ni - 1);
    const int ip = (i == nx) ? 1 : i + 1;
    const long long c = cidx(d, i, j, k), cip = cidx(d, ip, j, k), cjp = cidx(d, i, jp, k), ckp = cidx(d, i, j, kp);
    double mu_u_i = 1.0, mu_u_ip = 1.0, mu_v_j = 1.0, mu_v_jp = 1.0, mu_w = 1.0;
    if (MU == MU_PLANE) {
        const long long plane = (long long)d.nxp * d.nyp;
        const int q = i + d.nxp * j;
        mu_u_i = __ldg(mu + q);
        mu_u_ip = __ldg(mu + ip + d.nxp * j);
        mu_v_j = __ldg(mu + plane + q);
        mu_v_jp = __ldg(mu + plane + i + d.nxp * jp);
        mu_w = __ldg(mu + 2 * plane + q);
    }
    double u_i = un[c], u_ip = un[cip], v_j = vn[c], v_jp = vn[cjp], w_k = wn[c], w_kp = wn[ckp], pc = pn[c];
    const double fac = sor_factor(mu_u_i, mu_u_ip, mu_v_j, mu_v_jp, mu_w, mu_w, p);
    sor_cell_fac<1, PY, 1>(u_i, u_ip, v_j, v_jp, w_k, w_kp, pc, mu_u_i, mu_u_ip, mu_v_j, mu_v_jp, mu_w, mu_w, fac, p,
                           bc, i, j, k, nx, ny, nz);
    un[c] = u_i;
    un[cip] = u_ip;
    vn[c] = v_j;
    vn[cjp] = v_jp;
    wn[c] = w_k;
    wn[ckp] = w_kp;
    pn[c] = pc;
}

// The IBM factors (1 without IBM) and -omega/denom of every (i, j) column in
// colour-split planes (pidx2) for k_sor_sweep_splitv: [mu_u | mu_v | mu_w |
// fac], each split_plane_elems long.  fac is sor_factor of the column -- the
// FP64 expression the other kernels evaluate per cell; with z-invariant
// factors it is the same for every cell of the column, so the same bits.
template <int MU>
__global__ void k_split_tables(mdx_dims d, int py, mdx_sor_params p, const double* __restrict__ mu,
                               double* __restrict__ tab) {
    const long long np = (long long)d.nxp * d.nyp;
    const int ps = split_plane_elems(d);
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < np; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % d.nxp), j = (int)(t / d.nxp);
        double mu_u = 1.0, mu_v = 1.0, mu_w = 1.0;
        if (MU == MU_PLANE) {
            mu_u = __ldg(mu + t);
            mu_v = __ldg(mu + np + t);
            mu_w = __ldg(mu + 2 * np + t);
        }
        const int o = pidx2(d, i, j);
        tab[o] = mu_u;
        tab[ps + o] = mu_v;
        tab[2 * ps + o] = mu_w;
        double f = 0.0;
        if (i >= 1 && i <= d.nx && j >= 1 && j <= d.ny) {
            const int ip = i == d.nx ? 1 : i + 1;
            const int jp = (py && j == d.ny) ? 1 : j + 1;
            double mu_uip = 1.0, mu_vjp = 1.0;
            if (MU == MU_PLANE) {
                mu_uip = __ldg(mu + ip + (long long)d.nxp * j);
                mu_vjp = __ldg(mu + np + i + (long long)d.nxp * jp);
            }
            f = sor_factor(mu_u, mu_uip, mu_v, mu_vjp, mu_w, mu_w, p);
        }
        tab[3 * ps + o] = f;
    }
}

__device__ __forceinline__ void ld2(double (&a)[2], const double* q) {
    const double2 v = *reinterpret_cast<const double2*>(q);
    a[0] = v.x;
    a[1] = v.y;
}
__device__ __forceinline__ void ld2_ro(double (&a)[2], const double* __restrict__ q) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(q));
    a[0] = v.x;
    a[1] = v.y;
}
__device__ __forceinline__ void st2(double* q, const double (&a)[2]) {
    *reinterpret_cast<double2*>(q) = make_double2(a[0], a[1]);
}

// One FP64 colour sweep on the colour-split copies with two consecutive cells
// of the swept colour per thread, moved with 16-byte accesses: the layout
// and ownership of k_sor_sweep32v (k_sor_mixed.cu) -- a thread owns window w
// (positions 2w, 2w + 1) of its row in the swept colour's half and of the
// other half's rows (j + 1, k) and (j, k + 1); the x neighbours' faces u(i+1)
// are the window shifted by one in rows whose swept cells have odd i (window
// plus one scalar), the window itself in the others except the wrap of cell
// nx to position 0, and are stored one scalar per cell; positions without a
// swept cell are written back unchanged.  The factors come from
// k_split_tables.  The per-cell arithmetic is sor_cell_fac, as in
// k_sor_sweep_split, so the same bits.  Periodic x and z.
template <int PY>
__global__ void __launch_bounds__(128)
k_sor_sweep_splitv(mdx_dims d, mdx_bc_dev bc, mdx_sor_params p, int parity, int reverse, int nwin,
                   double* __restrict__ un, double* __restrict__ vn, double* __restrict__ wn,
                   double* __restrict__ pn, const double* __restrict__ tab) {
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long per_plane = (long long)nwin * d.ny;
    if (g >= per_plane * d.nz) return;
    const int kk = (int)(g / per_plane);
    const int rem = (int)(g - (long long)kk * per_plane);
    const int j = rem / nwin + 1;
    const int p0 = 2 * (rem - (j - 1) * nwin);
    const int k = reverse ? d.nz - kk : kk + 1;
    const int cs = 1 - parity;            // colour (i + j + k) & 1 of the swept cells
    const int eo = (cs + j + k) & 1;      // i & 1 of the swept cells of this row
    const int half = d.nx / 2;
    const int jp = (PY && j == d.ny) ? 1 : j + 1;
    const int kp = (k == d.nz) ? 1 : k + 1;
    const long long H = (long long)d.hs * d.nyp * d.nzp;
    const long long own = cs * H + ((long long)k * d.nyp + j) * d.hs + p0;
    const long long oth = (1 - cs) * H + ((long long)k * d.nyp + j) * d.hs;
    const long long ojp = (1 - cs) * H + ((long long)k * d.nyp + jp) * d.hs + p0;
    const long long okp = (1 - cs) * H + ((long long)kp * d.nyp + j) * d.hs + p0;
    const int PH = d.hs * d.nyp, ps = 2 * PH;
    const int hp = (eo + j) & 1;
    const int mown = hp * PH + j * d.hs + p0;
    const int mox = (1 - hp) * PH + j * d.hs;
    const int mjp = (1 - hp) * PH + jp * d.hs + p0;

    double u0[2], ux[2], v0[2], vy[2], w0[2], wz[2], q[2];
    double mu_u[2], mu_ux[2], mu_v[2], mu_vy[2], mu_w[2], fc[2];
    ld2(u0, un + own);
    ld2(v0, vn + own);
    ld2(w0, wn + own);
    ld2(q, pn + own);
    ld2(ux, un + oth + p0);
    ld2(vy, vn + ojp);
    ld2(wz, wn + okp);
    ld2_ro(mu_u, tab + mown);
    ld2_ro(mu_v, tab + ps + mown);
    ld2_ro(mu_w, tab + 2 * ps + mown);
    ld2_ro(fc, tab + 3 * ps + mown);
    ld2_ro(mu_ux, tab + mox + p0);
    ld2_ro(mu_vy, tab + ps + mjp);
    const int xe = eo ? p0 + 2 : 0;
    const bool need_xe = eo ? (p0 + 2 < d.hs) : (half >= p0 && half < p0 + 2);
    double uxe = 0.0, muxe = 0.0;
    if (need_xe) {
        uxe = un[oth + xe];
        muxe = __ldg(tab + mox + xe);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int pe = p0 + e;
        const bool valid = eo ? (pe < half) : (pe >= 1 && pe <= half);
        const bool wrap = !eo && pe == half;
        double u_ip, mu_ip;
        if (e == 0) {
            u_ip = eo ? ux[1] : (wrap ? uxe : ux[0]);
            mu_ip = eo ? mu_ux[1] : (wrap ? muxe : mu_ux[0]);
        } else {
            u_ip = (eo || wrap) ? uxe : ux[1];
            mu_ip = (eo || wrap) ? muxe : mu_ux[1];
        }
        if (valid) {
            const int i = 2 * pe + eo;
            sor_cell_fac<1, PY, 1>(u0[e], u_ip, v0[e], vy[e], w0[e], wz[e], q[e], mu_u[e], mu_ip, mu_v[e], mu_vy[e],
                                   mu_w[e], mu_w[e], fc[e], p, bc, i, j, k, d.nx, d.ny, d.nz);
            un[oth + (eo ? pe + 1 : (wrap ? 0 : pe))] = u_ip;
        }
    }
    st2(un + own, u0);
    st2(vn + own, v0);
    st2(wn + own, w0);
    st2(pn + own, q);
    st2(vn + ojp, vy);
    st2(wn + okp, wz);
}

// Every padded element of u, v, w, p between the reference layout and the
// colour-split copies (TO_SPLIT) or back.
template <bool TO_SPLIT>
__global__ void k_split_copy(mdx_dims d, double* __restrict__ a0, double* __restrict__ a1, double* __restrict__ a2,
                             double* __restrict__ a3, double* __restrict__ s0, double* __restrict__ s1,
                             double* __restrict__ s2, double* __restrict__ s3) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < d.npad; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % d.nxp);
        const long long r = t / d.nxp;
        const int j = (int)(r % d.nyp);
        const int k = (int)(r / d.nyp);
        const long long c = cidx(d, i, j, k);
        if (TO_SPLIT) {
            s0[c] = a0[t]; s1[c] = a1[t]; s2[c] = a2[t]; s3[c] = a3[t];
        } else {
            a0[t] = s0[c]; a1[t] = s1[c]; a2[t] = s2[c]; a3[t] = s3[c];
        }
    }
}

static mdx_sor_params sor_params(const mdx_ctx_t* ctx, double dg) {
    const mdx_grid_t& g = ctx->g;
    mdx_sor_params p;
    p.dx = g.dx; p.dy = g.dy; p.dz = g.dz;
    p.idx = 1.0 / g.dx; p.idy = 1.0 / g.dy; p.idz = 1.0 / g.dz;   // :54-60
    p.idx2 = p.idx * p.idx; p.idy2 = p.idy * p.idy; p.idz2 = p.idz * p.idz;
    p.idt = 1.0 / dg;
    p.sor = ctx->opts.sor;
    p.dt_gamma = dg;
    return p;
}

static bool sor_pxz(const mdx_ctx_t* ctx) {
    return ctx->bc.is_periodic[0] && ctx->bc.is_periodic[2] && ctx->mu_mode != MU_FULL;
}

static int shell_copy(mdx_ctx_t* ctx) {
    const mdx_dims& d = ctx->d;
    double** f = ctx->f;
    MDX_LAUNCH(ctx, MDX_T_OTHER, "shell copy", k_shell_copy,
               dim3((std::max(d.nxp, d.ny) + 31) / 32, (std::max(d.nyp, d.nz) + 7) / 8, 3), dim3(32, 8), 0, d,
               f[MDX_UN], f[MDX_VN], f[MDX_WN], f[MDX_US], f[MDX_VS], f[MDX_WS]);
    return MDX_OK;
}

// first: u, v, w are not set yet, the red sweep reads u*, v*, w* (sor_pxz only).
static int sor_iteration(mdx_ctx_t* ctx, const mdx_sor_params& p, bool first = false) {
    const mdx_dims& d = ctx->d;
    double** f = ctx->f;
    const int na = d.nx / 2;
    dim3 block(32, 4, 2);
    dim3 grid((na + 31) / 32, (d.ny + 3) / 4, (d.nz + 1) / 2);
    const bool pxz = sor_pxz(ctx);
    const bool py = ctx->bc.is_periodic[1] != 0;
    if (first) MDX_TRY(shell_copy(ctx));
    for (int parity = 0; parity < 2; ++parity) {
        const int rev = parity;   // red sweeps walk k up, black sweeps walk k down
        if (pxz) {
            auto kfn = ctx->mu_mode == MU_PLANE
                           ? (py ? k_sor_sweep_pxz<MU_PLANE, 1, false> : k_sor_sweep_pxz<MU_PLANE, 0, false>)
                           : (py ? k_sor_sweep_pxz<MU_ONE, 1, false> : k_sor_sweep_pxz<MU_ONE, 0, false>);
            if (first && parity == 0)
                kfn = ctx->mu_mode == MU_PLANE
                          ? (py ? k_sor_sweep_pxz<MU_PLANE, 1, true> : k_sor_sweep_pxz<MU_PLANE, 0, true>)
                          : (py ? k_sor_sweep_pxz<MU_ONE, 1, true> : k_sor_sweep_pxz<MU_ONE, 0, true>);
            MDX_LAUNCH(ctx, MDX_T_SOR_SWEEP, "sor sweep", kfn, grid, block, 0, d, ctx->bcd, p, parity, rev,
                       f[MDX_UN], f[MDX_VN], f[MDX_WN], f[MDX_PN], ctx->mu, f[MDX_US], f[MDX_VS], f[MDX_WS]);
        } else if (ctx->mu_mode == MU_ONE)
            MDX_LAUNCH(ctx, MDX_T_SOR_SWEEP, "sor sweep", k_sor_sweep<MU_ONE>, grid, block, 0, d, ctx->bcd, p, parity,
                       rev, f[MDX_UN], f[MDX_VN], f[MDX_WN], f[MDX_PN], ctx->mu);
        else if (ctx->mu_mode == MU_PLANE)
            MDX_LAUNCH(ctx, MDX_T_SOR_SWEEP, "sor sweep", k_sor_sweep<MU_PLANE>, grid, block, 0, d, ctx->bcd, p,
                       parity, rev, f[MDX_UN], f[MDX_VN], f[MDX_WN], f[MDX_PN], ctx->mu);
        else
            MDX_LAUNCH(ctx, MDX_T_SOR_SWEEP, "sor sweep", k_sor_sweep<MU_FULL>, grid, block, 0, d, ctx->bcd, p,
                       parity, rev, f[MDX_UN], f[MDX_VN], f[MDX_WN], f[MDX_PN], ctx->mu);
    }
    return MDX_OK;
}

// ---- red-black kernel variants and their autotuner ---------------------------
// Variants (all bit-identical per iteration):
//   MDX_SORV_SWEEPS    one launch per colour sweep
//   MDX_SORV_FUSED8    red+black pass, 60x5 tiles, two blocks per SM
//   MDX_SORV_FUSED16   red+black pass, 60x17 or (IBM factors) 60x13 tiles
//   MDX_SORV_SPLIT     one launch per colour sweep on colour-split copies
//                      (tol > 0 only: the copies cost two passes over u, v,
//                      w, p per projection)
//   MDX_SORV_SPLITV    the same with two cells per thread and 16-byte
//                      accesses, the column factors from tables
// All but the first need periodic x and z and mu = 1 or z-invariant.
// (the enum is in mdx_internal.cuh)

static int split_alloc(mdx_ctx_t* ctx) {
    const size_t bytes = sizeof(double) * (size_t)split_elems(ctx->d);
    for (int t = 0; t < 4; ++t)
        if (!ctx->split_f[t]) MDX_CUDA(ctx, cudaMalloc(&ctx->split_f[t], bytes));
    if (!ctx->split_tab) {
        const size_t tb = sizeof(double) * 4 * (size_t)split_plane_elems(ctx->d);
        MDX_CUDA(ctx, cudaMalloc(&ctx->split_tab, tb));
        MDX_CUDA(ctx, cudaMemsetAsync(ctx->split_tab, 0, tb, ctx->stream));
    }
    return MDX_OK;
}

// The column factors of this projection for k_sor_sweep_splitv.
static int split_tables(mdx_ctx_t* ctx, const mdx_sor_params& p) {
    const mdx_dims& d = ctx->d;
    const int py = ctx->bc.is_periodic[1] ? 1 : 0;
    const int nb = (int)std::min<long long>(((long long)d.nxp * d.nyp + 255) / 256, 1024);
    auto kfn = ctx->mu_mode == MU_PLANE ? k_split_tables<MU_PLANE> : k_split_tables<MU_ONE>;
    MDX_LAUNCH(ctx, MDX_T_OTHER, "split tables", kfn, nb, 256, 0, d, py, p, ctx->mu, ctx->split_tab);
    return MDX_OK;
}

static int sor_splitv_iteration(mdx_ctx_t* ctx, const mdx_sor_params& p) {
    const mdx_dims& d = ctx->d;
    double** s = ctx->split_f;
    const int nwin = (d.nx / 2 + 2) / 2;   // windows of two positions covering 0 .. nx/2
    const long long nthr = (long long)nwin * d.ny * d.nz;
    const int nb = (int)((nthr + 127) / 128);   // 128-thread blocks: 5 per SM at 92 registers
    auto kfn = ctx->bc.is_periodic[1] ? k_sor_sweep_splitv<1> : k_sor_sweep_splitv<0>;
    for (int parity = 0; parity < 2; ++parity)
        MDX_LAUNCH(ctx, MDX_T_SOR_SWEEP, "sor sweep split vec", kfn, nb, 128, 0, d, ctx->bcd, p, parity, parity, nwin,
                   s[0], s[1], s[2], s[3], ctx->split_tab);
    return MDX_OK;
}

// u, v, w, p into (to_split) or out of the colour-split copies.
static int split_copy(mdx_ctx_t* ctx, bool to_split) {
    const mdx_dims& d = ctx->d;
    double** f = ctx->f;
    double** s = ctx->split_f;
    const int nb = (int)std::min<long long>((d.npad + 255) / 256, 148 * 16);
    auto kfn = to_split ? k_split_copy<true> : k_split_copy<false>;
    MDX_LAUNCH(ctx, MDX_T_OTHER, "split copy", kfn, nb, 256, 0, d, f[MDX_UN], f[MDX_VN], f[MDX_WN], f[MDX_PN], s[0],
               s[1], s[2], s[3]);
    ctx->split_norms = to_split;
    return MDX_OK;
}

static int sor_split_iteration(mdx_ctx_t* ctx, const mdx_sor_params& p) {
    const mdx_dims& d = ctx->d;
    double** s = ctx->split_f;
    dim3 block(32, 4, 2);
    dim3 grid((d.nx / 2 + 31) / 32, (d.ny + 3) / 4, (d.nz + 1) / 2);
    const bool py = ctx->bc.is_periodic[1] != 0;
    auto kfn = ctx->mu_mode == MU_PLANE ? (py ? k_sor_sweep_split<MU_PLANE, 1> : k_sor_sweep_split<MU_PLANE, 0>)
                                        : (py ? k_sor_sweep_split<MU_ONE, 1> : k_sor_sweep_split<MU_ONE, 0>);
    for (int parity = 0; parity < 2; ++parity)
        MDX_LAUNCH(ctx, MDX_T_SOR_SWEEP, "sor sweep split", kfn, grid, block, 0, d, ctx->bcd, p, parity, parity, s[0],
                   s[1], s[2], s[3], ctx->mu);
    return MDX_OK;
}

static bool fused_ok(const mdx_ctx_t* ctx) {
    return ctx->bc.is_periodic[0] && ctx->bc.is_periodic[2] && ctx->mu_mode != MU_FULL;
}

// The second u, v, w.
static int pass_alloc(mdx_ctx_t* ctx) {
    for (int t = 0; t < 3; ++t)
        if (!ctx->sor_alt[t]) MDX_CUDA(ctx, cudaMalloc(&ctx->sor_alt[t], sizeof(double) * ctx->d.npad));
    return MDX_OK;
}

// The second state without an error where there is no room for it, or no
// allocation may be made: the sweeps do without.
static bool pass_ready(mdx_ctx_t* ctx) {
    if (ctx->sor_alt[2]) return true;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return false;
    for (int t = 0; t < 3; ++t)
        if (!ctx->sor_alt[t] && cudaMalloc(&ctx->sor_alt[t], sizeof(double) * ctx->d.npad) != cudaSuccess) {
            (void)cudaGetLastError();
            ctx->sor_alt[t] = nullptr;
            return false;
        }
    return true;
}

// The pass counts elements of an array in 32 bits.
static bool pass_fits(const mdx_ctx_t* ctx) { return ctx->d.npad < 1LL << 31; }

// Planes per block: the count that ends first, waves of resident blocks times
// (planes + 5 for the halo and the start); steps: those phases.
template <int RY>
static int pass_planes(const mdx_ctx_t* ctx, long long* steps) {
    using G = pass_geom<RY>;
    const mdx_dims& d = ctx->d;
    const long long tiles = (long long)((d.nx + PASS_TX - 1) / PASS_TX) * ((d.ny + G::TY - 1) / G::TY);
    const int slots = 148 * (RY == 8 ? 2 : 1);
    int best = d.nz;
    *steps = -1;
    for (int kz = d.nz; kz >= 4 || kz == d.nz; --kz) {
        const long long t = (tiles * ((d.nz + kz - 1) / kz) + slots - 1) / slots * (kz + 5);
        if (*steps < 0 || t < *steps) {
            *steps = t;
            best = kz;
        }
    }
    return best;
}

// One pass or two colour sweeps?  A phase of all blocks takes 1.75 us at 20
// rows, 1.57 at 16, the time of the two sweeps for 85 000 and 76 000 cells
// (20.6 us a million), whatever the grid; the sweeps win where tiles are
// ragged or the chunks short.  Measured, us an iteration, pass / sweeps:
// 180x150x140 59 / 78, 512x256x256 443 / 733, 240x102x96 37 / 49, 300x300x40
// 61 / 77, 256x128x128 (a fifth column of tiles with 16 of 60 cells) 82 / 86,
// 64x128x256 58 / 45, 128x64x64 17 / 16; with factors 180x150x140 63 / 78,
// 320x200x200 196 / 272.
static bool pass_wins(const mdx_ctx_t* ctx) {
    if (!sor_pxz(ctx) || !pass_fits(ctx)) return false;
    long long steps = 0;
    if (ctx->mu_mode == MU_PLANE) {
        pass_planes<16>(ctx, &steps);
        return steps * 76000 < ctx->d.nint;
    }
    pass_planes<20>(ctx, &steps);
    return steps * 85000 < ctx->d.nint;
}

// One iteration, u, v, w read from src and written to dst, p in place.
template <int RY>
static int sor_pass(mdx_ctx_t* ctx, const mdx_sor_params& p, double* const* src, double* const* dst) {
    using G = pass_geom<RY>;
    const mdx_dims& d = ctx->d;
    const bool py = ctx->bc.is_periodic[1] != 0, plane = ctx->mu_mode == MU_PLANE;
    // the factors' mode is the caller's: MU_PLANE never runs 20 rows, nor 1 16
    constexpr int M0 = RY == 16 ? MU_PLANE : MU_ONE, M1 = RY == 20 ? MU_ONE : MU_PLANE;
    auto kfn = plane ? (py ? k_sor_pass<M1, 1, RY> : k_sor_pass<M1, 0, RY>)
                     : (py ? k_sor_pass<M0, 1, RY> : k_sor_pass<M0, 0, RY>);
    const unsigned bit = 1u << ((RY == 8 ? 0 : 4) + (plane ? 2 : 0) + (py ? 1 : 0));
    if (!(ctx->pass_attr & bit)) {
        MDX_CUDA(ctx, cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::SMEM));
        ctx->pass_attr |= bit;
    }
    long long steps = 0;
    const int KZ = ctx->opts.sor_kz > 0 ? ctx->opts.sor_kz : pass_planes<RY>(ctx, &steps);
    const dim3 grid((d.nx + PASS_TX - 1) / PASS_TX, (d.ny + G::TY - 1) / G::TY, (d.nz + KZ - 1) / KZ);
    MDX_LAUNCH(ctx, MDX_T_SOR_SWEEP, "sor pass", kfn, grid, 32 * RY, G::SMEM, d, ctx->bcd, p, KZ, src[0], src[1],
               src[2], dst[0], dst[1], dst[2], ctx->f[MDX_PN], ctx->mu);
    return MDX_OK;
}

// u, v, w and the second state change places.
template <int RY>
static int sor_pass_swap(mdx_ctx_t* ctx, const mdx_sor_params& p) {
    double** f = ctx->f;
    const int ids[3] = {MDX_UN, MDX_VN, MDX_WN};
    double* cur[3] = {f[MDX_UN], f[MDX_VN], f[MDX_WN]};
    MDX_TRY(sor_pass<RY>(ctx, p, cur, ctx->sor_alt));
    for (int t = 0; t < 3; ++t) std::swap(f[ids[t]], ctx->sor_alt[t]);
    return MDX_OK;
}

static int sor_iterate(mdx_ctx_t* ctx, const mdx_sor_params& p, int variant) {
    if (variant == MDX_SORV_SPLIT) return sor_split_iteration(ctx, p);
    if (variant == MDX_SORV_SPLITV) return sor_splitv_iteration(ctx, p);
    if (variant == MDX_SORV_FUSED8) return sor_pass_swap<8>(ctx, p);
    if (variant == MDX_SORV_FUSED16) return (ctx->mu_mode == MU_PLANE ? sor_pass_swap<16>(ctx, p) : sor_pass_swap<20>(ctx, p));
    return sor_iteration(ctx, p);
}

// *variant: plain sweeps where the device refuses the on-chip run.
static int sor_iterations(mdx_ctx_t* ctx, const mdx_sor_params& p, int* variant, int n) {
    if (*variant == MDX_SORV_RESIDENT) {
        const int rc = n > 0 ? mdx_res_face64_run(ctx, p, n) : MDX_OK;
        if (rc != MDX_RES_REFUSED) return rc;
        *variant = MDX_SORV_SWEEPS;
    }
    for (int it = 0; it < n; ++it) MDX_TRY(sor_iterate(ctx, p, *variant));
    return MDX_OK;
}

// The IBM factors of this projection's dt_gamma.
static int mu_tables(mdx_ctx_t* ctx, double dg) {
    const mdx_dims& d = ctx->d;
    if (ctx->ibm_zero) {
        ctx->mu_mode = MU_ONE;
        return MDX_OK;
    }
    const bool plane = ctx->coef_zinv;
    const long long n = plane ? (long long)d.nxp * d.nyp : d.npad;
    if (!ctx->mu || ctx->mu_elems < 3 * n) {
        cudaFree(ctx->mu);
        ctx->mu = nullptr;
        MDX_CUDA(ctx, cudaMalloc(&ctx->mu, sizeof(double) * 3 * n));
        ctx->mu_elems = 3 * n;
    }
    ctx->mu_mode = plane ? MU_PLANE : MU_FULL;
    const int nb = (int)std::min<long long>((n + 255) / 256, 4096);
    MDX_LAUNCH(ctx, MDX_T_OTHER, "mu tables", k_mu_tables, nb, 256, 0, n, dg, ctx->f[MDX_COEF_U],
               ctx->f[MDX_COEF_V], ctx->f[MDX_COEF_W], ctx->mu);
    return MDX_OK;
}

int mdx_k_projection_redblack(mdx_ctx_t* ctx, double dg, mdx_solve_stats_t* st) {
    const mdx_dims& d = ctx->d;
    double** f = ctx->f;
    const size_t bytes = sizeof(double) * d.npad;
    MDX_TRY(mu_tables(ctx, dg));
    const mdx_solver_opts_t& o = ctx->opts;
    // kernel variant: the requested one, the tuned one, or -- while tuning --
    // the next untried candidate for each residual-check block
    const bool fok = fused_ok(ctx);
    int want = ctx->opts.sor_variant;
    if (want < MDX_SORV_AUTO || want > MDX_SORV_RESIDENT) want = MDX_SORV_AUTO;
    const bool warm = mdx_guess_supported(ctx) && (ctx->guess_mode != MDX_GUESS_ZERO || ctx->record_increments);
    // Where the state fits the SMs the on-chip run is taken without tuning:
    // to a tolerance it was the fastest on every grid and check_every measured
    // (ms a step, on chip / colour sweeps: 116x70x62 3.48 / 3.80 checking every
    // iteration, 1.57 / 2.80 every 50; 128x64x64 2.94 / 3.25 and 1.31 / 2.83).
    // A short fixed count pays more for the copies of u* and for taking the
    // boxes on chip and back than the sweeps that read u* (us a step, 1, 2, 3,
    // 4 iterations: 32x24x32 112 130 136 149 / 99 124 149 173, 128x64x64 204
    // 226 237 256 / 153 204 253 302, 128x96x80 320 351 379 408 / 210 284 356
    // 431).
    const int least = d.nint > 600000 ? 4 : 3;
    const bool brief = want == MDX_SORV_AUTO && o.tol <= 0.0 && o.n_iter < least && !warm;
    if ((want == MDX_SORV_AUTO || want == MDX_SORV_RESIDENT))
        want = !brief && mdx_res_face64_ok(ctx) ? MDX_SORV_RESIDENT : MDX_SORV_AUTO;
    if (want != MDX_SORV_SWEEPS && !fok) want = MDX_SORV_SWEEPS;
    if ((want == MDX_SORV_FUSED8 || want == MDX_SORV_FUSED16) && !pass_fits(ctx)) want = MDX_SORV_SWEEPS;
    // :63-84 -- u <- u* over the whole padded arrays; a fixed number of plain
    // sweeps does it in its first sweep (three copies of 30 MB, 35 us, on
    // 180x150x140)
    int fixed_v = want;
    if (want == MDX_SORV_AUTO) {
        fixed_v = ctx->sor_tuned > 0 ? ctx->sor_tuned : MDX_SORV_SWEEPS;
        if (o.tol <= 0.0 && !warm && ctx->sor_tuned == 0 && pass_wins(ctx) && pass_ready(ctx)) fixed_v = MDX_SORV_FUSED16;
    }
    const bool fixed_pass = fixed_v == MDX_SORV_FUSED8 || fixed_v == MDX_SORV_FUSED16;
    const bool copy_in_sweep = o.tol <= 0.0 && o.n_iter > 0 && !warm && sor_pxz(ctx) &&
                               (fixed_v == MDX_SORV_SWEEPS || fixed_pass);
    if (!copy_in_sweep) {
        MDX_CUDA(ctx, cudaMemcpyAsync(f[MDX_UN], f[MDX_US], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        MDX_CUDA(ctx, cudaMemcpyAsync(f[MDX_VN], f[MDX_VS], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        MDX_CUDA(ctx, cudaMemcpyAsync(f[MDX_WN], f[MDX_WS], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    }
    // Residual scale of this projection, on u* before any guess: converged
    // when ||div u|| <= max(tol*||div u*||, atol); the default atol is the
    // round-off level of the divergence, below which a relative target
    // cannot be met once u* is nearly solenoidal.
    double r0 = 0.0, umax = 0.0, atol = 0.0, target = 0.0;
    if (o.tol > 0.0) {
        double linf = 0.0;
        MDX_TRY(mdx_k_div_norms(ctx, f[MDX_UN], f[MDX_VN], f[MDX_WN], &r0, &linf, &umax));
        atol = (o.atol < 0.0) ? mdx_div_floor(ctx, umax) : o.atol;
        target = std::max(o.tol * r0, atol);
    }
    // warm start: record this projection's increment; apply a guess
    if (warm) MDX_TRY(mdx_warm_begin(ctx));
    bool guessed = false;
    double rg = r0;   // ||div u|| after the guess
    if (warm && ctx->guess_mode != MDX_GUESS_ZERO) MDX_TRY(mdx_guess_apply(ctx, dg, r0, &guessed, &rg));
    if (o.precision == MDX_PREC_MIXED) {   // FP32 sweeps in FP64 defect correction
        bool handled = false;
        MDX_TRY(mdx_k_projection_redblack_mixed(ctx, dg, st, &handled, r0, umax, atol));
        if (handled) {
            ctx->last.guessed = guessed ? 1 : 0;
            if (st) st->guessed = ctx->last.guessed;
            if (warm) MDX_TRY(mdx_warm_end(ctx, ctx->last.status == MDX_OK, ctx->last.iterations));
            return MDX_OK;
        }
    }
    const int may = o.tol > 0.0 ? want : fixed_v;   // a fixed count never tunes
    const bool splitv = may == MDX_SORV_AUTO || may == MDX_SORV_SPLITV;
    if (may == MDX_SORV_SPLIT || splitv) MDX_TRY(split_alloc(ctx));
    const mdx_sor_params p = sor_params(ctx, dg);
    if (splitv) MDX_TRY(split_tables(ctx, p));
    // where u, v, w, p live while the sweeps run: the colour-split copies for
    // MDX_SORV_SPLIT blocks, the reference arrays for the others
    bool in_split = false;
    bool fused_ready = false;
    auto layout_for = [&](int v) -> int {
        if ((v == MDX_SORV_FUSED8 || v == MDX_SORV_FUSED16) && !fused_ready) {
            // the passes write neither ghosts nor the values beyond y walls
            MDX_TRY(pass_alloc(ctx));
            const int ids[3] = {MDX_UN, MDX_VN, MDX_WN};
            for (int t = 0; t < 3; ++t)
                MDX_CUDA(ctx, cudaMemcpyAsync(ctx->sor_alt[t], f[ids[t]], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
            fused_ready = true;
        }
        if ((v == MDX_SORV_SPLIT || v == MDX_SORV_SPLITV) != in_split) {
            in_split = !in_split;
            MDX_TRY(split_copy(ctx, in_split));
        }
        return MDX_OK;
    };
    auto pick = [&]() -> int {
        if (want == MDX_SORV_RESIDENT && ctx->rs_refused) want = MDX_SORV_SWEEPS;
        if (want != MDX_SORV_AUTO) return want;
        if (ctx->sor_tuned > 0) return ctx->sor_tuned;
        auto out = [&](int v) { return !pass_fits(ctx) && (v == MDX_SORV_FUSED8 || v == MDX_SORV_FUSED16); };
        for (int v = MDX_SORV_SWEEPS; v < MDX_SORV_NUM; ++v)
            if (ctx->sor_tune_ms[v] <= 0.0 && !out(v)) return v;
        int best = MDX_SORV_SWEEPS;
        for (int v = MDX_SORV_SWEEPS; v < MDX_SORV_NUM; ++v)
            if (ctx->sor_tune_ms[v] < ctx->sor_tune_ms[best] && !out(v)) best = v;
        ctx->sor_tuned = best;
        return best;
    };
    mdx_solve_stats_t s{};
    s.guessed = guessed ? 1 : 0;
    if (o.tol <= 0.0) {
        int v = fixed_v;
        if (!copy_in_sweep) MDX_TRY(layout_for(v));
        if (copy_in_sweep && fixed_pass) MDX_TRY(pass_alloc(ctx));
        mdx_event_pair run{};
        mdx_sweep_run_begin(ctx, &run);
        if (copy_in_sweep && fixed_pass) {   // u* -> ... -> u, by turns through the second state
            MDX_TRY(shell_copy(ctx));
            double* const us[3] = {f[MDX_US], f[MDX_VS], f[MDX_WS]};
            double* const un[3] = {f[MDX_UN], f[MDX_VN], f[MDX_WN]};
            double* const* src = us;
            for (int left = o.n_iter; left > 0; --left) {
                double* const* dst = left % 2 ? un : ctx->sor_alt;
                MDX_TRY(v == MDX_SORV_FUSED8 ? sor_pass<8>(ctx, p, src, dst)
                        : ctx->mu_mode == MU_PLANE ? sor_pass<16>(ctx, p, src, dst)
                                                   : sor_pass<20>(ctx, p, src, dst));
                src = dst;
            }
        } else {
            if (copy_in_sweep) MDX_TRY(sor_iteration(ctx, p, true));
            MDX_TRY(sor_iterations(ctx, p, &v, o.n_iter - (copy_in_sweep ? 1 : 0)));
        }
        mdx_sweep_run_end(ctx, &run, v == MDX_SORV_RESIDENT || (copy_in_sweep && !fixed_pass) ? 2LL * o.n_iter
                                     : copy_in_sweep ? o.n_iter : -1);
        MDX_TRY(layout_for(MDX_SORV_SWEEPS));
        s.variant = v;
        s.iterations = o.n_iter;
        s.status = MDX_OK;
    } else {
        double linf = 0.0, r = rg;
        s.residual0 = r0;
        s.atol = atol;
        if (!std::isfinite(r0) || !std::isfinite(umax) || !std::isfinite(r)) {
            s.status = MDX_ERR_NONFINITE;
        } else if (r <= target) {
            s.status = MDX_OK;
            s.residual = (r0 > 0.0) ? r / r0 : 0.0;
        } else {
            int it = 0;
            s.status = MDX_NOT_CONVERGED;
            mdx_check_schedule cs;
            cs.start(o.check_every, o.check_mode, r);
            int block = cs.every;
            while (it < o.max_iter) {
                const int m = std::min(block, o.max_iter - it);
                int v = pick();
                MDX_TRY(layout_for(v));
                const bool timing_block = want == MDX_SORV_AUTO && ctx->sor_tuned == 0;
                if (timing_block) MDX_CUDA(ctx, cudaEventRecord(ctx->tune_ev[0], ctx->stream));
                mdx_event_pair run{};
                mdx_sweep_run_begin(ctx, &run);
                MDX_TRY(sor_iterations(ctx, p, &v, m));
                mdx_sweep_run_end(ctx, &run, v == MDX_SORV_RESIDENT ? 2LL * m : -1);
                if (timing_block) MDX_CUDA(ctx, cudaEventRecord(ctx->tune_ev[1], ctx->stream));
                it += m;
                s.variant = v;
                double** uvw = in_split ? ctx->split_f : nullptr;
                MDX_TRY(mdx_k_div_norms(ctx, uvw ? uvw[0] : f[MDX_UN], uvw ? uvw[1] : f[MDX_VN],
                                        uvw ? uvw[2] : f[MDX_WN], &r, &linf));
                MDX_TRY(mdx_res_check(ctx));
                if (timing_block) {   // the norms synchronised the stream; time per iteration
                    float ms = 0.f;
                    if (cudaEventElapsedTime(&ms, ctx->tune_ev[0], ctx->tune_ev[1]) == cudaSuccess)
                        ctx->sor_tune_ms[v] = ms > 0.f ? ms / m : 1e-9;
                }
                if (!std::isfinite(r)) { s.status = MDX_ERR_NONFINITE; break; }
                if (r <= target) { s.status = MDX_OK; break; }
                block = cs.next(it, r, target);
            }
            MDX_TRY(layout_for(MDX_SORV_SWEEPS));
            s.iterations = it;
            s.residual = r / r0;
        }
    }
    if (warm) MDX_TRY(mdx_warm_end(ctx, o.tol > 0.0 && s.status == MDX_OK, s.iterations));
    ctx->last = s;
    if (st) *st = s;
    return MDX_OK;
}
