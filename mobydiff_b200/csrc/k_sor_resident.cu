// k_sor_resident.cu -- red-black sweeps with the whole state on chip.
//
// One cooperative launch makes a run of iterations (the sweeps between two
// residual checks).  The grid is cut into one box of rows per SM: by rows in
// y times bz planes in z, each row whole in x.  A thread owns a fixed
// (i, j) column window and marches its planes; what only it touches stays in
// its registers for the whole run, what its block shares lies in shared
// memory, and only the values on the faces between boxes travel: each as a
// 16-byte word, its halves a payload and a sequence number each, written
// straight into the neighbouring block's inbox in global memory (L2) and
// polled there: there is no separate flag, no fence and no grid barrier, and
// a block waits for its own neighbours only.  Inboxes alternate by sweep: a
// block can only write sweep h's words after its neighbours' words of sweep
// h-1 arrived, which they sent after reading sweep h-2's.
//
// What bounds it: for small grids the chain of a sweep -- compute, one L2
// write, one L2 poll, one block barrier; 1.4 us a colour sweep on 64x32x32,
// of which 0.4 are the compute.  For grids that fill the SMs the compute and
// the face words: 2.7 + 2.1 us on 256x128x128 (47 KB of words each way per SM
// and sweep).  Measured per colour sweep, against the fastest of the other
// kernels on the same grid: potential form 256x128x128 4.7 us (6.9, one
// cooperative launch with grid barriers), 116x70x62 1.9 (6.1, a launch per
// sweep); FP32 faces 118x70x62 2.0 (6.2); FP64 faces 128x64x64 2.8 (6.2).
//
// Every wait is bounded: a block that gives up sets the host's error word and
// returns, and so do its neighbours.  Co-residency comes from the
// cooperative launch (one block per SM, at most as many blocks as SMs).
//
// Per-cell arithmetic: pot_e / sweep32_update (mdx_cell32.cuh) and
// sor_cell_fac (mdx_cell.cuh), as in the other kernels, so the same bits.
#include "mdx_cell.cuh"
#include "mdx_cell32.cuh"
#include "mdx_pot.cuh"
#include "mdx_resident.cuh"
#include "mdx_resident_dev.cuh"


namespace {

// ---------------------------------------------------------------------------
// Potential form (k_sor_mixed.cu): Phi of both colours of the box with a
// one-row halo in shared memory, r~ and the columns' coefficients in
// registers.  A thread owns positions q, q+1 of both colours (four cells) of
// its row in each of its planes.  In plane m its swept cells have odd i when
// the thread's parity t0 + m is odd (for the first colour; the other way
// round for the second), so the two coefficient sets are loaded in the order
// the planes alternate and no select is needed for them.
//
// The two cells of a window go through the packed FP32 instructions (each
// half rounded as the scalar one; c - x is fma(x, -1, c), one rounding), and
// planes are taken two at a time so that the second plane's loads are in
// flight while the first is computed.
// ---------------------------------------------------------------------------
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float lo2(f2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi2(f2 a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, 0xbf800000bf800000ull, a); }
__device__ __forceinline__ f2 ld2s(const float* p) { return *reinterpret_cast<const f2*>(p); }
__device__ __forceinline__ void st2s(float* p, f2 v) { *reinterpret_cast<f2*>(p) = v; }

template <int PY, int KZ>
__global__ void __launch_bounds__(512, 1)
k_pot_resident(pot_geom L, res_geom R, int iters, float* __restrict__ phi, const float* __restrict__ r,
               const float4* __restrict__ tab, word* __restrict__ box, unsigned seq, int* __restrict__ err) {
    constexpr int NB = 4, PG = KZ > 8 ? 1 : 2;   // words in flight, planes taken together (registers)
    extern __shared__ __align__(16) float S[];
    const int half = L.nx / 2, tpr = half / 2, ncol = L.nx + 2;
    const res_box b = make_box<PY>(L.ny, L.nz, R.nyb, (int)gridDim.x / R.nyb, tpr, 0, (int)blockIdx.x);
    const int tid = threadIdx.x, T = blockDim.x;
    const int RZ = (b.nj + 2) * half, SC = RZ * (b.nk + 2);   // one plane, one colour
    // the last group's second plane may lie one past the halo: read, not used
    int* const DT = reinterpret_cast<int*>(S + 2 * SC + RZ);  // where each received word goes
    const int nzw = b.nj * tpr, nyw = b.nk * tpr, nylo = b.ylo >= 0 ? nyw : 0;
    const int nw = 2 * nzw + nylo + (b.yhi >= 0 ? nyw : 0);
    // Phi with its halo (the copies of wrapped rows and planes are in global memory)
    for (int t = tid; t < 2 * (b.nk + 2) * (b.nj + 2) * tpr; t += T) {
        const int qi = t % tpr, row = t / tpr;
        const int jj = row % (b.nj + 2), rk = row / (b.nj + 2);
        const int kk = rk % (b.nk + 2), c = rk / (b.nk + 2);
        const float2 v = __ldcg(reinterpret_cast<const float2*>(phi + pot_row(L, c, b.j0 - 1 + jj, b.k0 - 1 + kk) + 4) + qi);
        *reinterpret_cast<float2*>(S + c * SC + kk * RZ + jj * half + 2 * qi) = v;
    }
    for (int t = tid; t < nw; t += T) {
        if (t < 2 * nzw) {
            const int hi = t >= nzw ? 1 : 0;
            DT[t] = hi * (b.nk + 1) * RZ + half + 2 * (t - hi * nzw);
        } else {
            const int y = t - 2 * nzw, hi = y >= nylo ? 1 : 0, x = y - hi * nylo, m = x / tpr;
            DT[t] = (m + 1) * RZ + hi * (b.nj + 1) * half + 2 * (x - m * tpr);
        }
    }
    const int jj = tid / tpr, qi = tid - jj * tpr, q = 2 * qi;
    const bool act = jj < b.nj;
    const int j = b.j0 + jj;
    const int o0 = RZ + (jj + 1) * half + q;           // own window of plane 0 of the box
    const bool par = ((1 + j + b.k0) & 1) != 0;        // first colour, plane 0: swept cells have odd i
    const int xl = (q == 0 ? half - 1 : -1);           // offset of the x neighbour outside the window, swept
    const int xr = (q + 2 == half ? 2 - half : 2);     // cells with odd i / even i (x periodic)
    const int xo[2] = {par ? xl : xr, par ? xr : xl};
    f2 rr[KZ][2], axl[2], axr[2], ayl[2], ayr[2], az[2], fc[2];
    if (act) {
        const float4* t0 = tab + j * ncol + 2 * q + 1;
        const float4* t1 = t0 + ncol;
        float4 c[5];
        float up[4];
#pragma unroll
        for (int m = 0; m < 5; ++m) c[m] = __ldg(t0 + m);
#pragma unroll
        for (int m = 0; m < 4; ++m) up[m] = __ldg(&t1[m].y);
#pragma unroll
        for (int s = 0; s < 2; ++s) {   // set s: the cells swept in planes of parity s
            const bool odd = (s == 0) == par;
            const float4 a0 = odd ? c[0] : c[1], a1 = odd ? c[2] : c[3], n0 = odd ? c[1] : c[2], n1 = odd ? c[3] : c[4];
            axl[s] = pack2(a0.x, a1.x);
            axr[s] = pack2(n0.x, n1.x);
            ayl[s] = pack2(a0.y, a1.y);
            ayr[s] = odd ? pack2(up[0], up[2]) : pack2(up[1], up[3]);
            az[s] = pack2(a0.z, a1.z);
            fc[s] = pack2(a0.w, a1.w);
        }
#pragma unroll
        for (int m = 0; m < KZ; ++m)
            if (m < b.nk)
#pragma unroll
                for (int c2 = 0; c2 < 2; ++c2)
                    rr[m][c2] = __ldg(reinterpret_cast<const f2*>(r + pot_row(L, c2, j, b.k0 + m) + 4 + q));
    }
    const bool slo = act && jj == 0 && b.ylo >= 0, shi = act && jj == b.nj - 1 && b.yhi >= 0;
    __syncthreads();

    // one cell pair: swept cells c, other colour's x window z0 and the value
    // xs beside it, rows ym, yp, planes zm, zp
    auto cells = [&](int s, f2 rc, f2 c, f2 z0, float xs, f2 ym, f2 yp, f2 zm, f2 zp) -> f2 {
        const bool odd = (s == 0) == par;
        const f2 zl = pack2(xs, lo2(z0)), zr = pack2(hi2(z0), xs);
        f2 e = fma2(axl[s], sub2(c, odd ? zl : z0), rc);   // pot_e
        e = fma2(axr[s], sub2(c, odd ? z0 : zr), e);
        e = fma2(ayl[s], sub2(c, ym), e);
        e = fma2(ayr[s], sub2(c, yp), e);
        e = fma2(az[s], add2(sub2(c, zm), sub2(c, zp)), e);
        return fma2(fc[s], e, c);
    };
    auto sweep = [&](auto csc, unsigned sq) -> bool {
        constexpr int CS = decltype(csc)::value;
        float* W = S + CS * SC;
        const int ph = (int)(sq & 1u), at = here(tid);
        if (act) {
            const float* o = S + (1 - CS) * SC + here(o0);   // the other colour, not written by this sweep
            float* w = W + here(o0);
            // this thread's values on the box's surface go to the neighbours
            // as they are made, so most have arrived when they are waited for
            auto out = [&](word* p, f2 v) { st_word(p, (unsigned)v, (unsigned)(v >> 32), sq); };
            word* const yl = inbox(box, R, b.ylo, ph) + b.wlo;
            word* const yu = inbox(box, R, b.yhi, ph) + b.whi;
            word* py = (slo ? yl : yu) + here(qi);
            auto out_y = [&](word* p, f2 v) {
                out(p, v);
                if (b.nj == 1 && slo && shi) out(p + (yu - yl), v);
            };
            f2 zm = ld2s(o - RZ), z0 = ld2s(o), vt = 0;
#pragma unroll
            for (int m = 0; m < KZ; m += PG) {
                if (m >= b.nk) break;
                constexpr int s0 = 1 - CS, s1 = CS;        // coefficient sets of even and odd planes' swept cells
                if constexpr (PG == 2) {
                    const f2 z1 = ld2s(o + RZ), z2 = ld2s(o + 2 * RZ);
                    const f2 ym0 = ld2s(o - half), yp0 = ld2s(o + half), c0 = ld2s(w);
                    const float xs0 = o[xo[s0]];
                    const f2 ym1 = ld2s(o + RZ - half), yp1 = ld2s(o + RZ + half), c1 = ld2s(w + RZ);
                    const float xs1 = (o + RZ)[xo[s1]];
                    const f2 v0 = cells(s0, rr[m][CS], c0, z0, xs0, ym0, yp0, zm, z1);
                    const f2 v1 = cells(s1, rr[m + 1][CS], c1, z1, xs1, ym1, yp1, z0, z2);
                    const bool two = m + 1 < b.nk;
                    st2s(w, v0);
                    if (two) st2s(w + RZ, v1);
                    if (m == 0) out(inbox(box, R, b.zlo, ph) + nzw + at, v0);
                    vt = two ? v1 : v0;
                    if (slo || shi) {
                        out_y(py, v0);
                        if (two) out_y(py + tpr, v1);
                        py += 2 * tpr;
                    }
                    zm = z1;
                    z0 = z2;
                    o += 2 * RZ;
                    w += 2 * RZ;
                } else {
                    const f2 z1 = ld2s(o + RZ), ym = ld2s(o - half), yp = ld2s(o + half), c = ld2s(w);
                    const float xs = o[xo[(m & 1) ? s1 : s0]];
                    vt = cells((m & 1) ? s1 : s0, rr[m][CS], c, z0, xs, ym, yp, zm, z1);
                    st2s(w, vt);
                    if (m == 0) out(inbox(box, R, b.zlo, ph) + nzw + at, vt);
                    if (slo || shi) {
                        out_y(py, vt);
                        py += tpr;
                    }
                    zm = z0;
                    z0 = z1;
                    o += RZ;
                    w += RZ;
                }
            }
            out(inbox(box, R, b.zhi, ph) + at, vt);
        }
        // the neighbours' values into the halo, NB words in flight per thread
        const word* in = inbox(box, R, b.self, ph);
        bool ok = true;
        for (int t = at; t < nw; t += NB * T) {
            word v[NB];
#pragma unroll
            for (int u = 0; u < NB; ++u)
                if (t + u * T < nw) v[u] = ld_word(in + t + u * T);
#pragma unroll
            for (int u = 0; u < NB; ++u)
                if (t + u * T < nw) {
                    ok = wait_word<WAIT_LIMIT_BEHIND>(in + t + u * T, sq, v[u]) && ok;
                    st2s(W + DT[t + u * T], (f2)v[u].a | (f2)v[u].b << 32);
                }
        }
        return __syncthreads_or(!ok) == 0;
    };
    for (int it = 0; it < iters; ++it) {
        // first colour i+j+k odd, as the face form
        if (!sweep(std::integral_constant<int, 1>(), seq + 2 * it + 1) ||
            !sweep(std::integral_constant<int, 0>(), seq + 2 * it + 2)) {
            if (tid == 0) *err = 1;
            return;
        }
    }
    // back to global memory with the copies of wrapped cells, rows and planes
    if (!act) return;
    for (int m = 0; m < b.nk; ++m)
        for (int c = 0; c < 2; ++c) {
            const int k = b.k0 + m;
            const float2 v = *reinterpret_cast<const float2*>(S + c * SC + o0 + m * RZ);
            float* g = phi + pot_row(L, c, j, k) + 4 + q;
            auto put = [&](int off) { *reinterpret_cast<float2*>(g + off) = v; };
            put(0);
            const bool odd = ((c + j + k) & 1) != 0;
            if (odd && q == 0) g[half] = v.x;               // cell nx+1 = cell 1
            if (!odd && q + 2 == half) g[-q - 1] = v.y;     // cell 0 = cell nx
            if (k == L.nz) put(-L.nz * L.rz);
            if (k == 1) put(L.nz * L.rz);
            if (PY && j == L.ny) put(-L.ny * L.hq);
            if (PY && j == 1) put(L.ny * L.hq);
        }
}

enum { MU_NONE = 0, MU_PLANES = 1 };   // IBM factors all 1, or one (i, j) plane per component

template <int PY, int MU>
struct faces64 {
    typedef double T;
    static constexpr bool HAS_R = false;
    static constexpr int WAIT = WAIT_LIMIT_BEHIND;
    mdx_dims d;
    mdx_bc_dev bc;
    mdx_sor_params p;
    double *u, *v, *w, *q;
    const double* mu;
    __device__ __forceinline__ long long at(int i, int j, int k) const { return pidx(d, i, j, k); }
    __device__ __forceinline__ T res(int, int, int) const { return 0.0; }
    __device__ __forceinline__ void column(face_col<T>& c, int i, int j) const {
        c.mu_u = c.mu_ux = c.mu_v = c.mu_vy = c.mu_w = 1.0;
        if (MU == MU_PLANES) {
            const long long np = (long long)d.nxp * d.nyp;
            const int ip = i == d.nx ? 1 : i + 1, jp = (PY && j == d.ny) ? 1 : j + 1;
            c.mu_u = __ldg(mu + i + (long long)d.nxp * j);
            c.mu_ux = __ldg(mu + ip + (long long)d.nxp * j);
            c.mu_v = __ldg(mu + np + i + (long long)d.nxp * j);
            c.mu_vy = __ldg(mu + np + i + (long long)d.nxp * jp);
            c.mu_w = __ldg(mu + 2 * np + i + (long long)d.nxp * j);
        }
        c.fac = sor_factor(c.mu_u, c.mu_ux, c.mu_v, c.mu_vy, c.mu_w, c.mu_w, p);
    }
    // inner: a row that touches no wall
    __device__ __forceinline__ void cell(const face_col<T>& c, T, T& u_i, T& u_ip, T& v_j, T& v_jp, T& w_k, T& w_kp,
                                         T& pc, int j, bool inner) const {
        const T one = 1.0;
        const T mu_u = MU ? c.mu_u : one, mu_ux = MU ? c.mu_ux : one, mu_v = MU ? c.mu_v : one,
                mu_vy = MU ? c.mu_vy : one, mu_w = MU ? c.mu_w : one;
        if (inner)
            sor_cell_fac<1, 1, 1>(u_i, u_ip, v_j, v_jp, w_k, w_kp, pc, mu_u, mu_ux, mu_v, mu_vy, mu_w, mu_w, c.fac, p,
                                  bc, 1, j, 1, d.nx, d.ny, d.nz);
        else
            sor_cell_fac<1, PY, 1>(u_i, u_ip, v_j, v_jp, w_k, w_kp, pc, mu_u, mu_ux, mu_v, mu_vy, mu_w, mu_w, c.fac, p,
                                   bc, 1, j, 1, d.nx, d.ny, d.nz);
    }
};

template <int PY>
struct faces32 {
    typedef float T;
    static constexpr bool HAS_R = true;
    static constexpr int WAIT = WAIT_LIMIT_AHEAD;
    mdx_dims d;
    mixed_params P;
    float *u, *v, *w, *q;
    const float *r, *mu, *fac;
    __device__ __forceinline__ long long at(int i, int j, int k) const { return cidx(d, i, j, k); }
    __device__ __forceinline__ T res(int i, int j, int k) const { return __ldg(r + cidx(d, i, j, k)); }
    __device__ __forceinline__ void column(face_col<T>& c, int i, int j) const {
        const int np = split_plane_elems(d);
        const int ip = i == d.nx ? 1 : i + 1, jp = (PY && j == d.ny) ? 1 : j + 1;
        c.mu_u = __ldg(mu + pidx2(d, i, j));
        c.mu_ux = __ldg(mu + pidx2(d, ip, j));
        c.mu_v = __ldg(mu + np + pidx2(d, i, j));
        c.mu_vy = __ldg(mu + np + pidx2(d, i, jp));
        c.mu_w = __ldg(mu + 2 * np + pidx2(d, i, j));
        c.fac = __ldg(fac + pidx2(d, i, j));
    }
    __device__ __forceinline__ void cell(const face_col<T>& c, T rc, T& u_i, T& u_ip, T& v_j, T& v_jp, T& w_k, T& w_kp,
                                         T& pc, int j, bool) const {
        sweep32_update(P, rc, u_i, u_ip, v_j, v_jp, w_k, w_kp, pc, c.mu_u, c.mu_ux, c.mu_v, c.mu_vy, c.mu_w, c.fac,
                       PY || j > 1, PY || j < d.ny);
    }
};

template <class A, int PY, int KZ, int NT>
__global__ void __launch_bounds__(NT, 1)
k_face_resident(const __grid_constant__ A a, res_geom R, int iters, word* __restrict__ box, unsigned seq,
                int* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const res_box b = make_box<PY>(a.d.ny, a.d.nz, R.nyb, (int)gridDim.x / R.nyb, R.tpr, 0, (int)blockIdx.x);
    if (!face_run_box<A, PY, KZ>(a, b, R, iters, box, seq, sm_raw) && threadIdx.x == 0) *err = 1;
}

// ---------------------------------------------------------------------------
// Host side: the cut of the grid, the inboxes, the launches.
// ---------------------------------------------------------------------------
struct res_shape { int kz, threads; };   // planes a thread can hold; threads its registers leave
struct res_plan {
    res_geom R{};
    int blocks = 0, threads = 0, shape = -1;
    size_t smem = 0;
};

// The cut with the shortest sweep: per plane a warp issues about `issue`
// cycles of the SM's time and no less than 100 in sequence, and a face word
// costs about a cycle.  ny rows and nz planes are spread over at most one
// block per SM; a box has at most the shape's planes and threads.
template <class SM>
bool make_plan(const mdx_ctx_t* ctx, int tpr, const res_shape* shapes, int nshapes, int issue, SM&& smem, res_plan* out) {
    const mdx_dims& d = ctx->d;
    int sms = 0, most = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device) != cudaSuccess ||
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    double best = 0.0;
    out->shape = -1;
    if (tpr < 1 || tpr > 128) return false;
    for (int s = 0; s < nshapes; ++s)
        for (int by0 = 1; by0 <= d.ny && by0 * tpr <= shapes[s].threads; ++by0) {
            const int nyb = (d.ny + by0 - 1) / by0, by = (d.ny + nyb - 1) / nyb;
            const int nzb = std::min(d.nz, sms / nyb);
            if (nzb < 1) continue;
            const int bz = (d.nz + nzb - 1) / nzb;
            const size_t bytes = smem(by, bz);
            if (bz > shapes[s].kz || bytes > (size_t)most) continue;
            const int warps = (by * tpr + 31) / 32;
            const double cost = (double)bz * std::max(issue * warps, 100) + (double)(by + bz) * tpr + 0.01 * s;
            if (out->shape >= 0 && cost >= best) continue;
            best = cost;
            out->R = res_geom{nyb, by, bz, tpr, 2 * (by + bz) * tpr};
            out->blocks = nyb * nzb;
            out->threads = (by * tpr + 31) & ~31;
            out->shape = s;
            out->smem = bytes;
        }
    return out->shape >= 0;
}

bool capturing(const mdx_ctx_t* ctx) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return cap != cudaStreamCaptureStatusNone;
}

// The kernels' error word: in the pinned block of the reductions' results.
int* err_word(const mdx_ctx_t* ctx) { return reinterpret_cast<int*>(ctx->red_host + 3); }

// Inboxes for the plan and `iters` iterations' sequence numbers.
int res_prepare(mdx_ctx_t* ctx, const res_plan& P, int iters) {
    MDX_TRY(mdx_reduce_init(ctx));
    MDX_TRY(mdx_res_check(ctx));
    const size_t bytes = sizeof(word) * 2 * (size_t)P.blocks * P.R.stride;
    if (ctx->rs_bytes < bytes) {
        cudaFree(ctx->rs_box);
        ctx->rs_box = nullptr;
        ctx->rs_bytes = 0;
        if (cudaMalloc(&ctx->rs_box, bytes) != cudaSuccess) {   // no room: the sweeps need none
            cudaGetLastError();
            ctx->rs_box = nullptr;
            ctx->rs_refused = true;
            return MDX_RES_REFUSED;
        }
        ctx->rs_bytes = bytes;
        ctx->rs_seq = 0;
    }
    const unsigned limit = res_limit(ctx->rs_polls);
    if (ctx->rs_seq == 0 || ctx->rs_seq < limit || ctx->rs_seq - limit >= SEQ_END - 2u * (unsigned)iters - 2u) {
        MDX_CUDA(ctx, cudaMemsetAsync(ctx->rs_box, 0, ctx->rs_bytes, ctx->stream));
        ctx->rs_seq = limit + 2;
    }
    return MDX_OK;
}

// A run of any length in launches whose numbers fit.
template <class F>
int res_pieces(int iters, F&& run) {
    constexpr int MOST = 1 << 27;
    for (; iters > MOST; iters -= MOST) MDX_TRY(run(MOST));
    return run(iters);
}

template <class F, class... Args>
int res_launch(mdx_ctx_t* ctx, const char* what, F fn, const res_plan& P, int iters, Args... args) {
    MDX_CUDA(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem));
    void* av[] = {&args...};
    mdx_event_pair p{};
    mdx_timer_begin(ctx, MDX_T_SOR_SWEEP, &p);
    const cudaError_t e =
        cudaLaunchCooperativeKernel((const void*)fn, dim3(P.blocks), dim3(P.threads), av, P.smem, ctx->stream);
    mdx_timer_end(ctx, &p);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        cudaGetLastError();
        ctx->rs_refused = true;
        return MDX_RES_REFUSED;
    }
    MDX_CUDA(ctx, e);
    ctx->rs_seq += 2u * (unsigned)iters;
    return mdx_check_launch(ctx, what);
}

const res_shape pot_shapes[] = {{4, 512}, {8, 512}, {16, 512}};
const res_shape face64_shapes[] = {{4, 384}, {8, 320}, {16, 256}};
const res_shape face32_shapes[] = {{4, 512}, {8, 512}, {16, 384}};

bool pot_plan(const mdx_ctx_t* ctx, res_plan* P) {
    const int half = ctx->d.nx / 2;
    return make_plan(ctx, half / 2, pot_shapes, 3, 10,
                     [&](int by, int bz) { return sizeof(float) * ((size_t)(by + 2) * (2 * bz + 5) * half + (size_t)(by + bz) * half); }, P);
}
template <typename T>
bool face_plan(const mdx_ctx_t* ctx, const res_shape* shapes, int issue, res_plan* P) {
    const int tpr = ctx->d.nx / 2;
    return make_plan(ctx, tpr, shapes, 3, issue,
                     [&](int by, int bz) { return face_smem<T>(by, bz, tpr); }, P);
}

template <int PY>
int pot_run(mdx_ctx_t* ctx, const pot_geom& L, int iters) {
    res_plan P;
    if (!pot_plan(ctx, &P)) return mdx_fail(ctx, MDX_ERR_ARG, "resident sweeps: the grid does not fit the SMs");
    MDX_TRY(res_prepare(ctx, P, iters));
    auto fn = P.shape == 0 ? k_pot_resident<PY, 4> : P.shape == 1 ? k_pot_resident<PY, 8> : k_pot_resident<PY, 16>;
    return res_launch(ctx, "pot resident", fn, P, iters, L, P.R, iters, ctx->pt_phi, (const float*)ctx->pt_r,
                      (const float4*)ctx->pt_tab, (word*)ctx->rs_box, ctx->rs_seq, err_word(ctx));
}

template <class A, int PY, int N4, int N8, int N16>
int face_run(mdx_ctx_t* ctx, const A& a, const res_plan& P, int iters) {
    MDX_TRY(res_prepare(ctx, P, iters));
    auto fn = P.shape == 0 ? k_face_resident<A, PY, 4, N4>
                           : P.shape == 1 ? k_face_resident<A, PY, 8, N8> : k_face_resident<A, PY, 16, N16>;
    return res_launch(ctx, "face resident", fn, P, iters, a, P.R, iters, (word*)ctx->rs_box, ctx->rs_seq, err_word(ctx));
}

template <int PY, int MU>
int face64_run(mdx_ctx_t* ctx, const mdx_sor_params& p, const res_plan& P, int iters) {
    double** f = ctx->f;
    const faces64<PY, MU> a{ctx->d, ctx->bcd, p, f[MDX_UN], f[MDX_VN], f[MDX_WN], f[MDX_PN], ctx->mu};
    return face_run<faces64<PY, MU>, PY, 384, 320, 256>(ctx, a, P, iters);
}
template <int PY>
int face32_run(mdx_ctx_t* ctx, const mixed_params& q, const res_plan& P, int iters) {
    const faces32<PY> a{ctx->d, q, ctx->mx_du, ctx->mx_dv, ctx->mx_dw, ctx->mx_dp, ctx->mx_r, ctx->mx_mu, ctx->mx_fac};
    return face_run<faces32<PY>, PY, 512, 512, 384>(ctx, a, P, iters);
}

}  // namespace

bool mdx_res_pot_ok(mdx_ctx_t* ctx) {
    res_plan P;
    return !ctx->rs_refused && pot_plan(ctx, &P) && !capturing(ctx);
}
bool mdx_res_face32_ok(mdx_ctx_t* ctx) {
    res_plan P;
    return !ctx->rs_refused && face_plan<float>(ctx, face32_shapes, 12, &P) && !capturing(ctx);
}
bool mdx_res_face64_ok(mdx_ctx_t* ctx) {
    res_plan P;
    return !ctx->rs_refused && ctx->bc.is_periodic[0] && ctx->bc.is_periodic[2] && ctx->mu_mode != MU_FULL &&
           face_plan<double>(ctx, face64_shapes, 18, &P) && !capturing(ctx);
}

int mdx_res_pot_run(mdx_ctx_t* ctx, const pot_geom& L, int iters) {
    return res_pieces(iters, [&](int n) { return ctx->bc.is_periodic[1] ? pot_run<1>(ctx, L, n) : pot_run<0>(ctx, L, n); });
}
int mdx_res_face32_run(mdx_ctx_t* ctx, const mixed_params& q, int iters) {
    res_plan P;
    if (!face_plan<float>(ctx, face32_shapes, 12, &P))
        return mdx_fail(ctx, MDX_ERR_ARG, "resident sweeps: the grid does not fit the SMs");
    return res_pieces(iters, [&](int n) { return ctx->bc.is_periodic[1] ? face32_run<1>(ctx, q, P, n) : face32_run<0>(ctx, q, P, n); });
}
int mdx_res_face64_run(mdx_ctx_t* ctx, const mdx_sor_params& p, int iters) {
    res_plan P;
    if (!face_plan<double>(ctx, face64_shapes, 18, &P))
        return mdx_fail(ctx, MDX_ERR_ARG, "resident sweeps: the grid does not fit the SMs");
    const bool py = ctx->bc.is_periodic[1] != 0;
    return res_pieces(iters, [&](int n) {
        if (ctx->mu_mode == MU_ONE) return py ? face64_run<1, MU_NONE>(ctx, p, P, n) : face64_run<0, MU_NONE>(ctx, p, P, n);
        return py ? face64_run<1, MU_PLANES>(ctx, p, P, n) : face64_run<0, MU_PLANES>(ctx, p, P, n);
    });
}

int mdx_res_check(mdx_ctx_t* ctx) {
    if (!ctx->red_host || *(volatile int*)err_word(ctx) == 0) return MDX_OK;
    MDX_CUDA(ctx, cudaStreamSynchronize(ctx->stream));   // runs queued behind it may set the word too
    *err_word(ctx) = 0;
    ctx->rs_seq = 0;   // the inboxes are cleared before the next run
    return mdx_fail(ctx, MDX_ERR_TIMEOUT, "resident red-black sweeps: a block gave up waiting for its neighbour");
}

void mdx_res_free(mdx_ctx_t* ctx) {
    cudaFree(ctx->rs_box);
    ctx->rs_box = nullptr;
    ctx->rs_bytes = 0;
    ctx->rs_seq = 0;
    ctx->rs_refused = false;
}
