// mdx_resident_dev.cuh -- device side of the on-chip red-black runs shared by
// the single-channel kernels (k_sor_resident.cu, which describes them) and the
// ensemble: a block's box of the grid, the words blocks exchange, the face
// form's sweeps of one box.
#pragma once

#include "mdx_internal.cuh"

#include <type_traits>

namespace {

struct res_box {          // one block's part of the grid
    int self;             // its number
    int j0, nj, k0, nk;   // first row and number of rows, first plane and number of planes
    int ylo, yhi, zlo, zhi;   // neighbouring blocks (-1: a wall)
    int wlo, whi;             // where this block's words start in ylo's y-hi and yhi's y-lo section
};

__device__ __forceinline__ int cut(int n, int b, int nb) { return (int)(((long long)n * b) / nb); }

// Box `at` of nyb x nzb, whose blocks are numbered from `first`.
template <int PY>
__device__ __forceinline__ res_box make_box(int ny, int nz, int nyb, int nzb, int tpr, int first, int at) {
    res_box b;
    b.self = first + at;
    const int yb = at % nyb, zb = at / nyb;
    b.j0 = 1 + cut(ny, yb, nyb);
    b.nj = cut(ny, yb + 1, nyb) - cut(ny, yb, nyb);
    b.k0 = 1 + cut(nz, zb, nzb);
    b.nk = cut(nz, zb + 1, nzb) - cut(nz, zb, nzb);
    b.ylo = yb > 0 ? b.self - 1 : (PY ? b.self + nyb - 1 : -1);
    b.yhi = yb + 1 < nyb ? b.self + 1 : (PY ? b.self - nyb + 1 : -1);
    b.zlo = zb > 0 ? b.self - nyb : b.self + (nzb - 1) * nyb;
    b.zhi = zb + 1 < nzb ? b.self + nyb : b.self - (nzb - 1) * nyb;
    auto rows = [&](int y) { return cut(ny, y + 1, nyb) - cut(ny, y, nyb); };
    const int lo = yb > 0 ? yb - 1 : nyb - 1, hi = yb + 1 < nyb ? yb + 1 : 0;
    b.wlo = (2 * rows(lo) + (PY || lo > 0 ? b.nk : 0)) * tpr;
    b.whi = 2 * rows(hi) * tpr;
    return b;
}

// The value, unknown to the compiler: what is computed from it inside the
// iteration loop is computed there again instead of being kept in registers
// across it (they hold the state).
__device__ __forceinline__ int here(int x) {
    asm volatile("" : "+r"(x));
    return x;
}

// Two 8-byte halves, each a 32-bit payload and the sequence number: a 64-bit
// access is atomic, so a half whose number matches holds its payload.  (One
// number for the whole 16 bytes was tried as a 128-bit access; words of the
// FP32 faces then came back with the payload of an earlier sweep.)
struct __align__(16) word { unsigned a, sa, b, sb; };

__device__ __forceinline__ void st_word(word* p, unsigned a, unsigned b, unsigned s) {
    asm volatile("{ .reg .b64 lo, hi; mov.b64 lo, {%1, %3}; mov.b64 hi, {%2, %3};"
                 " st.relaxed.gpu.global.v2.b64 [%0], {lo, hi}; }" ::"l"(p), "r"(a), "r"(b), "r"(s)
                 : "memory");
}
__device__ __forceinline__ word ld_word(const word* p) {
    word w;
    asm volatile("{ .reg .b64 lo, hi; ld.relaxed.gpu.global.v2.b64 {lo, hi}, [%4];"
                 " mov.b64 {%0, %1}, lo; mov.b64 {%2, %3}, hi; }"
                 : "=r"(w.a), "=r"(w.sa), "=r"(w.b), "=r"(w.sb)
                 : "l"(p)
                 : "memory");
    return w;
}
// Sequence numbers are 29 bits; the three above say how often a word that has
// not come is read before the block gives up (res_limit; 0: POLLS times, about a
// second).  So the limit needs no register in the sweeps: as a kernel argument
// it cost the FP64 runs 1 to 5 %.  WAIT_POLLS: always POLLS (the ensemble, whose
// numbers are 32 bits).  Where the limit is looked up decides a few registers:
// behind a first look at the word FP64 and potentials gain 1 to 3 % over POLLS
// and FP32 faces lose 1.7, in the loop's head FP64 loses 2 and FP32 faces 0 to
// 1.6.
constexpr int POLLS = 1 << 20;
constexpr unsigned SEQ_END = 1u << 29;
enum { WAIT_POLLS, WAIT_LIMIT_BEHIND, WAIT_LIMIT_AHEAD };
// Limits of 0, 1, 2, 4 .. 32 reads (polls < 0: the usual one).
inline unsigned res_limit(int polls) {
    unsigned c = 0;
    if (polls >= 0)
        for (c = 1; c < 7 && ((1 << c) >> 1) <= polls; ++c) {}
    return c * SEQ_END;
}
__device__ __forceinline__ int first_poll(unsigned seq) {   // the loop below counts up to POLLS
    const unsigned c = seq / SEQ_END;
    return c ? POLLS - ((1 << c) >> 2) : 0;
}
// False when the word did not come.
template <int MODE>
__device__ __forceinline__ bool wait_word(const word* p, unsigned seq, word& w) {
    if constexpr (MODE == WAIT_LIMIT_BEHIND) {
        if (w.sa == seq && w.sb == seq) return true;
        int n = first_poll(seq);
        do {
            if (n == POLLS) return false;
            ++n;
            w = ld_word(p);
        } while (w.sa != seq || w.sb != seq);
    } else {
        for (int n = MODE == WAIT_POLLS ? 0 : first_poll(seq); w.sa != seq || w.sb != seq; ++n) {
            if (n == POLLS) return false;
            w = ld_word(p);
        }
    }
    return true;
}

// Inbox of a block: two parities of [z-lo rows | z-hi rows | y-lo planes |
// y-hi planes], a row or plane of tpr words each, a wall's section empty; the
// stride is that of the largest box.  The halo words a thread of the block
// receives are those at its index, T apart.
struct res_geom {
    int nyb, by, bz;   // blocks along y; rows and planes of the largest box
    int tpr;           // words per row
    int stride;        // words of one inbox, at least 2 (by + bz) tpr
};
__device__ __forceinline__ word* inbox(word* box, const res_geom& R, int block, int parity) {
    return box + ((long long)block * 2 + parity) * R.stride;
}

// ---------------------------------------------------------------------------
// Face form: u, v, w, p of the box (FP64), or the corrections du, dv, dw, dp
// and r~ (FP32).  A thread owns the cell pairs (2 qi + 1, 2 qi + 2) of its
// row in each of its planes.  In registers: p (and r~) of both cells, the x
// face between them and the w faces of its columns, the box's top faces
// included; in shared memory: the x faces between pairs and the y faces.  A
// face lies between a cell of each colour, so a sweep touches it from one
// side only: no two threads of a sweep meet.  The y and z faces on the box's
// surface are held by both blocks; the one whose cell was swept sends it.
//
// F[m] / G[m] name the cell of plane m swept by the first / second colour;
// the column that is F in plane m is G in plane m + 1.  Their side s (0: odd
// i) alternates with the plane, so the factors are loaded in that order.
// ---------------------------------------------------------------------------
template <typename T> struct face_col { T mu_u, mu_ux, mu_v, mu_vy, mu_w, fac; };

__device__ __forceinline__ void send(word* p, double v, unsigned sq) {
    st_word(p, (unsigned)__double2loint(v), (unsigned)__double2hiint(v), sq);
}
__device__ __forceinline__ void send(word* p, float v, unsigned sq) { st_word(p, __float_as_uint(v), 0u, sq); }
__device__ __forceinline__ void value(const word& w, double& v) { v = __hiloint2double((int)w.b, (int)w.a); }
__device__ __forceinline__ void value(const word& w, float& v) { v = __uint_as_float(w.a); }

// Shared memory of a box of by x bz rows of tpr pairs (one plane past the box
// may be read).
template <typename T>
__host__ __device__ inline size_t face_smem(int by, int bz, int tpr) {
    return sizeof(T) * (size_t)(bz + 1) * tpr * (2 * (by + 1) + by) + sizeof(int) * 2 * (size_t)bz * tpr;
}

// `iters` red-black iterations of box b (at most KZ planes) by one block of at
// least nj tpr threads: state in from global memory, sweeps, state out.  False
// when a neighbour's word did not come (nothing is written then).
template <class A, int PY, int KZ>
__device__ __forceinline__ bool face_run_box(const A& a, const res_box& b, const res_geom& R, int iters, word* box,
                                             unsigned seq, unsigned char* sm_raw) {
    typedef typename A::T T;
    const int tpr = R.tpr, tid = threadIdx.x, NTH = blockDim.x;
    T* const V = reinterpret_cast<T*>(sm_raw);               // [nk][nj + 1][side][tpr]
    T* const U = V + b.nk * (b.nj + 1) * 2 * tpr;            // [nk][nj][tpr]
    const int VZ = (b.nj + 1) * 2 * tpr, UZ = b.nj * tpr;    // one plane
    const int jj = tid / tpr, qi = tid - jj * tpr;
    const bool act = jj < b.nj;
    const int j = b.j0 + jj, sb = (j + b.k0) & 1;            // side of F[0]
    const int qn = qi + 1 == tpr ? 0 : qi + 1;
    const bool slo = act && jj == 0 && b.ylo >= 0, shi = act && jj == b.nj - 1 && b.yhi >= 0;
    T pF[KZ], pG[KZ], um[KZ], wF[KZ + 1], wG[KZ + 1], rF[KZ], rG[KZ];
    face_col<T> col[2];                                      // the columns on side sb and on the other
    if (act) {
#pragma unroll
        for (int s = 0; s < 2; ++s) a.column(col[s], 2 * qi + 1 + (sb ^ s), j);
#pragma unroll
        for (int m = 0; m <= KZ; ++m)
            if (m <= b.nk) {   // the top faces wrap to plane 1
                const int k = b.k0 + m > a.d.nz ? 1 : b.k0 + m;
                wF[m] = a.w[a.at(2 * qi + 1 + (sb ^ (m & 1)), j, k)];
                wG[m] = a.w[a.at(2 * qi + 2 - (sb ^ (m & 1)), j, k)];
            }
#pragma unroll
        for (int m = 0; m < KZ; ++m)
            if (m < b.nk) {
                const int k = b.k0 + m;
                const int iF = 2 * qi + 1 + (sb ^ (m & 1)), iG = 2 * qi + 2 - (sb ^ (m & 1));
                pF[m] = a.q[a.at(iF, j, k)];
                pG[m] = a.q[a.at(iG, j, k)];
                if (A::HAS_R) {
                    rF[m] = a.res(iF, j, k);
                    rG[m] = a.res(iG, j, k);
                }
                um[m] = a.u[a.at(2 * qi + 2, j, k)];
                U[m * UZ + tid] = a.u[a.at(2 * qi + 1, j, k)];
                for (int s = 0; s < 2; ++s) {
                    V[m * VZ + (jj * 2 + s) * tpr + qi] = a.v[a.at(2 * qi + 1 + s, j, k)];
                    if (jj == b.nj - 1)
                        V[m * VZ + ((jj + 1) * 2 + s) * tpr + qi] =
                            a.v[a.at(2 * qi + 1 + s, (PY && j == a.d.ny) ? 1 : j + 1, k)];
                }
            }
    }
    // where the received y faces go: the offset of their side 0 and, in the
    // low bit, their side in the first colour's sweeps
    int* const DT = reinterpret_cast<int*>(U + b.nk * UZ);
    const int nzw = b.nj * tpr, nyw = b.nk * tpr, nylo = b.ylo >= 0 ? nyw : 0, nw = nylo + (b.yhi >= 0 ? nyw : 0);
    for (int t = tid; t < nw; t += NTH) {
        const int hi = t >= nylo ? 1 : 0, x = t - hi * nylo, m = x / tpr;
        const int row = hi ? b.j0 + b.nj : b.j0 - 1;   // the neighbour's row
        DT[t] = 2 * (m * VZ + hi * b.nj * 2 * tpr + x - m * tpr) + ((row + b.k0 + m) & 1);
    }
    const bool inner = PY || (j > 1 && j < a.d.ny);
    __syncthreads();

    // one colour sweep: X is swept, Y the other colour's cells
    auto sweep = [&](auto parc, unsigned sq, T(&pX)[KZ], T(&wX)[KZ + 1], T(&wY)[KZ + 1], const T(&rX)[KZ]) -> bool {
        constexpr int PAR = decltype(parc)::value;
        const int ph = (int)(sq & 1u), at = here(tid);
        const word* const in = inbox(box, R, b.self, ph);
        bool ok = true;
        word zl{}, zh{};
        if (act) {
            // sides of the even and odd planes' swept cells, as offsets
            const int se = sb ^ PAR, so = se ^ 1;
            T* const v0 = V + here(jj * 2 * tpr + qi);
            T* const u0 = U + here(jj * tpr);
            T *ve = v0 + (se ? tpr : 0), *vo = v0 + VZ + (so ? tpr : 0);
            T *ue = u0 + (se ? qn : qi), *uo = u0 + UZ + (so ? qn : qi);
            T top = wY[1];
            word* const yl = inbox(box, R, b.ylo, ph) + b.wlo;
            word* const yu = inbox(box, R, b.yhi, ph) + b.whi;
            word* py = (slo ? yl : yu) + here(qi);
            auto cell = [&](int m, int s, T* u, T* v) {   // and its values on the box's surface to the neighbours
                T x = *u, vj = v[0], vjp = v[2 * tpr];
                T ui = s ? um[m] : x, uip = s ? x : um[m];
                a.cell(col[(m + PAR) & 1], rX[m], ui, uip, vj, vjp, wX[m], wY[m + 1], pX[m], j, inner);
                um[m] = s ? ui : uip;
                *u = s ? uip : ui;
                v[0] = vj;
                v[2 * tpr] = vjp;
                top = wY[m + 1];
                if (slo || shi) {
                    send(py, slo ? vj : vjp, sq);
                    if (b.nj == 1 && slo && shi) send(py + (yu - yl), vjp, sq);
                    py += tpr;
                }
            };
#pragma unroll
            for (int m = 0; m < KZ; m += 2) {
                if (m >= b.nk) break;
                cell(m, se, ue, ve);
                if (m == 0) send(inbox(box, R, b.zlo, ph) + nzw + at, wX[0], sq);
                if (m + 1 >= b.nk) break;
                cell(m + 1, so, uo, vo);
                ve += 2 * VZ;
                vo += 2 * VZ;
                ue += 2 * UZ;
                uo += 2 * UZ;
            }
            send(inbox(box, R, b.zhi, ph) + at, top, sq);
            zl = ld_word(in + at);
            zh = ld_word(in + nzw + at);
        }
        // the y faces the neighbours' cells moved
        for (int t = at; t < nw; t += 2 * NTH) {
            word w[2];
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (t + e * NTH < nw) w[e] = ld_word(in + 2 * nzw + t + e * NTH);
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (t + e * NTH < nw) {
                    ok = wait_word<A::WAIT>(in + 2 * nzw + t + e * NTH, sq, w[e]) && ok;
                    const int dst = DT[t + e * NTH];
                    value(w[e], V[(dst >> 1) + ((dst ^ PAR) & 1 ? tpr : 0)]);
                }
        }
        // the z faces: those of the columns this block did not sweep there
        if (act) {
            ok = wait_word<A::WAIT>(in + at, sq, zl) && ok;
            ok = wait_word<A::WAIT>(in + nzw + at, sq, zh) && ok;
            value(zl, wY[0]);
            T v;
            value(zh, v);
#pragma unroll
            for (int m = 1; m <= KZ; ++m) wX[m] = m == b.nk ? v : wX[m];   // selected: the index stays a constant
        }
        return __syncthreads_or(!ok) == 0;
    };
    for (int it = 0; it < iters; ++it) {
        if (!sweep(std::integral_constant<int, 0>(), seq + 2 * it + 1, pF, wF, wG, rF) ||
            !sweep(std::integral_constant<int, 1>(), seq + 2 * it + 2, pG, wG, wF, rG))
            return false;
    }
    if (!act) return true;
#pragma unroll
    for (int m = 0; m < KZ; ++m) {
        if (m >= b.nk) break;
        const int k = b.k0 + m;
        const int iF = 2 * qi + 1 + (sb ^ (m & 1)), iG = 2 * qi + 2 - (sb ^ (m & 1));
        a.w[a.at(iF, j, k)] = wF[m];
        a.w[a.at(iG, j, k)] = wG[m];
        a.q[a.at(iF, j, k)] = pF[m];
        a.q[a.at(iG, j, k)] = pG[m];
        a.u[a.at(2 * qi + 2, j, k)] = um[m];
        a.u[a.at(2 * qi + 1, j, k)] = U[m * UZ + tid];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            a.v[a.at(2 * qi + 1 + s, j, k)] = V[m * VZ + (jj * 2 + s) * tpr + qi];
            if (!PY && j == a.d.ny) a.v[a.at(2 * qi + 1 + s, j + 1, k)] = V[m * VZ + ((jj + 1) * 2 + s) * tpr + qi];
        }
    }
    return true;
}

}  // namespace
