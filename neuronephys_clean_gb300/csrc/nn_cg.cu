// Single-kernel-per-iteration preconditioned CG (Chronopoulos & Gear, "s-step
// iterative methods for symmetric linear systems", J. Comput. Appl. Math. 25,
// 1989) for the 7-point backward-Euler operator
//   A = (1 + beta) I + alpha L_D,  (L_D v)_c = sum over the 6 faces f of
//   c_f (v_c - v_nb), zero values outside the grid (homogeneous Dirichlet),
// Jacobi preconditioner M = 1/diag, for grids that do not fit on the chip.
// With constant coefficients every c_f = 1; with a cell field D (the HET
// variant) c_f is the harmonic mean of D on the two sides of the face, D_c on
// a boundary face, and alpha c_f = 1 / (v_c + v_nb) with v = 1 / (2 alpha D).
//
// The solve is bound by memory, so the recurrences are arranged for the fewest
// bytes.  They run on u = M r and t = M s (s = A p) instead of r and s:
//   t_i = M A u_i + b_i t_{i-1}     u_{i+1} = u_i - a_i t_i
//   p_i = u_i + b_i p_{i-1}         x += a_i p_i
//   g = (r, u), d = (A u, u), rho = (r, r) of u_{i+1}   -> one reduction
//   b_{i+1} = g / g_old,  a_{i+1} = g / (d - b_{i+1} g / a_i)
// - A u is formed twice, for t_i and inside d, instead of being stored between
//   iterations, and d as an energy, sum of c_f (u_c - u_nb)^2 over the faces,
//   which needs each neighbour on one side only;
// - M follows from the faces that A u needs anyway;
// - p and x of a plane are touched in every second iteration, those of the even
//   and of the odd planes in turn: u_{i-1} = u_i + a_{i-1} t_{i-1} is at hand
//   there, so both directions are added at once (k_cg_flush adds the last one
//   where it is missing).
// That is 28 bytes a cell and iteration (24 with constant coefficients) of the
// 48 (40) that storing r, w, s, p, x, D and M moved.  256^3 with a cell field:
// 93 us an iteration against 155.
// Consecutive iterations march in opposite z directions, so that each begins on
// the planes that the one before left in L2.
//
// A block owns a tile of rows (up to 64 quads long) and a chunk of planes; a
// thread holds NR rows of a quad of x cells and marches in z with the planes
// behind and ahead in registers.  TMA copies bring planes of u and v with a
// frame of one row (and one quad, where tiles lie side by side) two steps ahead
// of use, those of t two and those of p and x one.  Boxes are zero outside the
// grid, which is the boundary condition; v has ghost cells.  The rows and the
// plane that the energies of the tile's far faces need beyond it are computed
// twice.  One barrier a plane: what the energies need of a neighbour thread's
// new u is exchanged through shared memory and used a plane later.  Every
// mbarrier wait is bounded.
// The last block to finish sums the block partials in FP64 and forms the next
// iteration's scalars, so no host round trip separates iterations.
// What bounds it: the arithmetic of two operator applications, at 12 warps an SM
// (the registers' limit) 45 % of the issue slots, beside 4.6 TB/s.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>

#include "nn_internal.cuh"
#include "nn_ptx.cuh"
#include "nn_quad.cuh"

namespace {
constexpr int CG_THREADS = 256;      // the elementwise kernels
constexpr int NR = 2;                // rows of a thread (256^3 with a cell field: 93 us; 1: 115, 3: 94, 4: 99)
constexpr int CG_MAX_THREADS = 384;  // k_cg_iter: 154 registers a thread with a cell field, 100 without
constexpr int STAGES = 4;            // planes of u and v in shared memory
constexpr int CG_MAX_QUADS = 64;     // row of a TMA box: 256 cells
constexpr uint32_t WAIT_LIMIT = 1u << 20;

enum { C_GAMMA = 0, C_ALPHA, C_BETA, C_RR, C_BB, C_DELTA, C_ALPHA_P, C_BETA_P, C_COUNT };

struct CgArgs {
    int nx, ny, nz;
    int nq;                       // quads in a row of the plan's vectors (the last one padded with zeros)
    int wq, cq;                   // quads of a tile: owned, computed (one more where another tile follows)
    int rows, rp;                 // rows of a tile: owned; computed by NR
    int ntx, nty, zc;             // tiles in x and y; planes of a tile
    float op_alpha, onepb, invd;  // invd: 1/diag for constant coefficients
    float c, inv_c;               // u = c M r, t = c M s, c a power of two (nn_jacobi_scale)
    int frame;                    // a quad beside the tile is loaded on both sides (more than one tile in x)
    float *u_out, *t_out;
    float *p, *x;                 // x: rows of 4 nq cells
    int it;                       // iteration
    int dir;                      // direction of the march in z, +1 or -1
    double* scal;
    double* partials;
    unsigned int* ticket;
    int* flags;  // [0] stop (1 converged, 2 max_iter, 3 error) [1] iterations [2] wait timeout
    double rtol2;
    int max_iter;
};

// Block totals of nsum thread values (FP64 from the thread on); the last block
// to arrive writes the grid totals to out[] in a fixed order.
template <int nsum>
__device__ __forceinline__ bool cg_reduce(const double* v, double* partials, unsigned int* ticket, double* out)
{
    __shared__ double ws[4][CG_MAX_THREADS / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int q = 0; q < nsum; ++q) {
        const double s = nn_warp_sum(v[q]);
        if (lane == 0) ws[q][w] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 0; q < nsum; ++q) {
            double s = 0.0;
            for (int u = 0; u < nw; ++u) s += ws[q][u];
            partials[(size_t)q * gridDim.x + blockIdx.x] = s;
        }
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
        for (int q = 0; q < nsum; ++q) s[q] += __ldcg(partials + (size_t)q * gridDim.x + b);
    for (int q = 0; q < nsum; ++q) {
        s[q] = nn_warp_sum(s[q]);
        if (lane == 0) ws[q][w] = s[q];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 0; q < nsum; ++q) {
            double t = 0.0;
            for (int u = 0; u < nw; ++u) t += ws[q][u];
            out[q] = t;
        }
        *ticket = 0;
    }
    __syncthreads();
    return true;
}

// Sum of many non-negative terms in two floats.
struct CgSum {
    float h = 0.0f, l = 0.0f;
    __device__ __forceinline__ void add(float v)
    {
        const float s = __fadd_rn(h, v), t = __fsub_rn(s, h);
        l = __fadd_rn(l, __fadd_rn(__fsub_rn(h, __fsub_rn(s, t)), __fsub_rn(v, t)));
        h = s;
    }
    __device__ __forceinline__ double value() const { return (double)h + (double)l; }
};

// The sums' scalars, by one thread of the last block to arrive.
__device__ void cg_scalars(const CgArgs& a, bool init, const double* out)
{
    const double g = out[0], d = out[1], rr = out[2], c2 = (double)a.c * a.c;  // g, d and rr times c2
    a.scal[C_RR] = rr / c2;
    a.scal[C_DELTA] = d;
    if (init) {
        a.scal[C_BB] = out[3];
        a.scal[C_GAMMA] = g;
        a.scal[C_ALPHA] = d != 0.0 ? g / d : 0.0;
        a.scal[C_BETA] = 0.0;
        a.scal[C_ALPHA_P] = 0.0;
        a.scal[C_BETA_P] = 0.0;
        a.flags[1] = 0;
        a.flags[2] = 0;
        a.flags[0] = (rr <= a.rtol2 * c2 * out[3]) ? 1 : 0;
        return;
    }
    const int it = a.flags[1] + 1;
    a.flags[1] = it;
    const double al = a.scal[C_ALPHA], bnew = g / a.scal[C_GAMMA];
    const double denom = d - bnew * g / al;
    a.scal[C_ALPHA_P] = al;
    a.scal[C_BETA_P] = a.scal[C_BETA];
    a.scal[C_BETA] = bnew;
    a.scal[C_ALPHA] = denom != 0.0 ? g / denom : 0.0;
    a.scal[C_GAMMA] = g;
    if (rr <= a.rtol2 * c2 * a.scal[C_BB]) a.flags[0] = 1;
    else if (it >= a.max_iter) a.flags[0] = 2;
    else if (!(std::isfinite(a.scal[C_ALPHA]) && std::isfinite(a.scal[C_BETA]))) a.flags[0] = 3;
}

__device__ __forceinline__ Quad quad_of(const float4& v) { return {{{v.x, v.y}}, {{v.z, v.w}}}; }
__device__ __forceinline__ float4 float4_of(const Quad& q) { return make_float4(q.a.v[0], q.a.v[1], q.b.v[0], q.b.v[1]); }
__device__ __forceinline__ Quad quad_all(float v) { return {vb<2>(v), vb<2>(v)}; }
__device__ __forceinline__ Quad operator+(const Quad& x, const Quad& y) { return {vadd(x.a, y.a), vadd(x.b, y.b)}; }
__device__ __forceinline__ Quad operator-(const Quad& x, const Quad& y) { return {vsub(x.a, y.a), vsub(x.b, y.b)}; }
__device__ __forceinline__ Quad operator*(const Quad& x, const Quad& y) { return {vmul(x.a, y.a), vmul(x.b, y.b)}; }
__device__ __forceinline__ Quad fma(const Quad& x, const Quad& y, const Quad& z)  // x y + z
{
    return {vfma(x.a, y.a, z.a), vfma(x.b, y.b, z.b)};
}
__device__ __forceinline__ Quad rcp(const Quad& x) { return {vrcp(x.a), vrcp(x.b)}; }
__device__ __forceinline__ float sum(const Quad& x)
{
    const V2 t = vadd(x.a, x.b);
    return t.v[0] + t.v[1];
}

// Shared memory of k_cg_iter in bytes: STAGES planes of u (and v) with a frame of
// one row and, beside other tiles, one quad; three planes of t and one each of p
// and x; two planes of what neighbours read of the new u: the first row of every
// thread and the first cell of every quad.
struct CgSmem {
    int box, own, ey, ex, total;
    __host__ __device__ CgSmem(int cq, int rp, bool frame, bool het)
    {
        box = ((cq + (frame ? 2 : 0)) * (NR * rp + 2) * 16 + 127) & ~127;
        own = (cq * NR * rp * 16 + 127) & ~127;
        ey = STAGES * box * (het ? 2 : 1) + 5 * own;
        ex = ey + 2 * rp * cq * 16;
        total = ex + 2 * NR * rp * cq * 4 + 128;  // the base is aligned to 128 bytes
    }
};

// INIT: r0 = b - A x and its sums in the place of an iteration's (tm_u, tm_t: x, b).
template <bool HET, bool INIT>
__global__ void __launch_bounds__(CG_MAX_THREADS, 1)
    k_cg_iter(const __grid_constant__ CUtensorMap tm_u, const __grid_constant__ CUtensorMap tm_v,
              const __grid_constant__ CUtensorMap tm_t, const __grid_constant__ CUtensorMap tm_p,
              const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CgArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bars[STAGES + 1];
    __shared__ int abort_flag;
    unsigned char* const smem = smem_raw + (-nn_smem_u32(smem_raw) & 127u);
    const int tid = threadIdx.x, cq = a.cq, rp = a.rp, BW = cq + (a.frame ? 2 : 0);
    const CgSmem L(cq, rp, a.frame != 0, HET);
    float4* const ey = reinterpret_cast<float4*>(smem + L.ey);  // [2][rp][cq]
    float* const ex = reinterpret_cast<float*>(smem + L.ex);    // [2][NR rp][cq]
    const int tx = blockIdx.x % a.ntx, ty = blockIdx.x / a.ntx % a.nty, tz = blockIdx.x / (a.ntx * a.nty);
    const int Q0 = tx * a.wq, Y0 = ty * a.rows, Z0 = tz * a.zc;
    const int n = min(a.zc, a.nz - Z0);                   // planes owned
    const int dir = a.dir, kf = dir > 0 ? Z0 : Z0 + n - 1;  // the first of them
    const int sy = 4 * a.nq, sz = sy * a.ny;              // vectors below 2^31 cells (plan check)
    // this thread's quad and rows
    const bool live = tid < cq * rp;
    const int q = live ? tid % cq : 0, m = live ? tid / cq : 0;
    const int gq = Q0 + q, j0 = Y0 + NR * m;
    const bool inx = live && gq < a.nq;
    bool in[NR], own[NR];
#pragma unroll
    for (int h = 0; h < NR; ++h) {
        in[h] = inx && j0 + h < a.ny;
        own[h] = in[h] && q < a.wq && NR * m + h < a.rows;
    }
    const bool has_l = gq > 0, has_r = gq + 1 < a.nq;
    const int pad = a.nx - 4 * gq;                        // cells of the quad inside the grid (>= 4: all)
    const int g0 = 4 * gq + sy * j0;                      // first row, without the plane
    const int sb = (NR * m + 1) * BW + q + (a.frame ? 1 : 0);  // first row in a box of u or v
    const int so = NR * m * cq + q;                        // and in one of t, p or x

    if (tid == 0) {
        abort_flag = 0;
        for (int s = 0; s <= STAGES; ++s) nn_mbar_init(&bars[s], 1);
        nn_mbar_fence_init();
    }
    __syncthreads();
    // launched as a programmatic dependent of the previous iteration (in a
    // synchronous solve): its scalars, flags and vectors are complete only now
    nn_grid_dep_wait();
    if (!INIT && a.flags[0]) return;

    const bool has_t = INIT || a.it > 0, has_p = a.it > 1;
    auto heavy = [&](int c) { return !INIT && ((kf + dir * c + a.it) & 1); };  // p and x of the plane's turn
    const int box_bytes = BW * (NR * rp + 2) * 16, own_bytes = cq * NR * rp * 16;
    const int bx = 4 * Q0 - (a.frame ? 4 : 0);
    auto slot_u = [&](int c) { return reinterpret_cast<float4*>(smem + ((c + 2) & (STAGES - 1)) * L.box); };
    auto slot_v = [&](int c) { return reinterpret_cast<float4*>(smem + (STAGES + ((c + 2) & (STAGES - 1))) * L.box); };
    auto slot_t = [&](int c) { return reinterpret_cast<float4*>(smem + L.ey - (5 - (c + 3) % 3) * L.own); };
    float4* const slot_p = reinterpret_cast<float4*>(smem + L.ey - 2 * L.own);
    float4* const slot_x = reinterpret_cast<float4*>(smem + L.ey - L.own);
    // by one thread: plane c of u and v (v has a ghost row and plane on every side) and of t
    auto load_uv = [&](int c, uint64_t* bar) {
        nn_tma_load_3d(slot_u(c), &tm_u, bx, Y0 - 1, kf + dir * c, bar);
        if (HET) nn_tma_load_3d(slot_v(c), &tm_v, bx, Y0, kf + dir * c + 1, bar);
    };
    auto load_t = [&](int c, uint64_t* bar) { nn_tma_load_3d(slot_t(c), &tm_t, 4 * Q0, Y0, kf + dir * c, bar); };
    // step c waits for barrier (c + 1) % 4: u and v of plane c + 1, t of plane c;
    // the last barrier is p's and x's
    auto issue = [&](int c) {  // at step c - 2
        if (c >= n) return;
        uint64_t* bar = &bars[(c + 1) & (STAGES - 1)];
        nn_mbar_expect_tx(bar, (HET ? 2 : 1) * box_bytes + (has_t ? own_bytes : 0));
        load_uv(c + 1, bar);
        if (has_t) load_t(c, bar);
    };
    if (tid == 0) {
        nn_mbar_expect_tx(&bars[0], 3 * (HET ? 2 : 1) * box_bytes + (has_t ? own_bytes : 0));
        load_uv(-2, &bars[0]);
        load_uv(-1, &bars[0]);
        load_uv(0, &bars[0]);
        if (has_t) load_t(-1, &bars[0]);
        issue(0);
    }
    const float alpha = INIT ? 0.0f : (float)a.scal[C_ALPHA], beta = INIT ? 0.0f : (float)a.scal[C_BETA];
    const float alpha_p = INIT ? 0.0f : (float)a.scal[C_ALPHA_P], beta_p = INIT ? 0.0f : (float)a.scal[C_BETA_P];
    const float ax = HET ? alpha : alpha * a.inv_c, axp = HET ? alpha_p : alpha_p * a.inv_c;  // of x
    const Quad onepb = quad_all(a.onepb);

    // registers carried along the march: u and v here; the faces and fluxes to
    // the plane behind (constant coefficients: u there); the new u there
    Quad uC[NR], vC[NR], fzP[NR], zP[NR], wP[NR];
    if (tid == 0 && !nn_mbar_wait(&bars[0], 0, WAIT_LIMIT)) {
        nn_mbar_wait(&bars[0], 0, WAIT_LIMIT);  // let the copies in flight land
        nn_mbar_wait(&bars[1], 0, WAIT_LIMIT);
        abort_flag = 1;
    }
    __syncthreads();
    if (!abort_flag)
#pragma unroll
        for (int h = 0; h < NR; ++h) {
            uC[h] = quad_of(slot_u(-1)[sb + h * BW]);
            zP[h] = quad_of(slot_u(-2)[sb + h * BW]);
            if (HET) {
                vC[h] = quad_of(slot_v(-1)[sb + h * BW]);
                fzP[h] = rcp(quad_of(slot_v(-2)[sb + h * BW]) + vC[h]);
                zP[h] = fzP[h] * (uC[h] - zP[h]);
            }
            wP[h] = quad_zero();
        }
    CgSum sg, sd, sr, sbb;
    float e_g = 0.0f, e_d = 0.0f, e_r = 0.0f, e_b = 0.0f;  // of four planes
    // faces and new u of the last plane, for the energies across threads
    float xf[NR] = {}, xu[NR] = {};
    Quad yf = quad_zero(), yu = quad_zero();
    auto across = [&](int c) -> float {  // those energies of plane c
        const int b = c & 1;
        float e = 0.0f;
#pragma unroll
        for (int h = 0; h < NR; ++h) {
            const float o = own[h] && has_r ? ex[((b * rp + m) * NR + h) * cq + q + 1] : 0.0f;
            e += own[h] ? xf[h] * (o - xu[h]) * (o - xu[h]) : 0.0f;
        }
        if (own[NR - 1]) {
            const Quad d = (m + 1 < rp ? quad_of(ey[(b * rp + m + 1) * cq + q]) : quad_zero()) - yu;
            e += sum(yf * d * d);
        }
        return e;
    };

    for (int c = -1; c < n; ++c) {
        // one thread polls (spinning threads would take issue slots from the
        // working warps); the block barrier publishes the landed planes, and
        // everyone is done with the slots of plane c - 1
        if (tid == 0 && !abort_flag) {
            bool ok = nn_mbar_wait(&bars[(c + 1) & (STAGES - 1)], ((c + 1) / STAGES) & 1, WAIT_LIMIT);
            if (ok && c >= 0 && heavy(c)) ok = nn_mbar_wait(&bars[STAGES], (c >> 1) & 1, WAIT_LIMIT);
            if (!ok) {
                // let the copies still in flight land before the block leaves
                nn_mbar_wait(&bars[(c + 1) & (STAGES - 1)], ((c + 1) / STAGES) & 1, WAIT_LIMIT);
                if (c >= 0 && heavy(c)) nn_mbar_wait(&bars[STAGES], (c >> 1) & 1, WAIT_LIMIT);
                if (c + 1 < n) nn_mbar_wait(&bars[(c + 2) & (STAGES - 1)], ((c + 2) / STAGES) & 1, WAIT_LIMIT);
                abort_flag = 1;
            }
        }
        __syncthreads();
        if (abort_flag) break;
        if (tid == 0) {
            issue(c + 2);
            if (c + 1 < n && heavy(c + 1)) {
                nn_mbar_expect_tx(&bars[STAGES], (has_p ? 2 : 1) * own_bytes);
                if (has_p) nn_tma_load_3d(slot_p, &tm_p, 4 * Q0, Y0, kf + dir * (c + 1), &bars[STAGES]);
                nn_tma_load_3d(slot_x, &tm_x, 4 * Q0, Y0, kf + dir * (c + 1), &bars[STAGES]);
            }
        }
        const int k = kf + dir * c, g = k * sz + g0;
        const bool ink = k >= 0 && k < a.nz, ownk = c >= 0;
        if (live) {
            const float4 *U = slot_u(c) + sb, *V = slot_v(c) + sb, *UN = slot_u(c + 1) + sb, *VN = slot_v(c + 1) + sb;
            Quad tC[NR];
#pragma unroll
            for (int h = 0; h < NR; ++h) tC[h] = has_t ? quad_of(slot_t(c)[so + h * cq]) : quad_zero();
            if (ownk && heavy(c))
#pragma unroll
                for (int h = 0; h < NR; ++h) {
                    if (!own[h]) continue;
                    // p_{i-1} of u_{i-1}, then p_i
                    Quad po = fma(quad_all(alpha_p), tC[h], uC[h]);
                    if (has_p) po = fma(quad_all(beta_p), quad_of(slot_p[so + h * cq]), po);
                    const Quad pn = fma(quad_all(beta), po, uC[h]);
                    const Quad xn = fma(quad_all(ax), pn, fma(quad_all(axp), po, quad_of(slot_x[so + h * cq])));
                    *reinterpret_cast<float4*>(a.p + g + h * sy) = float4_of(pn);
                    *reinterpret_cast<float4*>(a.x + g + h * sy) = float4_of(xn);
                }
            if (c >= 1) e_d += across(c - 1);
            const Quad uB = quad_of(U[-BW]), uA = quad_of(U[NR * BW]);
            Quad fy[NR + 1], gy[NR + 1];  // faces and fluxes below, between and above the rows
            if (HET) {
                fy[0] = rcp(quad_of(V[-BW]) + vC[0]);
                gy[0] = fy[0] * (uC[0] - uB);
#pragma unroll
                for (int h = 1; h < NR; ++h) {
                    fy[h] = rcp(vC[h - 1] + vC[h]);
                    gy[h] = fy[h] * (uC[h] - uC[h - 1]);
                }
                fy[NR] = rcp(vC[NR - 1] + quad_of(V[NR * BW]));
                gy[NR] = fy[NR] * (uA - uC[NR - 1]);
            }
            Quad uN[NR], vN[NR], wN[NR];
#pragma unroll
            for (int h = 0; h < NR; ++h) {
                const Quad u = uC[h];
                uN[h] = quad_of(UN[h * BW]);
                const float uL = has_l ? U[h * BW - 1].w : 0.0f, uR = has_r ? U[h * BW + 1].x : 0.0f;
                float fx[5];
                Quad fzN, gzN, w, dg, mi;
                if (HET) {
                    const Quad& v = vC[h];
                    const float vL = has_l ? V[h * BW - 1].w : at(v, 0), vR = has_r ? V[h * BW + 1].x : at(v, 3);
                    vN[h] = quad_of(VN[h * BW]);
                    fx[0] = nn_rcp(vL + at(v, 0));
                    fx[1] = nn_rcp(at(v, 0) + at(v, 1));
                    fx[2] = nn_rcp(at(v, 1) + at(v, 2));
                    fx[3] = nn_rcp(at(v, 2) + at(v, 3));
                    fx[4] = nn_rcp(at(v, 3) + vR);
                    fzN = rcp(v + vN[h]);
                    gzN = fzN * (uN[h] - u);
                    const float x0 = fx[0] * (at(u, 0) - uL), x1 = fx[1] * (at(u, 1) - at(u, 0));
                    const float x2 = fx[2] * (at(u, 2) - at(u, 1)), x3 = fx[3] * (at(u, 3) - at(u, 2));
                    const float x4 = fx[4] * (uR - at(u, 3));
                    const Quad gx = {{{x0 - x1, x1 - x2}}, {{x2 - x3, x3 - x4}}};
                    w = fma(onepb, u, (gx + (gy[h] - gy[h + 1])) + (zP[h] - gzN));
                    const Quad sx = {{{fx[0] + fx[1], fx[1] + fx[2]}}, {{fx[2] + fx[3], fx[3] + fx[4]}}};
                    dg = onepb + ((sx + (fy[h] + fy[h + 1])) + (fzP[h] + fzN));
                    mi = rcp(dg);
                } else {
                    const Quad sx = {{{uL + at(u, 1), at(u, 0) + at(u, 2)}}, {{at(u, 1) + at(u, 3), at(u, 2) + uR}}};
                    const Quad nb = (sx + ((h > 0 ? uC[h > 0 ? h - 1 : 0] : uB) + (h < NR - 1 ? uC[h < NR - 1 ? h + 1 : 0] : uA))) + (zP[h] + uN[h]);
                    w = fma(onepb, u, quad_all(a.op_alpha) * (quad_all(6.0f) * u - nb));
                    mi = quad_all(a.invd);
                }
                Quad rv, tv;
                if (INIT) {
                    rv = tC[h] - w;
                    if (!(in[h] && ink)) rv = quad_zero();
                    if (pad < 4)
#pragma unroll
                        for (int e = 1; e < 4; ++e)
                            if (e >= pad) at(rv, e) = 0.0f;
                    wN[h] = (HET ? mi : quad_all(a.c * a.invd)) * rv;
                } else {
                    tv = fma(quad_all(beta), tC[h], mi * w);
                    if (pad < 4)
#pragma unroll
                        for (int e = 1; e < 4; ++e)
                            if (e >= pad) at(tv, e) = 0.0f;
                    // (u is zero outside the grid and stays so)
                    wN[h] = fma(quad_all(in[h] && ink ? -alpha : 0.0f), tv, u);
                    rv = HET ? dg * wN[h] : wN[h];  // constant coefficients: scaled at the end
                }
                const Quad& nu = wN[h];
                if (own[h] && ownk) {
                    *reinterpret_cast<float4*>(a.u_out + g + h * sy) = float4_of(nu);
                    if (!INIT) *reinterpret_cast<float4*>(a.t_out + g + h * sy) = float4_of(tv);
                    // the mass term and the energies of the faces inside the
                    // quad, to the plane behind and on the grid's near sides
                    const Quad uu = nu * nu, dz = nu - wP[h];
                    e_g += sum(HET ? rv * nu : uu);
                    e_r += sum(HET ? rv * rv : uu);
                    if (INIT) e_b += sum(tC[h] * tC[h]);
                    Quad s = HET ? fma(onepb, uu, fzP[h] * dz * dz) : dz * dz;
                    if (k == (dir > 0 ? a.nz - 1 : 0)) s = HET ? fma(fzN, uu, s) : s + uu;
                    if (h == 0 && j0 == 0) s = HET ? fma(fy[0], uu, s) : s + uu;
                    float x = 0.0f;
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        const float dx = at(nu, e + 1) - at(nu, e);
                        x += (HET ? fx[e + 1] : 1.0f) * dx * dx;
                    }
                    if (!has_l) x += (HET ? fx[0] : 1.0f) * at(uu, 0);
                    x += sum(s);
                    e_d += HET ? x : a.op_alpha * x + a.onepb * sum(uu);
                }
                xf[h] = HET ? fx[4] : a.op_alpha;
                xu[h] = at(nu, 3);
                ex[(((c & 1) * rp + m) * NR + h) * cq + q] = at(nu, 0);
                wP[h] = nu;
                zP[h] = HET ? gzN : u;
                if (HET) fzP[h] = fzN;
            }
            ey[((c & 1) * rp + m) * cq + q] = float4_of(wN[0]);
#pragma unroll
            for (int h = 1; h < NR; ++h) {
                if (!(own[h - 1] && ownk)) continue;
                const Quad dy = wN[h] - wN[h - 1];
                const float y = sum(HET ? fy[h] * dy * dy : dy * dy);
                e_d += HET ? y : a.op_alpha * y;
            }
            yf = HET ? fy[NR] : quad_all(a.op_alpha);
            yu = wN[NR - 1];
#pragma unroll
            for (int h = 0; h < NR; ++h) {
                uC[h] = uN[h];
                if (HET) vC[h] = vN[h];
            }
        }
        if ((c & 3) == 3 || c == n - 1) {
            sd.add(e_d);
            sg.add(e_g);
            sr.add(e_r);
            if (INIT) sbb.add(e_b);
            e_d = e_g = e_r = e_b = 0.0f;
        }
    }
    __syncthreads();
    if (abort_flag) {
        if (tid == 0) {
            a.flags[2] = 1;
            a.flags[0] = 3;
        }
        return;
    }
    if (live) sd.add(across(n - 1));
    const double scale = HET ? 1.0 : (double)a.onepb + 6.0 * (double)a.op_alpha;  // r = scale u
    const double sums[4] = {scale * sg.value(), sd.value(), scale * scale * sr.value(), sbb.value()};
    double out[4];
    if (cg_reduce<INIT ? 4 : 3>(sums, a.partials, a.ticket, out) && tid == 0) cg_scalars(a, INIT, out);
}

// x (rows of nx) from xp (rows of 4 nq, possibly x itself) after a.it
// iterations: adds the last one's direction in the planes whose turn it was not.
__global__ void __launch_bounds__(CG_THREADS) k_cg_flush(const __grid_constant__ CgArgs a, const float* u, const float* t,
                                                         float* x)
{
    const float al = (float)a.scal[C_ALPHA_P], be = (float)a.scal[C_BETA_P], ax = al * a.inv_c;
    const bool same = x == a.x;  // then only those planes are touched
    const int first = same ? (a.it + 1) & 1 : 0, step = same ? 2 : 1;
    const int planes = (a.nz - first + step - 1) / step, psz = a.nx * a.ny;
    for (int64_t i = blockIdx.x * (int64_t)CG_THREADS + threadIdx.x; i < (int64_t)planes * psz;
         i += (int64_t)gridDim.x * CG_THREADS) {
        const int k = first + step * (int)(i / psz), row = (int)(i % psz) / a.nx + k * a.ny, e = (int)(i % psz) % a.nx;
        const int c = row * 4 * a.nq + e;
        float v = a.x[c];
        if (a.it > 0 && ((k + a.it) & 1)) v += ax * (u[c] + al * t[c] + (a.it > 1 ? be * a.p[c] : 0.0f));
        x[(int64_t)row * a.nx + e] = v;
    }
}

// src (rows of nx) as rows of 4 nq cells, zeros behind the row.
__global__ void __launch_bounds__(CG_THREADS) k_cg_pad(int nx, int nq, int rows, const float* src, float* dst)
{
    const int64_t G = (int64_t)4 * nq * rows;
    for (int64_t i = blockIdx.x * (int64_t)CG_THREADS + threadIdx.x; i < G; i += (int64_t)gridDim.x * CG_THREADS) {
        const int row = (int)(i / (4 * nq)), c = (int)(i - (int64_t)row * 4 * nq);
        dst[i] = c < nx ? src[(int64_t)row * nx + c] : 0.0f;
    }
}

// v = 1 / (2 alpha D) with a ghost row and plane on every side and behind the
// row, where it is that of the nearest cell.  Two neighbours with D = 0 have the
// face coefficient 0 / 0, an infinite D inf / inf: their v is NaN.
__global__ void __launch_bounds__(CG_THREADS) k_cg_field(int nx, int ny, int nz, int nq, const float* D, float half_ia,
                                                         float* v)
{
    const int64_t G = (int64_t)4 * nq * (ny + 2) * (nz + 2), sz = (int64_t)nx * ny;
    for (int64_t i = blockIdx.x * (int64_t)CG_THREADS + threadIdx.x; i < G; i += (int64_t)gridDim.x * CG_THREADS) {
        const int row = (int)(i / (4 * nq)), x = min((int)(i - (int64_t)row * 4 * nq), nx - 1);
        const int j = min(max(row % (ny + 2) - 1, 0), ny - 1), k = min(max(row / (ny + 2) - 1, 0), nz - 1);
        const int64_t c = x + (int64_t)nx * j + sz * k;
        const float d = D[c];
        float o = __fdiv_rn(half_ia, d);
        if (d == 0.0f &&
            ((x > 0 && D[c - 1] == 0.0f) || (x < nx - 1 && D[c + 1] == 0.0f) || (j > 0 && D[c - nx] == 0.0f) ||
             (j < ny - 1 && D[c + nx] == 0.0f) || (k > 0 && D[c - sz] == 0.0f) || (k < nz - 1 && D[c + sz] == 0.0f)))
            o = nanf("");
        if (isinf(d)) o = nanf("");
        v[i] = o;
    }
}
PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
        else
            cudaGetLastError();
    }
    return fn;
}

// Boxes of bx quads and by rows of one plane.
bool make_map(CUtensorMap* m, const float* base, int nq, int ny, int nz, int bx, int by)
{
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t gdim[3] = {(cuuint64_t)nq * 4, (cuuint64_t)ny, (cuuint64_t)nz};
    cuuint64_t gstride[2] = {(cuuint64_t)nq * 16, (cuuint64_t)nq * ny * 16};
    cuuint32_t box[3] = {(cuuint32_t)bx * 4, (cuuint32_t)by, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), gdim, gstride, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

// --------------------------------------------------------------- host side --

struct nn_cg_plan {
    nn_ctx* ctx = nullptr;
    int nx = 0, ny = 0, nz = 0, nq = 0;
    size_t cells = 0;              // of a padded vector
    float op_alpha = 0, onepb = 0, invd = 0, half_ia = 0, c = 1;
    const float* D = nullptr;      // caller's cell field (HET), not owned
    float *u[2] = {}, *t[2] = {}, *p = nullptr, *v = nullptr;
    float* xp = nullptr;           // x in rows of whole quads where the caller's is not
    CUtensorMap map_u[2], map_t[2], map_p, map_v, map_xp;
    double* scal = nullptr;
    double* partials = nullptr;
    unsigned int* ticket = nullptr;
    int* flags = nullptr;
    int wq = 0, cq = 0, rows = 0, rp = 0, ntx = 0, nty = 0, zc = 16;  // tiles (CgArgs)
    int threads = 0, elem_blocks = 0;
    size_t smem = 0;
    // timing of the iteration kernels
    bool timing = false;
    std::vector<cudaEvent_t> ev_a, ev_b;
    float last_ms = 0.0f;
    int last_iters = 0;
    // asynchronous solve in progress (nn_cg_async_*)
    struct {
        bool active = false;
        float* x = nullptr;
        CUtensorMap map_x;
        double rtol = 0.0;
        int max_iter = 0;
        int enqueued = 0;
        cudaStream_t cs = nullptr;
        cudaEvent_t e0 = nullptr, e1 = nullptr;
    } as;
    int tiles(int depth) const { return ntx * nty * ((nz + depth - 1) / depth); }
};

static void cg_free(nn_cg_plan* pl)
{
    for (int q = 0; q < 2; ++q) {
        nn_release(pl->u[q]);
        nn_release(pl->t[q]);
    }
    nn_release(pl->p);
    nn_release(pl->v);
    nn_release(pl->xp);
    nn_release(pl->scal);
    nn_release(pl->partials);
    nn_release(pl->ticket);
    nn_release(pl->flags);
}

void nn_cg_plan_destroy(nn_cg_plan* pl)
{
    if (!pl) return;
    if (pl->ctx) cudaStreamSynchronize(pl->ctx->stream);
    cg_free(pl);
    for (auto e : pl->ev_a) cudaEventDestroy(e);
    for (auto e : pl->ev_b) cudaEventDestroy(e);
    if (pl->as.e0) cudaEventDestroy(pl->as.e0);
    if (pl->as.e1) cudaEventDestroy(pl->as.e1);
    nn_ctx* ctx = pl->ctx;
    delete pl;
    nn_ctx_release(ctx);
}

static int box_quads(const nn_cg_plan* pl) { return pl->cq + (pl->ntx > 1 ? 2 : 0); }

static bool cg_maps(nn_cg_plan* pl)
{
    const int nq = pl->nq, ny = pl->ny, nz = pl->nz, bq = box_quads(pl), br = NR * pl->rp + 2;
    for (int q = 0; q < 2; ++q)
        if (!make_map(&pl->map_u[q], pl->u[q], nq, ny, nz, bq, br) ||
            !make_map(&pl->map_t[q], pl->t[q], nq, ny, nz, pl->cq, NR * pl->rp))
            return false;
    return make_map(&pl->map_p, pl->p, nq, ny, nz, pl->cq, NR * pl->rp) &&
           (!pl->D || make_map(&pl->map_v, pl->v, nq, ny + 2, nz + 2, bq, br)) &&
           (!pl->xp || make_map(&pl->map_xp, pl->xp, nq, ny, nz, pl->cq, NR * pl->rp));
}

// The plan's vectors, scalars and tensor maps, made once.
static nn_status cg_vectors(nn_cg_plan* pl)
{
    if (pl->flags) return NN_OK;
    nn_ctx* ctx = pl->ctx;
    nn_status st = NN_OK;
    for (int q = 0; q < 2 && st == NN_OK; ++q) {
        st = nn_alloc(ctx, &pl->u[q], pl->cells);
        if (st == NN_OK) st = nn_alloc(ctx, &pl->t[q], pl->cells);
    }
    if (st == NN_OK) st = nn_alloc(ctx, &pl->p, pl->cells);
    if (st == NN_OK && pl->D) st = nn_alloc(ctx, &pl->v, (size_t)4 * pl->nq * (pl->ny + 2) * (pl->nz + 2));
    if (st == NN_OK && (pl->nx % 4 || ((uintptr_t)pl->D & 15))) st = nn_alloc(ctx, &pl->xp, pl->cells);
    if (st == NN_OK) st = nn_alloc(ctx, &pl->scal, C_COUNT);
    if (st == NN_OK) st = nn_alloc(ctx, &pl->partials, (size_t)4 * pl->tiles(1));
    if (st == NN_OK) st = nn_alloc(ctx, &pl->ticket, 1);
    if (st == NN_OK) st = nn_alloc(ctx, &pl->flags, 4);
    if (st == NN_OK && !cg_maps(pl)) st = NN_ERR_UNSUPPORTED;
    if (st == NN_OK) st = nn_cuda_check(ctx, cudaMemsetAsync(pl->ticket, 0, sizeof(unsigned int), ctx->stream), "memset");
    if (st != NN_OK) cg_free(pl);
    return st;
}

// Tiles of the plan: whole rows where they fit, then the number of rows and
// planes with the least work of the busiest SM (one block each), where a block
// computes zc + 1 planes, loads two more, and a plane costs its quads and a
// barrier (the load of about 64 quads).
// Two kinds of grid march too shortly, or too few quads a plane, for one block to
// hide its copies' latency, and share an SM between blocks instead:
// - up to eight planes: tiles of at most 256 threads (192 with a cell field),
//   two or three to an SM by their registers.  us an iteration, the larger tile
//   and this one: 1024 x 1024 x 8 78 and 66 (88 and 81 with a cell field), 2048 x
//   2048 x 2 61 and 48;
// - a plane that is one tile of at most 128 threads: chunks of 6 to 12 planes, as
//   many as four blocks an SM take (their number counts in the reduction, so at
//   most sixteen).  us, 152 chunks and these: 4 x 4 x 4096 20 and 11, 12 x 12 x
//   20000 141 and 36, 32 x 32 x 4000 39 and 28.
static bool cg_shape(nn_cg_plan* pl, int sms, size_t smem_max)
{
    const int ny = pl->ny, nz = pl->nz;
    // (of a box row of 64 quads the frame takes two, the column computed twice one)
    pl->ntx = pl->nq <= CG_MAX_QUADS ? 1 : (pl->nq + CG_MAX_QUADS - 4) / (CG_MAX_QUADS - 3);
    pl->wq = (pl->nq + pl->ntx - 1) / pl->ntx;
    pl->ntx = (pl->nq + pl->wq - 1) / pl->wq;
    const int cq = pl->cq = pl->wq + (pl->ntx > 1);
    double best = -1.0;
    for (int rows = 1; rows <= ny && rows <= NR * CG_MAX_THREADS; ++rows) {
        const int nty = (ny + rows - 1) / rows, rp = (rows + (nty > 1) + NR - 1) / NR;
        if (rows > 1 && (ny + rows - 2) / (rows - 1) == nty) continue;  // no fewer tiles than with a row less
        const int threads = (cq * rp + 31) / 32 * 32;
        const size_t smem = CgSmem(cq, rp, pl->ntx > 1, pl->D != nullptr).total;
        if (threads > CG_MAX_THREADS || smem > smem_max || NR * rp > 200) break;  // (box rows: at most 256)
        if (nz <= 8 && best >= 0.0 && threads > (pl->D ? 192 : 256)) break;
        for (int waves = 1; waves <= 4; ++waves) {
            const int64_t cols = (int64_t)pl->ntx * nty;
            int64_t chunks = std::min<int64_t>(nz, std::max<int64_t>(1, (int64_t)waves * sms / cols));
            const int zc = (int)((nz + chunks - 1) / chunks);
            chunks = (nz + zc - 1) / zc;
            const double cost = (double)((cols * chunks + sms - 1) / sms) * (zc + 3) * ((double)NR * cq * rp + 64.0);
            if (best >= 0.0 && cost >= best) continue;
            best = cost;
            pl->rows = rows;
            pl->rp = rp;
            pl->nty = nty;
            pl->zc = zc;
            pl->threads = threads;
            pl->smem = smem;
        }
    }
    if (pl->ntx * pl->nty == 1 && pl->threads <= 128)
        pl->zc = std::max(std::min(std::max(6, (nz + 4 * sms - 1) / (4 * sms)), 12), (nz + 16 * sms - 1) / (16 * sms));
    return best >= 0.0;
}

// Grids whose padded vectors have at most 2^31 - 1 cells; otherwise UNSUPPORTED
// and the caller keeps the two-kernel PCG.  D (null for constant coefficients)
// stays owned by the caller.  lazy: the vectors are allocated at the first use.
nn_status nn_cg_plan_create(nn_ctx* ctx, int nx, int ny, int nz, double alpha, double beta, const float* D, bool lazy,
                            nn_cg_plan** out)
{
    *out = nullptr;
    const int nq = (int)(((int64_t)nx + 3) / 4);
    if (nx < 1 || ny < 1 || nz < 1 || (double)4 * nq * ny * nz > (double)INT32_MAX || !encode_fn())
        return NN_ERR_UNSUPPORTED;
    int smem_max = 0;
    NN_CUDA(ctx, cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
    nn_cg_plan* pl = new nn_cg_plan();
    pl->ctx = ctx;
    nn_ctx_retain(ctx);
    pl->nx = nx; pl->ny = ny; pl->nz = nz; pl->nq = nq;
    pl->cells = (size_t)4 * nq * ny * nz;
    pl->op_alpha = (float)alpha;
    pl->onepb = (float)(1.0 + beta);
    pl->invd = (float)(1.0 / (1.0 + beta + 6.0 * alpha));
    pl->half_ia = 0.5f / pl->op_alpha;
    pl->c = nn_jacobi_scale(alpha, beta, D != nullptr);
    pl->D = D;
    pl->elem_blocks = nn_grid_for(ctx, (int64_t)pl->cells, CG_THREADS, 8);
    // (the reduction's static shared memory is beside the tile's)
    nn_status st = cg_shape(pl, ctx->num_sms, (size_t)smem_max - 1024) ? NN_OK : NN_ERR_UNSUPPORTED;
    if (st == NN_OK && !lazy) st = cg_vectors(pl);
    for (auto* f : {&k_cg_iter<false, false>, &k_cg_iter<false, true>, &k_cg_iter<true, false>, &k_cg_iter<true, true>})
        if (st == NN_OK)
            st = nn_cuda_check(ctx, cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max - 1024),
                               "cudaFuncSetAttribute(k_cg_iter)");
    if (st != NN_OK) {
        nn_cg_plan_destroy(pl);
        return st;
    }
    *out = pl;
    return NN_OK;
}

void nn_cg_set_timing(nn_cg_plan* pl, bool on) { pl->timing = on; }
void nn_cg_last_timing(const nn_cg_plan* pl, float* ms, int* iters)
{
    *ms = pl->last_ms;
    *iters = pl->last_iters;
}

// Arguments of iteration it (-1: the initial residual).
static CgArgs cg_args(nn_cg_plan* pl, float* x, double rtol, int max_iter, int it)
{
    CgArgs a;
    const int pin = it & 1;
    a.nx = pl->nx; a.ny = pl->ny; a.nz = pl->nz; a.nq = pl->nq;
    a.wq = pl->wq; a.cq = pl->cq; a.rows = pl->rows; a.rp = pl->rp;
    a.ntx = pl->ntx; a.nty = pl->nty; a.zc = pl->zc;
    a.op_alpha = pl->op_alpha; a.onepb = pl->onepb; a.invd = pl->invd;
    a.c = pl->c; a.inv_c = 1.0f / pl->c;
    a.frame = pl->ntx > 1;
    a.u_out = pl->u[pin ^ 1];
    a.t_out = pl->t[pin ^ 1];
    a.p = pl->p;
    a.x = pl->xp ? pl->xp : x;
    a.it = it;
    a.dir = it & 1 ? -1 : 1;
    a.scal = pl->scal;
    a.partials = pl->partials;
    a.ticket = pl->ticket;
    a.flags = pl->flags;
    a.rtol2 = rtol * rtol;
    a.max_iter = max_iter;
    return a;
}

// the field, r0, u0 and the first scalars on stream cs
static nn_status enqueue_init(nn_cg_plan* pl, const float* d_b, float* d_x, double rtol, int max_iter, cudaStream_t cs)
{
    nn_ctx* ctx = pl->ctx;
    NN_CUDA(ctx, cudaMemsetAsync(pl->ticket, 0, sizeof(unsigned int), cs));  // clean after an aborted solve
    if (pl->D) {
        k_cg_field<<<pl->elem_blocks, CG_THREADS, 0, cs>>>(pl->nx, pl->ny, pl->nz, pl->nq, pl->D, pl->half_ia, pl->v);
        NN_CHECK_LAUNCH(ctx, "k_cg_field");
    }
    const CgArgs a = cg_args(pl, d_x, rtol, max_iter, -1);  // writes u[0]
    const int nq = pl->nq, ny = pl->ny, nz = pl->nz;
    if (pl->xp) {
        k_cg_pad<<<pl->elem_blocks, CG_THREADS, 0, cs>>>(pl->nx, nq, ny * nz, d_x, pl->xp);
        NN_CHECK_LAUNCH(ctx, "k_cg_pad");
    }
    CUtensorMap map_u, map_t = pl->map_t[1];  // x with the frame, b
    bool ok = make_map(&map_u, a.x, nq, ny, nz, box_quads(pl), NR * pl->rp + 2);
    if (pl->xp || ((uintptr_t)d_b & 15)) {
        k_cg_pad<<<pl->elem_blocks, CG_THREADS, 0, cs>>>(pl->nx, nq, ny * nz, d_b, pl->t[1]);
        NN_CHECK_LAUNCH(ctx, "k_cg_pad");
    } else {
        ok = ok && make_map(&map_t, d_b, nq, ny, nz, pl->cq, NR * pl->rp);
    }
    if (!ok) return nn_fail(ctx, NN_ERR_UNSUPPORTED, "nn_cg: tensor map of x or b");
    if (pl->D)
        k_cg_iter<true, true><<<pl->tiles(pl->zc), pl->threads, pl->smem, cs>>>(map_u, pl->map_v, map_t, map_t, map_t, a);
    else
        k_cg_iter<false, true><<<pl->tiles(pl->zc), pl->threads, pl->smem, cs>>>(map_u, map_u, map_t, map_t, map_t, a);
    NN_CHECK_LAUNCH(ctx, "k_cg_iter");
    return NN_OK;
}

// x as the iterations read it
static nn_status x_map(nn_cg_plan* pl, float* d_x, CUtensorMap* m)
{
    if (pl->xp) *m = pl->map_xp;
    else if (((uintptr_t)d_x & 15) || !make_map(m, d_x, pl->nq, pl->ny, pl->nz, pl->cq, NR * pl->rp))
        return nn_fail(pl->ctx, NN_ERR_INVALID_ARG, "PCG: x must be a 16-byte aligned device vector");
    return NN_OK;
}

// iterations it0 .. it0 + n - 1 (each a no-op once the device flag is set)
// pdl: each iteration a programmatic dependent of the kernel before it
// (synchronous solves; an overlapped solve's waiting blocks would hold SM
// room the neuron updates use)
static nn_status enqueue_iters(nn_cg_plan* pl, float* d_x, const CUtensorMap& map_x, double rtol, int max_iter, int it0,
                               int n, cudaStream_t cs, bool pdl = false)
{
    nn_ctx* ctx = pl->ctx;
    const CUtensorMap& map_v = pl->D ? pl->map_v : pl->map_p;
    for (int it = it0; it < it0 + n; ++it) {
        const CgArgs a = cg_args(pl, d_x, rtol, max_iter, it);
        auto* f = pl->D ? &k_cg_iter<true, false> : &k_cg_iter<false, false>;
        if (pdl) {
            NN_CUDA(ctx, nn_launch_pdl(f, dim3(pl->tiles(pl->zc)), dim3(pl->threads), pl->smem, cs,
                                       pl->map_u[it & 1], map_v, pl->map_t[it & 1], pl->map_p, map_x, a));
            ctx->launches++;
            continue;
        }
        f<<<pl->tiles(pl->zc), pl->threads, pl->smem, cs>>>(pl->map_u[it & 1], map_v, pl->map_t[it & 1], pl->map_p, map_x,
                                                            a);
        NN_CHECK_LAUNCH(ctx, "k_cg_iter");
    }
    return NN_OK;
}

// what x lacks after n finished iterations
static nn_status enqueue_flush(nn_cg_plan* pl, float* d_x, int n, cudaStream_t cs)
{
    if (n == 0) return NN_OK;
    const CgArgs a = cg_args(pl, d_x, 0.0, 0, n);  // reads what the last one wrote
    k_cg_flush<<<pl->elem_blocks, CG_THREADS, 0, cs>>>(a, pl->u[n & 1], pl->t[n & 1], d_x);
    NN_CHECK_LAUNCH(pl->ctx, "k_cg_flush");
    return NN_OK;
}

// Asynchronous solve on stream cs: the init and n iterations are enqueued
// with no host read; nn_cg_async_more adds iterations; nn_cg_async_finish
// waits for the stream, completes the solve if n was not enough and reports.
nn_status nn_cg_async_begin(nn_cg_plan* pl, const float* d_b, float* d_x, double rtol, int max_iter, int n,
                            cudaStream_t cs)
{
    nn_ctx* ctx = pl->ctx;
    NN_TRY(cg_vectors(pl));
    NN_TRY(x_map(pl, d_x, &pl->as.map_x));
    if (!pl->as.e0) NN_CUDA(ctx, cudaEventCreate(&pl->as.e0));
    if (!pl->as.e1) NN_CUDA(ctx, cudaEventCreate(&pl->as.e1));
    pl->as.active = true;
    pl->as.x = d_x;
    pl->as.rtol = rtol;
    pl->as.max_iter = max_iter;
    pl->as.cs = cs;
    pl->as.enqueued = 0;
    if (pl->timing) NN_CUDA(ctx, cudaEventRecord(pl->as.e0, cs));
    NN_TRY(enqueue_init(pl, d_b, d_x, rtol, max_iter, cs));
    return nn_cg_async_more(pl, n);
}

nn_status nn_cg_async_more(nn_cg_plan* pl, int n)
{
    if (!pl->as.active) return NN_ERR_INVALID_ARG;
    n = std::min(n, pl->as.max_iter - pl->as.enqueued);
    if (n <= 0) return NN_OK;
    NN_TRY(enqueue_iters(pl, pl->as.x, pl->as.map_x, pl->as.rtol, pl->as.max_iter, pl->as.enqueued, n, pl->as.cs));
    pl->as.enqueued += n;
    if (pl->timing) NN_CUDA(pl->ctx, cudaEventRecord(pl->as.e1, pl->as.cs));
    return NN_OK;
}

nn_status nn_cg_async_finish(nn_cg_plan* pl, int* iters, double* relres, int* converged)
{
    nn_ctx* ctx = pl->ctx;
    if (!pl->as.active) return NN_ERR_INVALID_ARG;
    cudaStream_t cs = pl->as.cs;
    int h_flags[4] = {0, 0, 0, 0};
    while (true) {
        NN_CUDA(ctx, cudaMemcpyAsync(h_flags, pl->flags, sizeof h_flags, cudaMemcpyDeviceToHost, cs));
        NN_CUDA(ctx, cudaStreamSynchronize(cs));
        if (h_flags[0] || pl->as.enqueued >= pl->as.max_iter) break;
        NN_TRY(nn_cg_async_more(pl, 16));
    }
    if (h_flags[2]) return nn_fail(ctx, NN_ERR_TIMEOUT, "k_cg_iter: a TMA pipeline wait timed out");
    NN_TRY(enqueue_flush(pl, pl->as.x, h_flags[1], cs));
    double h_scal[C_COUNT];
    NN_CUDA(ctx, cudaMemcpyAsync(h_scal, pl->scal, sizeof h_scal, cudaMemcpyDeviceToHost, cs));
    NN_CUDA(ctx, cudaStreamSynchronize(cs));
    pl->as.active = false;
    if (pl->timing) {
        float ms = 0.0f;
        NN_CUDA(ctx, cudaEventElapsedTime(&ms, pl->as.e0, pl->as.e1));
        pl->last_ms = ms;
        pl->last_iters = h_flags[1];
    }
    if (iters) *iters = h_flags[1];
    if (relres) *relres = h_scal[C_BB] > 0 ? std::sqrt(h_scal[C_RR] / h_scal[C_BB]) : 0.0;
    if (converged) *converged = h_flags[0] == 1;
    return NN_OK;
}

// Solve A x = b (x holds the initial guess).  Iterations are enqueued in
// chunks; the host reads the device flags once per chunk.
nn_status nn_cg_run(nn_cg_plan* pl, const float* d_b, float* d_x, double rtol, int max_iter, int* iters,
                    double* relres, int* converged)
{
    nn_ctx* ctx = pl->ctx;
    cudaStream_t cs = ctx->stream;
    NN_TRY(cg_vectors(pl));
    CUtensorMap map_x;
    NN_TRY(x_map(pl, d_x, &map_x));
    NN_TRY(enqueue_init(pl, d_b, d_x, rtol, max_iter, cs));
    int h_flags[4] = {0, 0, 0, 0};
    int it = 0, nchunks = 0;
    const int chunk = 16;
    while (true) {
        NN_CUDA(ctx, cudaMemcpyAsync(h_flags, pl->flags, sizeof h_flags, cudaMemcpyDeviceToHost, cs));
        NN_CUDA(ctx, cudaStreamSynchronize(cs));
        if (h_flags[0] || it >= max_iter) break;
        if (pl->timing) {
            if ((int)pl->ev_a.size() <= nchunks) {
                cudaEvent_t e1, e2;
                NN_CUDA(ctx, cudaEventCreate(&e1));
                NN_CUDA(ctx, cudaEventCreate(&e2));
                pl->ev_a.push_back(e1);
                pl->ev_b.push_back(e2);
            }
            NN_CUDA(ctx, cudaEventRecord(pl->ev_a[nchunks], cs));
        }
        const int n = std::min(chunk, max_iter - it);
        NN_TRY(enqueue_iters(pl, d_x, map_x, rtol, max_iter, it, n, cs, true));
        it += n;
        if (pl->timing) NN_CUDA(ctx, cudaEventRecord(pl->ev_b[nchunks], cs));
        ++nchunks;
    }
    if (h_flags[2]) return nn_fail(ctx, NN_ERR_TIMEOUT, "k_cg_iter: a TMA pipeline wait timed out");
    NN_TRY(enqueue_flush(pl, d_x, h_flags[1], cs));
    double h_scal[C_COUNT];
    NN_CUDA(ctx, cudaMemcpyAsync(h_scal, pl->scal, sizeof h_scal, cudaMemcpyDeviceToHost, cs));
    NN_CUDA(ctx, cudaStreamSynchronize(cs));
    if (pl->timing) {
        float tot = 0.0f;
        for (int c = 0; c < nchunks; ++c) {
            float ms = 0.0f;
            NN_CUDA(ctx, cudaEventElapsedTime(&ms, pl->ev_a[c], pl->ev_b[c]));
            tot += ms;
        }
        pl->last_ms = tot;
        pl->last_iters = h_flags[1];
    }
    if (iters) *iters = h_flags[1];
    if (relres) *relres = h_scal[C_BB] > 0 ? std::sqrt(h_scal[C_RR] / h_scal[C_BB]) : 0.0;
    if (converged) *converged = h_flags[0] == 1;
    return NN_OK;
}

// Tile-depth autotuner: time `iters` iterations (after two untimed ones) of
// every candidate depth on this plan's own operator -- right-hand side d_b,
// d_x as scratch (overwritten) -- and keep the fastest.  The residual target
// is never reached, so every timed iteration does its full work.
nn_status nn_cg_plan_autotune(nn_cg_plan* pl, const float* d_b, float* d_x, int iters, int* zc_out, float* ms_out)
{
    nn_ctx* ctx = pl->ctx;
    cudaStream_t cs = ctx->stream;
    if (iters < 1) return NN_ERR_INVALID_ARG;
    NN_TRY(cg_vectors(pl));
    CUtensorMap map_x;
    NN_TRY(x_map(pl, d_x, &map_x));
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    NN_CUDA(ctx, cudaEventCreate(&e0));
    NN_CUDA(ctx, cudaEventCreate(&e1));
    const int zc0 = pl->zc;
    int best_zc = zc0;
    float best = 1e30f;
    nn_status st = NN_OK;
    const double rtol = 1e-30;
    const int max_iter = 1 << 30;
    int prev_zc = 0;
    for (int zc : {4, 6, 8, 12, 16, 24, 32}) {
        if (st != NN_OK || prev_zc >= pl->nz) break;  // deeper tiles than the grid change nothing
        prev_zc = zc;
        pl->zc = zc;
        st = nn_cuda_check(ctx, cudaMemsetAsync(d_x, 0, sizeof(float) * (size_t)pl->nx * pl->ny * pl->nz, cs), "memset");
        if (st == NN_OK) st = enqueue_init(pl, d_b, d_x, rtol, max_iter, cs);
        if (st == NN_OK) st = enqueue_iters(pl, d_x, map_x, rtol, max_iter, 0, 2, cs);
        if (st == NN_OK) st = nn_cuda_check(ctx, cudaEventRecord(e0, cs), "event");
        if (st == NN_OK) st = enqueue_iters(pl, d_x, map_x, rtol, max_iter, 2, iters, cs);
        if (st == NN_OK) st = nn_cuda_check(ctx, cudaEventRecord(e1, cs), "event");
        int h_flags[4] = {0, 0, 0, 0};
        if (st == NN_OK)
            st = nn_cuda_check(ctx, cudaMemcpyAsync(h_flags, pl->flags, sizeof h_flags, cudaMemcpyDeviceToHost, cs),
                               "copy");
        if (st == NN_OK) st = nn_cuda_check(ctx, cudaStreamSynchronize(cs), "nn_cg_plan_autotune");
        float ms = 0.0f;
        if (st == NN_OK) st = nn_cuda_check(ctx, cudaEventElapsedTime(&ms, e0, e1), "event");
        if (st == NN_OK && h_flags[2]) st = nn_fail(ctx, NN_ERR_TIMEOUT, "k_cg_iter: a TMA pipeline wait timed out");
        // iterations that stopped early (exact solution, non-finite) are no timing
        if (st == NN_OK && h_flags[0] == 0 && ms / iters < best) {
            best = ms / iters;
            best_zc = zc;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    pl->zc = st == NN_OK ? best_zc : zc0;
    if (zc_out) *zc_out = pl->zc;
    if (ms_out) *ms_out = best < 1e30f ? best : 0.0f;
    return st;
}

int nn_cg_plan_tile_depth(const nn_cg_plan* pl) { return pl->zc; }

// Set the tile depth (4 .. 32).
void nn_cg_plan_set_tile_depth(nn_cg_plan* pl, int zc) { pl->zc = zc; }
