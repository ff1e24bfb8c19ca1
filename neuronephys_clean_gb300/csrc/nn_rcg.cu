// Resident preconditioned CG: the whole solve in one kernel, for grids whose
// vectors fit in the registers and shared memory of the GPU.
//
// Same operator and recurrences as nn_cg.cu (7-point backward Euler, Jacobi
// preconditioner, Chronopoulos and Gear's one-reduction form), written in the
// scaled residual u = M r, with w' = M A u and s' = M s:
//   s' = w' + b s'    p = u + b p    x += a p    u -= a s'    w' = M A u
//   g = (r, u) = (u, u/M),  d = (w, u) = (w'/M, u),  rho = (r, r)
// so that the preconditioner is needed only inside the stencil pass, where
// the diagonal is the sum of the face coefficients at hand.
//
// What bounds it.  A launch per iteration that moved ten vectors through L2 and
// paid a grid's start, tail and reduction took 22 us an iteration at 128^3 and
// 5 us at 32^3; two launches an iteration (nn_pcg.cu) 54 us at 97 x 83 x 150.
// Here nothing but the bricks' faces and the three sums leaves the SM: an
// iteration costs one exchange between the blocks (3 us) and the arithmetic on
// the block's own cells.  Measured per iteration: 3.2 us at 32^3, 4.2 at 64^3,
// 9.0 at 128^3 (solve to 1e-6: 2.13 ms -> 0.85), and with a cell field 4.5 at
// 48^3, 9.0 at 97 x 83 x 150 (9.8 ms -> 1.8).
//
// Precision.  The cells are FP32, and so are the sums within a warp; across
// warps and blocks the sums are FP64, as are the scalars and the convergence
// test.  The FP64 pipe's latencies (65 cycles an addition, 570 a division) lie
// between the exchange and the next update, 0.6 us an iteration more than sums
// and scalars in pairs of floats would take; divisions as such took 0.6 us more
// (8^3: 2.45 us in pairs, 3.65 with plain divisions, 3.0).
//
// Layout.  A block owns a brick of whole x rows, by x bz of them.  A thread
// owns one quad of four x cells in each of the brick's bz planes, so p and
// s' stay in registers (8 bz of them) and the z neighbours pass from plane to
// plane; u (and the cell field) lie in shared memory with a one-cell halo, w'
// in a private slot per thread.  x is read by nothing during the solve: it
// stays in L2 and takes two directions every second iteration, loaded while
// the block waits for the others (in registers it spilled).  The halo keeps its own copy of s', so a block needs only
// w' of its neighbours' faces, which are published together with the partial
// sums: one exchange an iteration.
//
// Exchange.  Every published 64-bit word carries 32 bits of data and a 32-bit
// tag (the iteration number), and a reader polls the word until the tag is
// the one it waits for.  So data and signal travel together: no fence, no
// counter, no second round trip.  Two buffers alternate; a block writes
// iteration i + 2 only after it has read every block's sums of i + 1, which
// each block publishes after its last read of i.  The blocks wait on one
// another, so the launch is cooperative; every poll is bounded.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>

#include "nn_hh.cuh"
#include "nn_internal.cuh"
#include "nn_quad.cuh"

namespace {
constexpr int RT = 512;               // most threads of a block
constexpr int POLL_LIMIT = 1 << 22;   // some seconds
constexpr int MAX_BLOCKS = 160;

typedef unsigned long long u64;

__device__ __forceinline__ void st_tagged(ulonglong2* p, uint32_t a, uint32_t b, uint32_t tag)
{
    const u64 t = (u64)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | a), "l"(t | b) : "memory");
}
__device__ __forceinline__ ulonglong2 ld_tagged(const ulonglong2* p)
{
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
// four values in one 32-byte sector
struct Tagged4 {
    u64 w[4];
};
__device__ __forceinline__ void st_tagged4(Tagged4* p, const float (&v)[4], uint32_t tag)
{
    const u64 t = (u64)tag << 32;
    asm volatile("st.relaxed.gpu.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(t | __float_as_uint(v[0])),
                 "l"(t | __float_as_uint(v[1])), "l"(t | __float_as_uint(v[2])), "l"(t | __float_as_uint(v[3]))
                 : "memory");
}
__device__ __forceinline__ Tagged4 ld_tagged4(const Tagged4* p)
{
    Tagged4 v;
    asm volatile("ld.relaxed.gpu.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(v.w[0]), "=l"(v.w[1]), "=l"(v.w[2]), "=l"(v.w[3])
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ bool tagged(const Tagged4& v, uint32_t tag)
{
    return (uint32_t)(v.w[0] >> 32) == tag && (uint32_t)(v.w[1] >> 32) == tag && (uint32_t)(v.w[2] >> 32) == tag &&
           (uint32_t)(v.w[3] >> 32) == tag;
}
__device__ __forceinline__ bool tagged(const ulonglong2& v, uint32_t tag)
{
    return (uint32_t)(v.x >> 32) == tag && (uint32_t)(v.y >> 32) == tag;
}

// A double as the two data words of a tagged pair.
__device__ __forceinline__ void st_tagged(ulonglong2* p, double v, uint32_t tag)
{
    st_tagged(p, (uint32_t)__double2loint(v), (uint32_t)__double2hiint(v), tag);
}
__device__ __forceinline__ double tagged_double(const ulonglong2& v)
{
    return __hiloint2double((int)(uint32_t)v.y, (int)(uint32_t)v.x);
}

// n / d.  The FP64 pipe has a latency of 65 cycles (a division takes 570), so a
// float's reciprocal of the mantissa (error e < 2^-21) is refined once, by
// Halley's third-order step x (1 + e + e e), whose error e^3 is below FP64's
// rounding; the exponent goes to n, beside that chain.
__device__ __forceinline__ double fast_div(double n, double d)
{
    const int hi = __double2hiint(d), lo = __double2loint(d), e = hi >> 20 & 0x7ff;
    if (e < 2 || e > 2044) return n / d;  // zero, subnormal, non-finite, or of an extreme reciprocal
    const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, lo);
    const float s = nn_rcp(__int_as_float((hi & 0xfffff) << 3 | (unsigned)lo >> 29 | 0x3f800000));  // (0.5, 1]
    const unsigned b = __float_as_uint(s);
    const double x = __hiloint2double((int)((b >> 3) + (896u << 20)), (int)(b << 29));
    const double r = fma(-m, x, 1.0);
    const double ns = n * __hiloint2double((hi & (int)0x80000000) | (2046 - e) << 20, 0);
    return ns * fma(x, fma(r, r, r), x);
}

struct RcgArgs {
    int nx, ny, nz;
    int by, bz, nyb, nb;       // brick, bricks along y, bricks in all
    int quads, pitch, hq;      // quads a row, shared row pitch, halo quads of a brick
    float op_alpha, onepb, invd;
    float half_ia;             // 1 / (2 alpha)
    float c, inv_c;            // u = c M r, c a power of two (nn_jacobi_scale)
    double diag;               // constant coefficients: 1 / invd
    double rtol2;
    const float* b;
    float* x;
    const float* D;
    float4* xw;                // x during the solve: [block][plane][thread]
    ulonglong2* rec;           // [2][nb][4]: tagged g, d, rho, (b, b)
    Tagged4* halo;             // [2][nb][hq]: tagged w' of a brick's faces
    unsigned* epoch;           // first tag of the next solve
    double* scal;              // out: rho, (b, b)
    int* flags;                // out: [0] 1 converged, 2 max_iter, 3 error  [1] iterations  [2] a wait gave up
    int max_iter;
};

// One solve by the a.nb blocks that call this with ranks 0 .. a.nb - 1, first
// tag base + 1.  Returns the last tag used; fail: a wait gave up.
template <int NZ, bool HET>
__device__ __forceinline__ uint32_t rcg_solve(const RcgArgs& a, const int rank, const uint32_t base, float4* smem4,
                                              bool& fail)
{
    __shared__ __align__(16) float ws[4][RT / 32];
    __shared__ double wp[4][MAX_BLOCKS / 32];
    __shared__ double s_gamma, s_den, s_lim, s_bb, s_rr;  // the first thread's, kept out of everyone's registers
    static_assert(MAX_BLOCKS == 160, "five groups of 32 blocks");
    __shared__ float sc_alpha, sc_beta;
    __shared__ int sc_stop, sc_fail;
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int jb = rank % a.nyb, kb = rank / a.nyb;
    const int y0 = jb * a.by, z0 = kb * a.bz;
    const int byn = min(a.by, a.ny - y0), bzn = min(a.bz, a.nz - z0);
    const int rows = a.by + 2, psz = rows * a.pitch;  // shared plane
    float* U = reinterpret_cast<float*>(smem4);
    float* Ds = U + (HET ? (a.bz + 2) * psz : 0);
    float4* W = reinterpret_cast<float4*>(Ds + (a.bz + 2) * psz);
    float4* SH = W + a.bz * T;
    float4* WH = SH + a.hq;
    int2* HT = reinterpret_cast<int2*>(WH + a.hq);  // per halo quad: shared place, face slot it comes from (-1: none)
    const int q = tid % a.quads, j = tid / a.quads;
    const bool act = j < byn;
    const int i0 = 4 * q;
    const int ub = psz + (min(j, a.by - 1) + 1) * a.pitch + 4 + i0;  // own quad in plane 0
    const int64_t gsz = (int64_t)a.nx * a.ny;
    const int64_t g0 = i0 + (int64_t)a.nx * (y0 + j) + gsz * z0;
    const bool full = i0 + 4 <= a.nx;
    // halo duty is on all warps but the first (there are two or more), which
    // polls the sums
    const int ht = tid - 32, hstep = T - 32;
    const int yq = a.bz * a.quads, zq = a.by * a.quads;  // halo quads: y-, y+ (yq each), z-, z+ (zq each)

    // halo quad h: its place in shared memory, the brick and face slot it
    // comes from (-1: outside the grid or the brick), the first cell's index
    auto halo_at = [&](int h, int& sm, int& src, int& slot, int64_t& g) {
        int f, r;
        if (h < 2 * yq) { f = h >= yq; r = h - f * yq; }
        else { f = 2 + (h - 2 * yq >= zq); r = h - 2 * yq - (f - 2) * zq; }
        const int line = r / a.quads, hx = r - line * a.quads;
        int lj, lk;
        if (f < 2) {
            lk = line;
            lj = f ? byn : -1;
            src = f ? (jb + 1 < a.nyb ? rank + 1 : -1) : (jb > 0 ? rank - 1 : -1);
            slot = (f ? 0 : yq) + r;
            if (lk >= bzn) src = -1;
        } else {
            lj = line;
            lk = f == 3 ? bzn : -1;
            src = f == 3 ? (z0 + a.bz < a.nz ? rank + a.nyb : -1) : (kb > 0 ? rank - a.nyb : -1);
            slot = 2 * yq + (f == 3 ? 0 : zq) + r;
            if (lj >= byn) src = -1;
        }
        sm = (lk + 1) * psz + (lj + 1) * a.pitch + 4 + 4 * hx;
        g = 4 * hx + (int64_t)a.nx * (y0 + lj) + gsz * (z0 + lk);
    };

    Quad P[NZ], S[NZ];
#pragma unroll
    for (int k = 0; k < NZ; ++k) P[k] = S[k] = quad_zero();
    float4* xw = a.xw + (size_t)rank * a.bz * T + tid;  // the thread's x

    // ---- load x with halo; with a cell field, v = 1 / (2 alpha D): the face
    // coefficient alpha 2 D D' / (D + D') is 1 / (v + v'), and a copy of the
    // cell's own v outside the grid gives the boundary face alpha D
    for (int c = tid; c < (a.bz + 2) * psz / 4; c += T) reinterpret_cast<float4*>(U)[c] = make_float4(0, 0, 0, 0);
    if (tid == 0) sc_fail = 0;
    if (tid < 4 * (RT / 32)) (&ws[0][0])[tid] = 0.0f;
    if (tid < 4 * (MAX_BLOCKS / 32)) (&wp[0][0])[tid] = 0.0;
    __syncthreads();
    bool poison = false;  // two neighbours with D = 0: their face coefficient is 0 / 0
    if (act) {
#pragma unroll
        for (int k = 0; k < NZ; ++k) {
            if (k >= bzn) break;
            Quad x = quad_zero(), v = quad_zero();
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (i0 + e < a.nx) {
                    const int64_t c = g0 + k * gsz + e;
                    at(x, e) = a.x[c];
                    if (HET) {
                        const float d = a.D[c];
                        at(v, e) = __fdiv_rn(a.half_ia, d);
                        poison |= isinf(d);  // 2 D1 D2 / (D1 + D2) = inf / inf
                        if (d == 0.0f)
                            poison |= (i0 + e > 0 && a.D[c - 1] == 0.0f) || (i0 + e < a.nx - 1 && a.D[c + 1] == 0.0f) ||
                                      (y0 + j > 0 && a.D[c - a.nx] == 0.0f) ||
                                      (y0 + j < a.ny - 1 && a.D[c + a.nx] == 0.0f) ||
                                      (z0 + k > 0 && a.D[c - gsz] == 0.0f) || (z0 + k < a.nz - 1 && a.D[c + gsz] == 0.0f);
                    }
                }
            quad_st(U + ub + k * psz, x);
            quad_st(reinterpret_cast<float*>(xw + k * T), x);
            if (HET) {
                float* row = Ds + ub + k * psz;
                quad_st(row, v);
                if (q == 0) row[-1] = v.a.v[0];
                if (q == a.quads - 1) row[a.nx - i0] = row[a.nx - i0 - 1];
            }
        }
    }
    for (int h = tid; h < a.hq; h += T) {
        int sm, src, slot;
        int64_t g;
        halo_at(h, sm, src, slot, g);
        SH[h] = make_float4(0, 0, 0, 0);
        HT[h] = make_int2(sm, src < 0 ? -1 : src * a.hq + slot);
        const int lj = h < 2 * yq ? 0 : (h - 2 * yq) % zq / a.quads, lk = h < 2 * yq ? h % yq / a.quads : 0;
        if (lj >= byn || lk >= bzn) continue;
        const int hx = (sm - 4) % a.pitch;  // x of the quad's first cell
        // the brick's own cell beside a cell outside the grid
        const int64_t in = h < yq ? a.nx : h < 2 * yq ? -(int64_t)a.nx : h < 2 * yq + zq ? gsz : -gsz;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (hx + e >= a.nx) break;
            if (src >= 0) U[sm + e] = a.x[g + e];
            if (HET) Ds[sm + e] = __fdiv_rn(a.half_ia, a.D[src >= 0 ? g + e : g + in + e]);
        }
    }
    __syncthreads();

    // ---- stencil over the thread's column: out(k, u, A u, diag) per plane
    const V2 onepb = vb<2>(a.onepb), alpha2 = vb<2>(a.op_alpha), six = vb<2>(6.0f), minus = vb<2>(-1.0f);
    const bool edge_l = lane == 0 || q == 0, edge_r = lane == 31 || q == a.quads - 1;
    // all threads take part (x neighbours pass between lanes); those without
    // a quad read their clamped row and call nothing
    auto column = [&](auto out) {
        Quad um = quad_ld(U + ub - psz), uc = quad_ld(U + ub), vc, cz;
        if (HET) {
            const Quad vm = quad_ld(Ds + ub - psz);
            vc = quad_ld(Ds + ub);
            cz = {vrcp(vadd(vc.a, vm.a)), vrcp(vadd(vc.b, vm.b))};
        }
#pragma unroll
        for (int k = 0; k < NZ; ++k) {
            if (k >= bzn) break;
            const float* u = U + ub + k * psz;
            const Quad ym = quad_ld(u - a.pitch), yp = quad_ld(u + a.pitch), un = quad_ld(u + psz);
            float xl = __shfl_up_sync(0xffffffffu, uc.b.v[1], 1), xr = __shfl_down_sync(0xffffffffu, uc.a.v[0], 1);
            if (edge_l) xl = u[-1];
            if (edge_r) xr = u[4];
            Quad A, dg;
            if (!HET) {
                V2 na{{xl + uc.a.v[1], uc.a.v[0] + uc.b.v[0]}}, nb{{uc.a.v[1] + uc.b.v[1], uc.b.v[0] + xr}};
                na = vadd(vadd(vadd(vadd(na, ym.a), yp.a), um.a), un.a);
                nb = vadd(vadd(vadd(vadd(nb, ym.b), yp.b), um.b), un.b);
                // 6 u - (neighbours) before alpha: a coefficient 1 + beta + 6 alpha
                // rounded to FP32 would shift the mass term by 6 alpha 2^-24
                A = {vfma(alpha2, vfma(six, uc.a, vmul(minus, na)), vmul(onepb, uc.a)),
                     vfma(alpha2, vfma(six, uc.b, vmul(minus, nb)), vmul(onepb, uc.b))};
            } else {
                const float* d = Ds + ub + k * psz;
                const Quad vm = quad_ld(d - a.pitch), vp = quad_ld(d + a.pitch), vn = quad_ld(d + psz);
                float dl = __shfl_up_sync(0xffffffffu, vc.b.v[1], 1), dr = __shfl_down_sync(0xffffffffu, vc.a.v[0], 1);
                if (edge_l) dl = d[-1];
                if (edge_r) dr = d[4];
                // x faces: coefficients and fluxes of the quad's five faces
                const float c0 = nn_rcp(dl + vc.a.v[0]), c1 = nn_rcp(vc.a.v[0] + vc.a.v[1]);
                const float c2 = nn_rcp(vc.a.v[1] + vc.b.v[0]), c3 = nn_rcp(vc.b.v[0] + vc.b.v[1]);
                const float c4 = nn_rcp(vc.b.v[1] + dr);
                const float f0 = c0 * (uc.a.v[0] - xl), f1 = c1 * (uc.a.v[0] - uc.a.v[1]);
                const float f2 = c2 * (uc.a.v[1] - uc.b.v[0]), f3 = c3 * (uc.b.v[0] - uc.b.v[1]);
                const float f4 = c4 * (uc.b.v[1] - xr);
                auto half = [&](const V2& cx, const V2& fx, const V2& u0, const V2& ym1, const V2& yp1, const V2& um1,
                                const V2& un1, const V2& v0, const V2& vm1, const V2& vp1, const V2& vn1, V2& czh,
                                V2& A1, V2& d1) {
                    const V2 cm = vrcp(vadd(v0, vm1)), cp = vrcp(vadd(v0, vp1)), cn = vrcp(vadd(v0, vn1));
                    V2 acc = vfma(cm, vsub(u0, ym1), fx);
                    acc = vfma(cp, vsub(u0, yp1), acc);
                    acc = vfma(czh, vsub(u0, um1), acc);
                    acc = vfma(cn, vsub(u0, un1), acc);
                    A1 = vfma(onepb, u0, acc);
                    d1 = vadd(vadd(vadd(vadd(vadd(cx, cm), cp), czh), cn), onepb);
                    czh = cn;
                };
                half({{c0 + c1, c1 + c2}}, {{f0 + f1, f2 - f1}}, uc.a, ym.a, yp.a, um.a, un.a, vc.a, vm.a, vp.a, vn.a,
                     cz.a, A.a, dg.a);
                half({{c2 + c3, c3 + c4}}, {{f3 - f2, f4 - f3}}, uc.b, ym.b, yp.b, um.b, un.b, vc.b, vm.b, vp.b, vn.b,
                     cz.b, A.b, dg.b);
                vc = vn;
            }
            if (act) out(k, uc, A, dg);
            um = uc;
            uc = un;
        }
    };
    // the four values of plane k on the brick's faces, for the neighbours
    const bool face[4] = {act && j == 0 && jb > 0, act && j == byn - 1 && jb + 1 < a.nyb, kb > 0, z0 + a.bz < a.nz};
    auto publish = [&](int k, const Quad& v, uint32_t tag) {
        Tagged4* f = a.halo + ((size_t)(tag & 1) * a.nb + rank) * a.hq;
        const float c[4] = {v.a.v[0], v.a.v[1], v.b.v[0], v.b.v[1]};
        auto put = [&](int slot) { st_tagged4(f + slot, c, tag); };
        if (face[0]) put(k * a.quads + q);
        if (face[1]) put(yq + k * a.quads + q);
        if (k == 0 && face[2]) put(2 * yq + j * a.quads + q);
        if (k == bzn - 1 && face[3]) put(2 * yq + zq + j * a.quads + q);
    };
    // the neighbours' faces into out(h, shared place, values); RB quads in flight
    auto receive = [&](uint32_t tag, auto out) {
        constexpr int RB = 2;  // (three spill)
        if (ht < 0) return;
        const Tagged4* f = a.halo + (size_t)(tag & 1) * a.nb * a.hq;
        for (int h = ht; h < a.hq; h += RB * hstep) {
            int2 at[RB];
            Tagged4 v[RB];
#pragma unroll
            for (int m = 0; m < RB; ++m) {
                at[m] = h + m * hstep < a.hq ? HT[h + m * hstep] : make_int2(0, -1);
                if (at[m].y >= 0) v[m] = ld_tagged4(f + at[m].y);
            }
#pragma unroll
            for (int m = 0; m < RB; ++m) {
                if (at[m].y < 0) continue;
                int it = 0;
                while (!tagged(v[m], tag)) {
                    if (++it > POLL_LIMIT || *(volatile int*)&sc_fail) {
                        sc_fail = 1;
                        break;
                    }
                    v[m] = ld_tagged4(f + at[m].y);
                }
                out(h + m * hstep, at[m].x,
                    make_float4(__uint_as_float((uint32_t)v[m].w[0]), __uint_as_float((uint32_t)v[m].w[1]),
                                __uint_as_float((uint32_t)v[m].w[2]), __uint_as_float((uint32_t)v[m].w[3])));
            }
        }
    };
    auto vmask = [&](Quad& v) {  // zeros in the cells past the row's end
        if (!full)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (i0 + e >= a.nx) at(v, e) = 0.0f;
    };

    // ---- u0 = M (b - A x0)
    float acc_b = 0.0f;
    const V2 idg = vb<2>(a.invd);
    column([&](int k, const Quad&, const Quad& A, const Quad& dg) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (i0 + e < a.nx) {
                const float bv = a.b[g0 + k * gsz + e];
                at(S[k], e) = HET ? __fdividef(bv - at(A, e), at(dg, e)) : (bv - at(A, e)) * (a.c * a.invd);
                if (poison) at(S[k], e) = nanf("");
                acc_b += bv * bv;
            }
        publish(k, S[k], base + 1);
    });
    __syncthreads();
    if (act) {
#pragma unroll
        for (int k = 0; k < NZ; ++k) {
            if (k >= bzn) break;
            quad_st(U + ub + k * psz, S[k]);
            S[k] = quad_zero();
        }
    }
    receive(base + 1, [&](int, int sm, float4 v) { *reinterpret_cast<float4*>(U + sm) = v; });

    uint32_t tag = base + 2;
    int it = -1;
    float al_prev = 0.0f;
    bool owed = false;  // x lacks the last direction, al_prev P
    for (;; ++tag) {
        __syncthreads();
        if (sc_fail) break;
        // ---- w' = M A u, the sums and the faces
        V2 ag{{0, 0}}, ad{{0, 0}}, ar{{0, 0}};
        column([&](int k, const Quad& u, const Quad& A, const Quad& dg) {
            Quad w, r;
            if (HET) {
                w = {vmul(A.a, vrcp(dg.a)), vmul(A.b, vrcp(dg.b))};
                r = {vmul(u.a, dg.a), vmul(u.b, dg.b)};
                vmask(w);
                vmask(r);
            } else {
                w = {vmul(A.a, idg), vmul(A.b, idg)};
                r = u;
                vmask(w);
            }
            publish(k, w, tag);
            quad_st(reinterpret_cast<float*>(W + k * T + tid), w);
            ag = vfma(r.b, u.b, vfma(r.a, u.a, ag));
            if (HET) {
                Quad m = A;
                vmask(m);
                ad = vfma(m.b, u.b, vfma(m.a, u.a, ad));
                ar = vfma(r.b, r.b, vfma(r.a, r.a, ar));
            } else {
                ad = vfma(A.b, u.b, vfma(A.a, u.a, ad));
            }
        });
        // block sums: FP32 within a warp, FP64 across warps and blocks
        const float v0 = nn_warp_sumf(ag.v[0] + ag.v[1]), v1 = nn_warp_sumf(ad.v[0] + ad.v[1]);
        const float v2 = HET ? nn_warp_sumf(ar.v[0] + ar.v[1]) : 0.0f;
        const float v3 = it < 0 ? nn_warp_sumf(acc_b) : 0.0f;
        if (lane == 0) {
            ws[0][warp] = v0;
            ws[1][warp] = v1;
            ws[2][warp] = v2;
            ws[3][warp] = v3;
        }
        __syncthreads();
        const int hl = lane & 15, up = lane >> 4;  // lanes 0-15: g, rho; 16-31: d, (b, b)
        const int np = (HET || it < 0) ? 2 : 1;    // pairs of sums to exchange: {g, d} and {rho, (b, b)}
        ulonglong2* rec = a.rec + 4 * (size_t)(tag & 1) * a.nb;
        if (warp == 0) {
            // lanes 4 w .. 4 w + 3: sum w, four warps each
            const int w = lane >> 2 & 3;
            const float4 v = *reinterpret_cast<const float4*>(&ws[w][4 * (lane & 3)]);
            double s0 = ((double)v.x + (double)v.y) + ((double)v.z + (double)v.w);
            s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
            s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
            if (lane == 4 * w && w < 2 * np) st_tagged(rec + 4 * rank + w, s0, tag);
        }
        // x takes two directions every second iteration: loaded here, behind
        // the wait
        Quad X[NZ];
        if (owed && act)
#pragma unroll
            for (int k = 0; k < NZ; ++k)
                if (k < bzn) X[k] = quad_ldcg(xw + k * T);
        receive(tag, [&](int h, int, float4 v) { WH[h] = v; });
        // every block adds all blocks' sums in the same order: a record a
        // thread, then warps (without the steps that would add zeros), then the
        // first warp
        // (rgamma, factor: 1 / g and 1 / (g a) = den / g^2 of the last iteration,
        // formed while the first thread waits)
        double rgamma = 0.0, factor = 0.0;
        for (int c0 = 32 * warp; c0 < a.nb; c0 += T) {
            const int c = c0 + lane;
            double t[4] = {0.0, 0.0, 0.0, 0.0};
            if (c < a.nb) {
                ulonglong2 v[4];
#pragma unroll
                for (int w = 0; w < 4; ++w)
                    if (w < 2 * np) v[w] = ld_tagged(rec + 4 * c + w);
                if (c == 0 && it >= 0) {
                    rgamma = 1.0 / s_gamma;
                    factor = s_den != 0.0 ? rgamma * rgamma * s_den : (double)INFINITY;
                }
#pragma unroll
                for (int w = 0; w < 4; ++w)
                    if (w < 2 * np) {
                        int n = 0;
                        while (!tagged(v[w], tag)) {
                            if (++n > POLL_LIMIT || *(volatile int*)&sc_fail) {
                                sc_fail = 1;
                                break;
                            }
                            v[w] = ld_tagged(rec + 4 * c + w);
                        }
                        t[w] = tagged_double(v[w]);
                    }
            }
            __syncwarp();
#pragma unroll
            for (int pr = 0; pr < 2; ++pr) {
                if (pr >= np) break;
                const double t0 = t[2 * pr], t1 = t[2 * pr + 1];
                double r = (up ? t1 : t0) + __shfl_xor_sync(0xffffffffu, up ? t0 : t1, 16);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
                    if (o < a.nb) r += __shfl_xor_sync(0xffffffffu, r, o);
                if (hl == 0) wp[2 * pr + up][c0 >> 5] = r;
            }
        }
        __syncthreads();
        if (warp == 0) {
            // lane w: sum w
            const double* t = wp[lane & 3];
            const double r = ((t[0] + t[1]) + (t[2] + t[3])) + t[4];
            const double d = __shfl_sync(0xffffffffu, r, 1);
            const double r2 = np > 1 ? __shfl_sync(0xffffffffu, r, 2) : 0.0;
            const double r3 = np > 1 ? __shfl_sync(0xffffffffu, r, 3) : 0.0;
            if (lane == 0) {
                // g = (r, u); with constant coefficients r holds (c r = diag u)
                // g / diag, which be and den, ratios of g, may use as it is
                const double g = HET ? r : r * a.diag;
                const double rr = HET ? r2 : g * a.diag;
                double den = d, be = 0.0;
                if (it < 0) {
                    s_bb = r3;
                    s_lim = a.rtol2 * ((double)a.c * a.c * r3);
                } else {
                    be = r * rgamma;
                    den = fma(-(r * r), factor, d);  // d - be g / a
                }
                const double al = den != 0.0 ? fast_div(g, den) : 0.0;
                const int stop = rr <= s_lim                       ? 1
                                 : it + 1 >= a.max_iter            ? 2
                                 : it < 0                          ? 0
                                 : !(isfinite(al) && isfinite(be)) ? 3
                                                                   : 0;
                s_gamma = r;
                s_den = den;
                s_rr = rr;
                sc_alpha = (float)al;
                sc_beta = (float)be;
                sc_stop = stop;
            }
        }
        __syncthreads();
        ++it;
        if (sc_fail || sc_stop) break;
        // ---- s', p, x, u (own cells and halo)
        const float al = sc_alpha, be = sc_beta;
        if (act) {
            const V2 al2 = vb<2>(al * a.inv_c), nal2 = vb<2>(-al), be2 = vb<2>(be), ap2 = vb<2>(al_prev * a.inv_c);
#pragma unroll
            for (int k = 0; k < NZ; ++k) {
                if (k >= bzn) break;
                float* up = U + ub + k * psz;
                const Quad w = quad_ld(reinterpret_cast<const float*>(W + k * T + tid)), u = quad_ld(up);
                S[k] = {vfma(be2, S[k].a, w.a), vfma(be2, S[k].b, w.b)};
                quad_st(up, {vfma(nal2, S[k].a, u.a), vfma(nal2, S[k].b, u.b)});
                const Quad p{vfma(be2, P[k].a, u.a), vfma(be2, P[k].b, u.b)};
                if (owed) {
                    const Quad x{vfma(ap2, P[k].a, X[k].a), vfma(ap2, P[k].b, X[k].b)};
                    quad_st(reinterpret_cast<float*>(xw + k * T), {vfma(al2, p.a, x.a), vfma(al2, p.b, x.b)});
                }
                P[k] = p;
            }
        }
        al_prev = al;
        owed = !owed;
        if (ht >= 0)
            for (int h = ht; h < a.hq; h += hstep) {
                const int2 at = HT[h];
                if (at.y < 0) continue;
                const float4 w = WH[h];
                float4 s = SH[h];
                s = make_float4(w.x + be * s.x, w.y + be * s.y, w.z + be * s.z, w.w + be * s.w);
                SH[h] = s;
                float4* up = reinterpret_cast<float4*>(U + at.x);
                const float4 u = *up;
                *up = make_float4(u.x - al * s.x, u.y - al * s.y, u.z - al * s.z, u.w - al * s.w);
            }
    }
    if (act) {
#pragma unroll
        for (int k = 0; k < NZ; ++k) {
            if (k >= bzn) break;
            Quad x = quad_ldcg(xw + k * T);
            if (owed) x = {vfma(vb<2>(al_prev * a.inv_c), P[k].a, x.a), vfma(vb<2>(al_prev * a.inv_c), P[k].b, x.b)};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (i0 + e < a.nx) a.x[g0 + k * gsz + e] = at(x, e);
        }
    }
    fail = sc_fail;
    if (tid == 0) {
        if (fail) {
            a.flags[2] = 1;
            a.flags[0] = 3;
        } else if (rank == 0) {
            a.flags[0] = sc_stop;
            a.flags[1] = it;
            a.flags[2] = 0;
            a.scal[0] = s_rr * a.inv_c * a.inv_c;
            a.scal[1] = s_bb;
        }
    }
    return tag;
}

template <int NZ, bool HET>
__global__ void __launch_bounds__(RT, 1) k_rcg(const RcgArgs a)
{
    extern __shared__ float4 smem4[];
    bool fail;
    const uint32_t base = *reinterpret_cast<volatile unsigned*>(a.epoch);
    const uint32_t tag = rcg_solve<NZ, HET>(a, blockIdx.x, base, smem4, fail);
    if (!fail && blockIdx.x == 0 && threadIdx.x == 0) *a.epoch = tag + 2;
}

// Many independent solves in one launch (the fields of a batch of networks).
// The blocks are split into groups; a group solves the instances of its list
// one after another.  Before each it exchanges a tag that says every block has
// left the previous solve (its buffers may be written again) and carries the
// last tag used, since a block without a brick in a solve has not counted its
// iterations.
struct RcgGroup {
    int first, count, width;   // its instances in the list, its blocks
    int64_t rec, halo, xw;     // its parts of the buffers
};
struct RcgBatchArgs {
    const RcgArgs* inst;       // per instance: shape and operator
    const int64_t* off;        // first cell of each instance
    const int2* block;         // per block: group, rank
    const RcgGroup* group;
    const int* list;
    const float* b;
    float* x;
    ulonglong2* start;         // [2][blocks]: tags of the exchange before a solve
    uint32_t seq;              // first of those tags
    unsigned* epoch;           // per group
    double* scal;              // [instances][2]
    int* flags;                // [instances][4]
    double rtol2;
    int max_iter;
};

template <int NZ>
__global__ void __launch_bounds__(RT, 1) k_rcg_batch(const RcgBatchArgs B)
{
    extern __shared__ float4 smem4[];
    __shared__ RcgArgs a;
    __shared__ unsigned last;
    __shared__ int gave_up;
    const int tid = threadIdx.x, rank = B.block[blockIdx.x].y, first = (int)blockIdx.x - rank;
    const RcgGroup g = B.group[B.block[blockIdx.x].x];
    unsigned* epoch = B.epoch + B.block[blockIdx.x].x;
    uint32_t tag = *reinterpret_cast<volatile unsigned*>(epoch);
    if (tid == 0) gave_up = 0;
    for (int k = 0; k < g.count; ++k) {
        const uint32_t s = B.seq + k;
        ulonglong2* slot = B.start + (size_t)(s & 1) * gridDim.x + first;
        __syncthreads();
        if (tid == 0) {
            const int q = B.list[g.first + k];
            a = B.inst[q];
            a.b = B.b + B.off[q];
            a.x = B.x + B.off[q];
            a.flags = B.flags + 4 * q;
            a.scal = B.scal + 2 * q;
            a.rtol2 = B.rtol2;
            a.max_iter = B.max_iter;
            st_tagged(slot + rank, tag, 0, s);
        }
        __syncthreads();
        if (tid < g.width) {
            int n = 0;
            ulonglong2 v = ld_tagged(slot + tid);
            while (!tagged(v, s)) {
                if (++n > POLL_LIMIT) {
                    gave_up = 1;
                    break;
                }
                v = ld_tagged(slot + tid);
            }
            if (tid == 0) last = (unsigned)v.x;  // the first block has a brick in every solve: its tag is the latest
        }
        __syncthreads();
        if (gave_up) {
            if (tid == 0) {
                a.flags[2] = 1;
                a.flags[0] = 3;
            }
            return;
        }
        tag = last;
        bool fail = false;
        if (rank < a.nb) tag = rcg_solve<NZ, false>(a, rank, tag, smem4, fail);
        if (fail) return;
    }
    // the group's blocks have all read it: they have been through the last start
    if (rank == 0 && tid == 0) *epoch = tag + 2;
}

const void* batch_kernel_of(int nz)
{
    switch (nz) {
        case 1: return (const void*)k_rcg_batch<1>;
        case 2: return (const void*)k_rcg_batch<2>;
        case 3: return (const void*)k_rcg_batch<3>;
        case 4: return (const void*)k_rcg_batch<4>;
        case 5: return (const void*)k_rcg_batch<5>;
        case 6: return (const void*)k_rcg_batch<6>;
        default: return (const void*)k_rcg_batch<7>;
    }
}

template <bool HET>
const void* kernel_of(int nz)
{
    switch (nz) {
        case 1: return (const void*)k_rcg<1, HET>;
        case 2: return (const void*)k_rcg<2, HET>;
        case 3: return (const void*)k_rcg<3, HET>;
        case 4: return (const void*)k_rcg<4, HET>;
        case 5: return (const void*)k_rcg<5, HET>;
        case 6: return HET ? nullptr : (const void*)k_rcg<6, false>;
        case 7: return HET ? nullptr : (const void*)k_rcg<7, false>;
        default: return nullptr;
    }
}
}  // namespace

static void rcg_operator(RcgArgs& a, double alpha, double beta, bool het)
{
    a.c = nn_jacobi_scale(alpha, beta, het);
    a.inv_c = 1.0f / a.c;
    a.op_alpha = (float)alpha;
    a.onepb = (float)(1.0 + beta);
    a.invd = (float)(1.0 / (1.0 + beta + 6.0 * alpha));
    a.half_ia = (float)(0.5 / alpha);
    a.diag = 1.0 / (double)a.invd;
}

struct nn_rcg_plan {
    nn_ctx* ctx = nullptr;
    RcgArgs a{};
    const void* kernel = nullptr;
    int threads = 0;
    size_t smem = 0, rec_bytes = 0, halo_bytes = 0;
    bool timing = false;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    float last_ms = 0.0f;
    int last_iters = 0;
};

void nn_rcg_plan_destroy(nn_rcg_plan* pl)
{
    if (!pl) return;
    if (pl->ctx) cudaStreamSynchronize(pl->ctx->stream);
    nn_release(pl->a.xw);
    nn_release(pl->a.rec);
    nn_release(pl->a.halo);
    nn_release(pl->a.epoch);
    nn_release(pl->a.scal);
    nn_release(pl->a.flags);
    if (pl->e0) cudaEventDestroy(pl->e0);
    if (pl->e1) cudaEventDestroy(pl->e1);
    nn_ctx* ctx = pl->ctx;
    delete pl;
    nn_ctx_release(ctx);
}

static nn_status rcg_reset(nn_rcg_plan* pl, cudaStream_t cs)
{
    NN_CUDA(pl->ctx, cudaMemsetAsync(pl->a.rec, 0, pl->rec_bytes, cs));
    NN_CUDA(pl->ctx, cudaMemsetAsync(pl->a.halo, 0, pl->halo_bytes, cs));
    NN_CUDA(pl->ctx, cudaMemsetAsync(pl->a.epoch, 0, sizeof(unsigned), cs));
    return NN_OK;
}

// Brick of the grid: the (by, bz) whose blocks fit the chip (one a SM, threads
// and shared memory) at the least estimated cycles of an iteration.  Measured
// on bricks of 8 to 512 quads a plane: a plane costs about 600 cycles of
// latency and 1.3 a quad, 1.6 times that with a cell field; a round of halo
// loads (two a thread, the first warp has none) about 600.
// limit: blocks to use at most; all_threads: blocks of RT threads.  Returns the
// estimate, 0 where nothing fits.
static double rcg_shape(int limit, bool het, bool all_threads, RcgArgs& a, int& threads, size_t& smem)
{
    const int quads = (a.nx + 3) / 4;
    const int nzmax = het ? 5 : 7;
    if (quads > RT) return 0.0;
    double best = 0.0;
    for (int by = 1; by <= std::min(a.ny, RT / quads); ++by)
        for (int bz = 1; bz <= std::min(a.nz, nzmax); ++bz) {
            const int nyb = (a.ny + by - 1) / by;
            const int64_t nb = (int64_t)nyb * ((a.nz + bz - 1) / bz);
            if (nb > limit) continue;
            // a thread polls one block's sums, and spare warps share the halo
            const int Q = quads * by, T = all_threads ? RT : std::max(192, (Q + 31) / 32 * 32);
            const int pitch = 4 * quads + 8, hq = 2 * quads * (by + bz);
            const size_t sm = (size_t)(bz + 2) * (by + 2) * pitch * 4 * (het ? 2 : 1) +
                              ((size_t)bz * T + 2 * (size_t)hq) * 16 + (size_t)hq * 8;
            if (sm > 225 * 1024) continue;
            const double cost = (het ? 1.6 : 1.0) * bz * (600.0 + 1.3 * Q) +
                                600.0 * ((hq + 2 * (T - 32) - 1) / (2 * (T - 32))) + 3.0 * nb;
            if (best > 0.0 && cost >= best) continue;
            best = cost;
            a.by = by; a.bz = bz; a.nyb = nyb; a.nb = (int)nb;
            a.quads = quads; a.pitch = pitch; a.hq = hq;
            threads = T;
            smem = sm;
        }
    return best;
}

// NN_ERR_UNSUPPORTED when the grid does not fit (the caller keeps its other
// solvers).  D stays owned by the caller and is read at each solve.
nn_status nn_rcg_plan_create(nn_ctx* ctx, int nx, int ny, int nz, double alpha, double beta, const float* D,
                             nn_rcg_plan** out)
{
    *out = nullptr;
    RcgArgs a{};
    a.nx = nx; a.ny = ny; a.nz = nz;
    int threads = 0, coop = 0;
    size_t smem = 0;
    if (rcg_shape(std::min(ctx->num_sms, MAX_BLOCKS), D != nullptr, false, a, threads, smem) == 0.0)
        return NN_ERR_UNSUPPORTED;
    const void* kernel = D ? kernel_of<true>(a.bz) : kernel_of<false>(a.bz);
    if (!kernel) return NN_ERR_UNSUPPORTED;
    NN_CUDA(ctx, cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
    NN_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024));
    int per_sm = 0;
    NN_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    if (!coop || per_sm < 1) return NN_ERR_UNSUPPORTED;
    rcg_operator(a, alpha, beta, D != nullptr);
    a.D = D;
    nn_rcg_plan* pl = new nn_rcg_plan();
    pl->ctx = ctx;
    nn_ctx_retain(ctx);
    pl->a = a;
    pl->kernel = kernel;
    pl->threads = threads;
    pl->smem = smem;
    pl->rec_bytes = sizeof(ulonglong2) * 8 * (size_t)a.nb;
    pl->halo_bytes = sizeof(Tagged4) * 2 * (size_t)a.nb * a.hq;
    nn_status st = nn_alloc(ctx, &pl->a.rec, 8 * (size_t)a.nb);
    if (st == NN_OK) st = nn_alloc(ctx, &pl->a.xw, (size_t)a.nb * a.bz * threads);
    if (st == NN_OK) st = nn_alloc(ctx, &pl->a.halo, 2 * (size_t)a.nb * a.hq);
    if (st == NN_OK) st = nn_alloc(ctx, &pl->a.epoch, 1);
    if (st == NN_OK) st = nn_alloc(ctx, &pl->a.scal, 2);
    if (st == NN_OK) st = nn_alloc(ctx, &pl->a.flags, 4);
    if (st == NN_OK) st = rcg_reset(pl, ctx->stream);
    if (st != NN_OK) {
        nn_rcg_plan_destroy(pl);
        return st;
    }
    // solves may run on other streams
    st = nn_cuda_check(ctx, cudaStreamSynchronize(ctx->stream), "nn_rcg_plan_create");
    if (st != NN_OK) {
        nn_rcg_plan_destroy(pl);
        return st;
    }
    *out = pl;
    return NN_OK;
}

void nn_rcg_set_timing(nn_rcg_plan* pl, bool on) { pl->timing = on; }
void nn_rcg_last_timing(const nn_rcg_plan* pl, float* ms, int* iters)
{
    *ms = pl->last_ms;
    *iters = pl->last_iters;
}

// The whole solve on stream cs (x: initial guess in, solution out).
nn_status nn_rcg_begin(nn_rcg_plan* pl, const float* d_b, float* d_x, double rtol, int max_iter, cudaStream_t cs)
{
    nn_ctx* ctx = pl->ctx;
    pl->a.b = d_b;
    pl->a.x = d_x;
    pl->a.rtol2 = rtol * rtol;
    pl->a.max_iter = max_iter;
    if (pl->timing && !pl->e0) {
        NN_CUDA(ctx, cudaEventCreate(&pl->e0));
        NN_CUDA(ctx, cudaEventCreate(&pl->e1));
    }
    if (pl->timing) NN_CUDA(ctx, cudaEventRecord(pl->e0, cs));
    void* args[] = {&pl->a};
    NN_CUDA(ctx, cudaLaunchCooperativeKernel(pl->kernel, dim3(pl->a.nb), dim3(pl->threads), args, pl->smem, cs));
    ctx->launches++;
    if (pl->timing) NN_CUDA(ctx, cudaEventRecord(pl->e1, cs));
    return NN_OK;
}

nn_status nn_rcg_finish(nn_rcg_plan* pl, cudaStream_t cs, int* iters, double* relres, int* converged)
{
    nn_ctx* ctx = pl->ctx;
    int h_flags[4] = {0, 0, 0, 0};
    double h_scal[2] = {0.0, 0.0};
    NN_CUDA(ctx, cudaMemcpyAsync(h_flags, pl->a.flags, sizeof h_flags, cudaMemcpyDeviceToHost, cs));
    NN_CUDA(ctx, cudaMemcpyAsync(h_scal, pl->a.scal, sizeof h_scal, cudaMemcpyDeviceToHost, cs));
    NN_CUDA(ctx, cudaStreamSynchronize(cs));
    if (h_flags[2]) {
        NN_TRY(rcg_reset(pl, cs));
        NN_CUDA(ctx, cudaMemsetAsync(pl->a.flags, 0, sizeof h_flags, cs));
        NN_CUDA(ctx, cudaStreamSynchronize(cs));
        return nn_fail(ctx, NN_ERR_TIMEOUT, "k_rcg: a block's wait for its neighbours gave up");
    }
    if (pl->timing) {
        NN_CUDA(ctx, cudaEventElapsedTime(&pl->last_ms, pl->e0, pl->e1));
        pl->last_iters = h_flags[1];
    }
    if (iters) *iters = h_flags[1];
    if (relres) *relres = h_scal[1] > 0 ? std::sqrt(h_scal[0] / h_scal[1]) : 0.0;
    if (converged) *converged = h_flags[0] == 1;
    return NN_OK;
}

// ------------------------------------------------------------------ batches --

struct nn_rcg_batch {
    nn_ctx* ctx = nullptr;
    int n_inst = 0, blocks = 0, longest = 0;
    const void* kernel = nullptr;
    size_t smem = 0;
    RcgBatchArgs B{};
    // everything in one allocation; the first `zero` bytes hold the tagged words
    unsigned char* mem = nullptr;
    size_t zero = 0;
};

void nn_rcg_batch_destroy(nn_rcg_batch* pl)
{
    if (!pl) return;
    if (pl->ctx) cudaStreamSynchronize(pl->ctx->stream);
    nn_release(pl->mem);
    nn_ctx* ctx = pl->ctx;
    delete pl;
    nn_ctx_release(ctx);
}

static nn_status batch_reset(nn_rcg_batch* pl, cudaStream_t cs)
{
    NN_CUDA(pl->ctx, cudaMemsetAsync(pl->mem, 0, pl->zero, cs));
    pl->B.seq = 1;
    return NN_OK;
}

// Groups and their lists: columns of blocks, filled with instances from the
// largest side down so that no column is estimated to run longer than a bound;
// the least bound for which the columns fit the chip, by bisection.  An
// instance's estimate is the cycles of an iteration on the column's blocks
// times its side, to which its iterations are about proportional.
//
// NN_ERR_UNSUPPORTED when an instance does not fit, and for batches of so many
// small instances that the two launches an iteration of nn_bpcg.cu are faster: a
// block goes through its list one solve after another, each iteration with an
// exchange of about 3 us, while those launches work on all instances at once.
// Both times are estimated, in us and with as many iterations as the side (they
// are proportional to it in both): here the list's cycles, 5,500 more an
// iteration, and 12 us an instance; there 17 us an iteration, 14.5 ps a cell
// (instances in whole blocks of 2,048 cells), and 100 us.  The estimates agree
// with measured times to 30 %, so the resident form has to be 1.25 times as fast
// by them.  Measured, resident / two launches, us: 300 of 8^3 192 / 310, 600 of
// 8^3 356 / 334, 5000 of 8^3 2726 / 1051, 100 of 16^3 204 / 405, 600 of 16^3 1104 /
// 659, 300 of 24^3 1094 / 1290, 600 of 32^3 4568 / 7145, 256 of 64^3 22366 / 45362.
constexpr double EST_CYCLES_US = 1900.0, EST_EXCHANGE = 5500.0, EST_SOLVE_US = 12.0;
constexpr double EST_TWO_US = 17.0, EST_TWO_CELL_US = 14.5e-6, EST_TWO_SOLVE_US = 100.0, EST_MARGIN = 1.25;

nn_status nn_rcg_batch_create(nn_ctx* ctx, int n_inst, const int* sides, const int64_t* off, double alpha_unit,
                              double beta, nn_rcg_batch** out)
{
    *out = nullptr;
    const int sms = std::min(ctx->num_sms, MAX_BLOCKS);
    struct Shape {
        double cost = 0.0;
        RcgArgs a{};
        size_t smem = 0;
    };
    static const int widths[] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 14, 16, 19, 22, 25, 30, 38, 50, 76, 152};
    constexpr int W = sizeof widths / sizeof *widths;
    std::map<int, std::vector<Shape>> table;  // by side: a shape a width
    for (int b = 0; b < n_inst; ++b) table[sides[b]];
    for (auto& e : table) {
        e.second.resize(W);
        for (int w = 0; w < W; ++w) {
            Shape& s = e.second[(size_t)w];
            int threads = 0;
            s.a.nx = s.a.ny = s.a.nz = e.first;
            if (widths[w] <= sms) s.cost = rcg_shape(widths[w], false, true, s.a, threads, s.smem) * e.first;
            if (s.cost == 0.0) s.cost = -1.0;
        }
    }
    // the two-launch form's time; what one list would take that was spread over
    // the chip, at the least, answers for most batches without packing
    auto us = [](double cost, int side) { return (cost + EST_EXCHANGE * side) / EST_CYCLES_US + EST_SOLVE_US; };
    double two = EST_TWO_SOLVE_US + EST_TWO_US * table.rbegin()->first, least = 0.0;
    std::map<int, double> share;  // by side: blocks times time, over the chip
    for (const auto& e : table) {
        double s = 0.0;
        for (int w = 0; w < W; ++w) {
            const double c = e.second[(size_t)w].cost;
            if (c > 0.0 && (s == 0.0 || widths[w] * us(c, e.first) < s)) s = widths[w] * us(c, e.first);
        }
        share[e.first] = s / sms;
    }
    std::vector<const std::vector<Shape>*> shape((size_t)n_inst);
    for (int b = 0; b < n_inst; ++b) {
        const double g = sides[b];
        shape[(size_t)b] = &table[sides[b]];
        two += g * std::ceil(g * g * g / 2048.0) * 2048.0 * EST_TWO_CELL_US;
        least += share[sides[b]];
    }
    if (EST_MARGIN * least > two) return NN_ERR_UNSUPPORTED;
    std::vector<int> order((size_t)n_inst);
    for (int b = 0; b < n_inst; ++b) order[(size_t)b] = b;
    std::stable_sort(order.begin(), order.end(), [&](int p, int q) { return sides[p] > sides[q]; });
    struct Column {
        int w;  // of widths
        double height;
        std::vector<int> list;
    };
    std::vector<Column> cols;
    auto pack = [&](double bound) {
        cols.clear();
        int used = 0;
        for (int b : order) {
            const std::vector<Shape>& s = *shape[(size_t)b];
            Column* best = nullptr;
            double left = 0.0;
            for (Column& c : cols) {
                const double cost = s[(size_t)c.w].cost, rest = bound - c.height - cost;
                if (cost > 0.0 && rest >= 0.0 && (!best || rest < left)) {
                    best = &c;
                    left = rest;
                }
            }
            if (!best) {
                for (int w = 0; w < W; ++w) {
                    if (widths[w] > sms - used) return false;
                    if (s[(size_t)w].cost > 0.0 && s[(size_t)w].cost <= bound) {
                        used += widths[w];
                        cols.push_back({w, 0.0, {}});
                        best = &cols.back();
                        break;
                    }
                }
                if (!best) return false;
            }
            best->height += s[(size_t)best->w].cost;
            best->list.push_back(b);
        }
        return true;
    };
    double hi = 0.0;
    for (int b : order) {
        const std::vector<Shape>& s = *shape[(size_t)b];
        const double c = s[(size_t)(widths[W - 1] <= sms ? W - 1 : W - 2)].cost;
        if (c <= 0.0) return NN_ERR_UNSUPPORTED;
        hi += c;
    }
    hi *= 1.0 + 1e-9;  // (the sum of a column's costs in another order)
    double lo = 0.0;
    if (!pack(hi)) return NN_ERR_UNSUPPORTED;
    for (int q = 0; q < 14; ++q) {
        const double mid = 0.5 * (lo + hi);
        (pack(mid) ? hi : lo) = mid;
    }
    if (!pack(hi)) return NN_ERR_UNSUPPORTED;
    for (const Column& c : cols) {
        double t = 0.0;
        for (int b : c.list) t += us((*shape[(size_t)b])[(size_t)c.w].cost, sides[b]);
        if (EST_MARGIN * t > two) return NN_ERR_UNSUPPORTED;
    }

    nn_rcg_batch* pl = new nn_rcg_batch();
    pl->ctx = ctx;
    nn_ctx_retain(ctx);
    pl->n_inst = n_inst;
    std::vector<RcgArgs> inst((size_t)n_inst);
    std::vector<RcgGroup> group;
    std::vector<int2> block;
    std::vector<int> list;
    int nz = 1;
    size_t n_rec = 0, n_halo = 0, n_xw = 0;
    for (const Column& c : cols) {
        const int width = widths[c.w];
        RcgGroup g{(int)list.size(), (int)c.list.size(), width, (int64_t)n_rec, (int64_t)n_halo, (int64_t)n_xw};
        size_t halo = 0, xw = 0;
        for (int b : c.list) {
            const Shape& s = (*shape[(size_t)b])[(size_t)c.w];
            RcgArgs a = s.a;
            rcg_operator(a, alpha_unit * sides[b] * sides[b], beta, false);
            nz = std::max(nz, a.bz);
            pl->smem = std::max(pl->smem, s.smem);
            halo = std::max(halo, 2 * (size_t)a.nb * a.hq);
            xw = std::max(xw, (size_t)a.nb * a.bz * RT);
            inst[(size_t)b] = a;
            list.push_back(b);
        }
        for (int r = 0; r < width; ++r) block.push_back({(int)group.size(), r});
        n_rec += 8 * (size_t)width;
        n_halo += halo;
        n_xw += xw;
        pl->longest = std::max(pl->longest, g.count);
        group.push_back(g);
    }
    pl->blocks = (int)block.size();
    pl->kernel = batch_kernel_of(nz);
    const size_t N = (size_t)n_inst;
    size_t bytes = 0;
    auto part = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const size_t o_rec = part(sizeof(ulonglong2) * n_rec), o_halo = part(sizeof(Tagged4) * n_halo);
    const size_t o_start = part(sizeof(ulonglong2) * 2 * block.size()), o_epoch = part(sizeof(unsigned) * group.size());
    pl->zero = bytes;
    const size_t o_xw = part(sizeof(float4) * n_xw), o_scal = part(sizeof(double) * 2 * N), o_flags = part(sizeof(int) * 4 * N);
    const size_t o_inst = part(sizeof(RcgArgs) * N), o_off = part(sizeof(int64_t) * N);
    const size_t o_block = part(sizeof(int2) * block.size()), o_group = part(sizeof(RcgGroup) * group.size());
    const size_t o_list = part(sizeof(int) * list.size());
    nn_status st = nn_alloc(ctx, &pl->mem, bytes);
    if (st != NN_OK) {
        nn_rcg_batch_destroy(pl);
        return st;
    }
    auto at = [&](size_t o) { return (void*)(pl->mem + o); };
    for (const RcgGroup& g : group)
        for (int k = 0; k < g.count; ++k) {
            RcgArgs& a = inst[(size_t)list[(size_t)(g.first + k)]];
            a.rec = (ulonglong2*)at(o_rec) + g.rec;
            a.halo = (Tagged4*)at(o_halo) + g.halo;
            a.xw = (float4*)at(o_xw) + g.xw;
        }
    pl->B.inst = (const RcgArgs*)at(o_inst);
    pl->B.off = (const int64_t*)at(o_off);
    pl->B.block = (const int2*)at(o_block);
    pl->B.group = (const RcgGroup*)at(o_group);
    pl->B.list = (const int*)at(o_list);
    pl->B.start = (ulonglong2*)at(o_start);
    pl->B.epoch = (unsigned*)at(o_epoch);
    pl->B.scal = (double*)at(o_scal);
    pl->B.flags = (int*)at(o_flags);
    std::vector<unsigned char> host(bytes - o_inst);
    auto put = [&](size_t o, const void* h, size_t n) { std::memcpy(host.data() + (o - o_inst), h, n); };
    put(o_inst, inst.data(), sizeof(RcgArgs) * N);
    put(o_off, off, sizeof(int64_t) * N);
    put(o_block, block.data(), sizeof(int2) * block.size());
    put(o_group, group.data(), sizeof(RcgGroup) * group.size());
    put(o_list, list.data(), sizeof(int) * list.size());
    st = nn_cuda_check(ctx, cudaMemcpyAsync(at(o_inst), host.data(), host.size(), cudaMemcpyHostToDevice, ctx->stream), "copy");
    if (st == NN_OK) st = batch_reset(pl, ctx->stream);
    int coop = 0, per_sm = 0;
    if (st == NN_OK)
        st = nn_cuda_check(ctx, cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device), "attribute");
    if (st == NN_OK)
        st = nn_cuda_check(ctx, cudaFuncSetAttribute(pl->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024),
                           "cudaFuncSetAttribute(k_rcg_batch)");
    if (st == NN_OK)
        st = nn_cuda_check(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pl->kernel, RT, pl->smem), "occupancy");
    if (st == NN_OK && (!coop || per_sm < 1)) st = NN_ERR_UNSUPPORTED;
    // solves may run on other streams, and the host arrays go
    const cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (st == NN_OK) st = nn_cuda_check(ctx, e, "nn_rcg_batch_create");
    if (st != NN_OK) {
        nn_rcg_batch_destroy(pl);
        return st;
    }
    *out = pl;
    return NN_OK;
}

nn_status nn_rcg_batch_begin(nn_rcg_batch* pl, const float* d_b, float* d_x, double rtol, int max_iter, cudaStream_t cs)
{
    nn_ctx* ctx = pl->ctx;
    pl->B.b = d_b;
    pl->B.x = d_x;
    pl->B.rtol2 = rtol * rtol;
    pl->B.max_iter = max_iter;
    void* args[] = {&pl->B};
    NN_CUDA(ctx, cudaLaunchCooperativeKernel(pl->kernel, dim3(pl->blocks), dim3(RT), args, pl->smem, cs));
    ctx->launches++;
    pl->B.seq += (uint32_t)pl->longest;
    return NN_OK;
}

// Per instance: iterations and outcome (1 converged).
nn_status nn_rcg_batch_finish(nn_rcg_batch* pl, cudaStream_t cs, int* iters, int* flags)
{
    nn_ctx* ctx = pl->ctx;
    std::vector<int> f(4 * (size_t)pl->n_inst);
    NN_CUDA(ctx, cudaMemcpyAsync(f.data(), pl->B.flags, sizeof(int) * f.size(), cudaMemcpyDeviceToHost, cs));
    NN_CUDA(ctx, cudaStreamSynchronize(cs));
    for (int b = 0; b < pl->n_inst; ++b) {
        if (f[4 * (size_t)b + 2]) {
            NN_TRY(batch_reset(pl, cs));
            NN_CUDA(ctx, cudaMemsetAsync(pl->B.flags, 0, sizeof(int) * f.size(), cs));
            NN_CUDA(ctx, cudaStreamSynchronize(cs));
            return nn_fail(ctx, NN_ERR_TIMEOUT, "k_rcg_batch: a block's wait for its neighbours gave up");
        }
        flags[b] = f[4 * (size_t)b];
        iters[b] = f[4 * (size_t)b + 1];
    }
    return NN_OK;
}
