// Reference-semantics primitives: the reference HH leapfrog step, the
// AtomicCoupling threshold/compaction/push, the network factory's in-degree
// and chunked lists, and the ParacrineModule (trilinear scatter/interpolation
// + Crank-Nicolson 27-point CG).  Each function cites the reference code whose
// behaviour it reproduces.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "nn_hh.cuh"
#include "nn_internal.cuh"
#include "nn_pair.cuh"

// =============================================================== leapfrog ==

extern "C" void nn_leapfrog_params_reference(nn_leapfrog_params* p, int variant)
{
    if (!p) return;
    // src/defines.cuh:87-102
    p->gna = 120.0f; p->ena = 55.0f; p->gk = 36.0f; p->ek = -72.0f; p->gl = 0.3f; p->el = -50.0f;
    p->Tmax = 1.0f; p->Vt = -20.0f; p->Kp = 3.0f; p->Ar = 5.0f; p->Ad = 0.18f;
    p->g_local = 0.1f; p->e_local = 0.0f; p->g_gaba = 0.1f; p->e_gaba = -70.0f;
    p->g_exc = 0.1f; p->e_exc = 0.0f;
    p->noise_mean = 3.0f; p->noise_intensity = 1.5f;
    if (variant == 1) {
        // src_wholebrain/ephys.cuh:56-61: grey AMPA only, zero-mean noise of intensity 2
        p->g_local = 0.1f; p->g_gaba = 0.0f; p->g_exc = 0.0f;
        p->noise_mean = 0.0f; p->noise_intensity = 2.0f;
    }
}

namespace {
// small blocks: a network of 15k neurons then spreads over most of the chip
constexpr int LF_THREADS = 64;

struct LFVars { float* v[NN_HH_NUM_VARS]; };

// Leapfrog_HH (src/ephys.cu:28-96), evaluated in the precision the
// reference's expressions have.  Its double literals (3.5, 0.1, 0.07, 0.125,
// 1.0) promote alpha_m, alpha_n, beta_h, the products 0.07 * e^x and
// 0.125 * e^x, and the output sigmoid to FP64, each rounded to float on
// assignment; exponentials of float arguments (alpha_h, beta_m, beta_n, the
// sigmoid's) are FP32 calls; the gate, synapse and membrane updates are FP32
// (Float = float, src/defines.cuh:50-55).  The expressions keep the
// reference's operand order, so each rounds as the reference's does.  The
// removable singularities of alpha_m (V = -35) and alpha_n (V = -50), 0/0 in
// the reference, take their limits (1 and 0.1) there.  V = -35 and V = -50
// are the only float inputs whose FP64 argument 3.5 + 0.1 V (or -5 - 0.1 V)
// lies within 1e-9 of zero, fused or not (the neighbouring floats give
// 3.8e-7), so the test is an FP32 compare, off the FP64 pipe that bounds
// this kernel.
__device__ __noinline__ float lf_rate_am(float V)
{
    if (V == -35.0f) return 1.0f;
    return (float)((3.5 + 0.1 * V) / (1 - exp(-3.5 - 0.1 * V)));
}

__device__ __noinline__ float lf_rate_an(float V)
{
    if (V == -50.0f) return 0.1f;
    return (float)((-0.5 - 0.01 * V) / (exp(-5 - 0.1 * V) - 1));
}

__device__ __noinline__ float lf_rate_bh(float V) { return (float)(1 / (exp(-3 - 0.1 * V) + 1)); }

// The same roundings without the FP64 pipe.  It issues one warp instruction
// in 16 cycles, and the five FP64 expressions of a neuron (three exponentials
// and four divisions among them) held the step at 181 us per million neurons (38 us now, 78 % issue-active).
// Here they are evaluated in pairs of floats to about 2^-43; where the result
// lies so near the midpoint of two floats (2^-39 relative) that this cannot
// say how FP64 rounds, and close to the two singularities, where the FP64
// expression itself cancels, the FP64 expression is evaluated after all
// (A. Ziv, "Fast evaluation of elementary mathematical functions with
// correctly rounded last bit", ACM TOMS 17, 1991).  All three exponentials
// are e^{-V/10} times a constant; that one is table-driven (P. T. P. Tang,
// "Table-driven implementation of the exponential function in IEEE
// floating-point arithmetic", ACM TOMS 15, 1989): 2^(j/32) sits in lane j of
// the warp and comes by shuffle, the remainder |s| <= ln 2 / 64 by its series.

// 2^(j/32) as pairs
__device__ const Pair lf_exp_table[32] = {
    {0x1p+0f, 0.0f}, {0x1.059b0ep+0f, -0x1.9d4f52p-25f}, {0x1.0b5586p+0f, 0x1.9f3122p-25f}, {0x1.11301ep+0f, -0x1.fdb496p-25f},
    {0x1.172b84p+0f, -0x1.c15742p-27f}, {0x1.1d4874p+0f, -0x1.d2e8cap-25f}, {0x1.2387a6p+0f, 0x1.ceac48p-25f}, {0x1.29e9ep+0f, -0x1.5c0424p-25f},
    {0x1.306fep+0f, 0x1.4636e2p-25f}, {0x1.371a74p+0f, -0x1.18aac6p-25f}, {0x1.3dea64p+0f, 0x1.824684p-25f}, {0x1.44e086p+0f, 0x1.8624b4p-30f},
    {0x1.4bfdaep+0f, -0x1.593abcp-25f}, {0x1.5342b6p+0f, -0x1.2c561p-25f}, {0x1.5ab07ep+0f, -0x1.5bd5ecp-27f}, {0x1.6247ecp+0f, -0x1.f8b55p-25f},
    {0x1.6a09e6p+0f, 0x1.9fcef4p-26f}, {0x1.71f75ep+0f, 0x1.1d8beep-25f}, {0x1.7a1148p+0f, -0x1.829fdp-25f}, {0x1.82589ap+0f, -0x1.accc7cp-26f},
    {0x1.8ace54p+0f, 0x1.15506ep-27f}, {0x1.93737cp+0f, -0x1.e64744p-25f}, {0x1.9c4918p+0f, 0x1.51f848p-27f}, {0x1.a5503cp+0f, -0x1.b83b54p-25f},
    {0x1.ae89fap+0f, -0x1.a94b14p-26f}, {0x1.b7f77p+0f, -0x1.a09438p-25f}, {0x1.c199bep+0f, -0x1.3d56b2p-27f}, {0x1.cb720ep+0f, -0x1.8837ccp-27f},
    {0x1.d5818ep+0f, -0x1.822dbcp-27f}, {0x1.dfc974p+0f, -0x1.908c94p-25f}, {0x1.ea4afap+0f, 0x1.52486cp-27f}, {0x1.f50766p+0f, -0x1.246ebp-26f}};

// e^{-V/10} with 0.1 as the double 0.1, |V| <= 400; all lanes of the warp.
// tab: lane j's table entry; x receives V/10.
__device__ __forceinline__ Pair lf_exp_tenth(float V, const Pair& tab, Pair& x)
{
    const float ph = __fmul_rn(0x1.99999ap-4f, V);
    x = pair_norm(ph, __fmaf_rn(-0x1.99999ap-30f, V, __fmaf_rn(0x1.99999ap-4f, V, -ph)));
    const float n = rintf(x.h * -0x1.715476p+5f);  // 32 / ln 2
    // s = -x - n ln2/32: the first 13 bits of ln2/32 make an exact product and
    // an exact difference, two more floats the rest
    const float a = __fmaf_rn(-n, 0x1.62ep-6f, -x.h);
    const float c = __fmul_rn(n, 0x1.0bfbe8p-20f), e = __fmaf_rn(n, 0x1.0bfbe8p-20f, -c);
    Pair s = pair_two_sum(a, -c);
    s = pair_norm(s.h, __fsub_rn(__fsub_rn(s.l, e), __fmaf_rn(n, 0x1.cf79acp-45f, x.l)));
    // e^s - 1 = s + s^2/2 + s^3 (1/6 + s/24 + s^2/120)
    const float h2 = __fmul_rn(s.h, s.h), l2 = __fmaf_rn(2.0f * s.h, s.l, __fmaf_rn(s.h, s.h, -h2));
    const float cub = h2 * s.h * (1.0f / 6.0f + s.h * (1.0f / 24.0f + s.h * (1.0f / 120.0f)));
    const Pair m = pair_add(s, Pair{0.5f * h2, __fadd_rn(0.5f * l2, cub)});
    const int k = (int)n;
    const Pair t{__shfl_sync(0xffffffffu, tab.h, k & 31), __shfl_sync(0xffffffffu, tab.l, k & 31)};
    const Pair r = pair_add(t, pair_mul(t, m));
    const float p2 = __int_as_float((127 + (k >> 5)) << 23);
    return {r.h * p2, r.l * p2};
}

// a / (1 - e^{-a}) = 1 + a/2 + a^2/12 - a^4/720 + a^6/30240 - ... for |a| < 0.35
__device__ __forceinline__ Pair lf_series(const Pair& a)
{
    const Pair z = pair_mul(a, a), z2 = pair_mul(z, z);
    const float y = z.h;
    const float rest =
        y * y * y * (1.0f / 30240.0f + y * (-1.0f / 1209600.0f + y * (1.0f / 47900160.0f + y * -5.28419014e-10f)));
    const Pair t = pair_add(pair_mul(z, Pair{0x1.555556p-4f, -0x1.555556p-29f}),    // 1/12
                            pair_mul(z2, Pair{-0x1.6c16c2p-10f, 0x1.27d27ep-35f}));  // -1/720
    const Pair r = pair_add(pair_add(Pair{1.0f, 0.0f}, Pair{0.5f * a.h, 0.5f * a.l}), t);
    return pair_norm(r.h, __fadd_rn(r.l, rest));
}

// Whether every value within 2^-39 (relative) of h + l rounds to h.
__device__ __forceinline__ bool lf_rounds(const Pair& r) { return __fmaf_rn(r.l, 1.0f + 0x1p-13f, r.h) == r.h; }

// alpha_m, alpha_n and beta_h of the reference's expressions (all lanes).
__device__ __forceinline__ void lf_rates(float V, const Pair& tab, float& am, float& an, float& bh)
{
    const bool in = fabsf(V) <= 400.0f;
    Pair x;
    const Pair e = lf_exp_tenth(in ? V : 0.0f, tab, x);
    const Pair e1 = pair_mul(e, Pair{0x1.eec102p-6f, -0x1.c6c026p-32f});  // e^{-3.5 - V/10}
    const Pair e2 = pair_mul(e, Pair{0x1.b993fep-8f, 0x1.aa6ec4p-41f});   // e^{-5 - V/10}
    const Pair e3 = pair_mul(e, Pair{0x1.97db0cp-5f, 0x1.99d616p-30f});   // e^{-3 - V/10}
    const Pair a1 = pair_add(Pair{3.5f, 0.0f}, x), a2 = pair_add(Pair{5.0f, 0.0f}, x);
    const Pair m = fabsf(a1.h) < 0.35f ? lf_series(a1)
                                       : pair_div(a1, pair_add(Pair{1.0f, 0.0f}, Pair{-e1.h, -e1.l}));
    // numerator 0.5 + 0.01 V with the double 0.01: a2/10 - 3.47e-19 V
    Pair n;
    if (fabsf(a2.h) < 0.35f) {
        const Pair f = lf_series(a2);
        n = pair_mul(f, Pair{0x1.99999ap-4f, -0x1.99999ap-30f});
        n = pair_norm(n.h, __fadd_rn(n.l, __fdividef(-3.46944695e-19f * V * f.h, a2.h)));
    } else {
        const float ph = __fmul_rn(0x1.47ae14p-7f, V);
        const Pair q = pair_norm(ph, __fmaf_rn(0x1.eb851ep-33f, V, __fmaf_rn(0x1.47ae14p-7f, V, -ph)));
        n = pair_div(pair_add(Pair{0.5f, 0.0f}, q), pair_add(Pair{1.0f, 0.0f}, Pair{-e2.h, -e2.l}));
    }
    const Pair h = pair_div(Pair{1.0f, 0.0f}, pair_add(e3, Pair{1.0f, 0.0f}));
    am = m.h;
    an = n.h;
    bh = h.h;
    if (!(in && lf_rounds(m) && fabsf(a1.h) > 0x1p-12f)) am = lf_rate_am(V);
    if (!(in && lf_rounds(n) && fabsf(a2.h) > 0x1p-12f)) an = lf_rate_an(V);
    if (!(in && lf_rounds(h))) bh = lf_rate_bh(V);
}

// (float)(0.07 * e) and (float)(Tmax / (1.0 + e)) of a float e >= 0
__device__ __noinline__ float lf_seven_fp64(float e) { return (float)(0.07 * e); }
__device__ __noinline__ float lf_sigmoid_fp64(float Tmax, float e) { return (float)(Tmax / (1.0 + e)); }
__device__ __forceinline__ float lf_seven(float e)
{
    const Pair r = pair_mulf(Pair{0x1.1eb852p-4f, -0x1.47ae14p-32f}, e);
    return e > 1e-25f && e < 1e30f && lf_rounds(r) ? r.h : lf_seven_fp64(e);
}
__device__ __forceinline__ float lf_sigmoid(float Tmax, float e)
{
    const Pair r = pair_div(Pair{Tmax, 0.0f}, pair_two_sum(1.0f, e));
    return e < 1e15f && fabsf(Tmax) > 1e-10f && fabsf(Tmax) < 1e10f && lf_rounds(r) ? r.h : lf_sigmoid_fp64(Tmax, e);
}

// One neuron's step (zi: its standard-normal noise draw; tab: the lane's entry
// of the exponential's table).  All lanes of the warp take part; those with
// store unset compute a neuron that is there and write nothing.
__device__ __forceinline__ void lf_neuron(const LFVars& s, int i, float timestep, const nn_leapfrog_params& p,
                                          float zi, const Pair& tab, bool store)
{
    {
        const float local_in = s.v[NN_HH_LOCAL_IN][i], local_num_in = s.v[NN_HH_LOCAL_COUNT][i];
        const float Iin = s.v[NN_HH_IIN][i], Inum_in = s.v[NN_HH_ICOUNT][i];
        const float Ein = s.v[NN_HH_EIN][i], Enum_in = s.v[NN_HH_ECOUNT][i];
        const float appcur = s.v[NN_HH_APPCUR][i];
        const float V = s.v[NN_HH_V][i], M = s.v[NN_HH_M][i], N = s.v[NN_HH_N][i], H = s.v[NN_HH_H][i];
        const float local_Y = s.v[NN_HH_LOCAL_Y][i], IY = s.v[NN_HH_IY][i], EY = s.v[NN_HH_EY][i];

        float Am, An, Bh;
        lf_rates(V, tab, Am, An, Bh);
        const float Ah = lf_seven(expf(-V / 20 - 3));
        const float Bm = 4 * expf(-(V + 60) / 18);
        const float Bn = 0.125f * expf(-(V + 60) / 80);  // a power of two: no rounding of its own

        const float new_M = (Am * timestep + (1 - timestep / 2 * (Am + Bm)) * M) / (timestep / 2 * (Am + Bm) + 1);
        const float new_N = (An * timestep + (1 - timestep / 2 * (An + Bn)) * N) / (timestep / 2 * (An + Bn) + 1);
        const float new_H = (Ah * timestep + (1 - timestep / 2 * (Ah + Bh)) * H) / (timestep / 2 * (Ah + Bh) + 1);

        const float Ar = p.Ar, Ad = p.Ad;
        const float local_T = local_num_in > 0 ? local_in / local_num_in : 0;
        const float new_local_Y = (Ar * local_T * timestep + (1 - timestep / 2 * (Ar * local_T + Ad)) * local_Y) /
                                  (timestep / 2 * (Ar * local_T + Ad) + 1);
        const float I_T = Inum_in > 0 ? Iin / Inum_in : 0;
        const float new_IY = (Ar * I_T * timestep + (1 - timestep / 2 * (Ar * I_T + Ad)) * IY) /
                             (timestep / 2 * (Ar * I_T + Ad) + 1);
        const float E_T = Enum_in > 0 ? Ein / Enum_in : 0;
        const float new_EY = (Ar * E_T * timestep + (1 - timestep / 2 * (Ar * E_T + Ad)) * EY) /
                             (timestep / 2 * (Ar * E_T + Ad) + 1);

        // G, E and the membrane update with every rounding explicit, in the
        // order and fusion the reference kernel has when nvcc builds it for
        // sm_103a (found by comparing the two kernels' outputs on the same
        // states: the reference forms E * dt inside a fused multiply-add on
        // top of the rounded (noise + I_app) * dt; left to the compiler, this
        // source fused the other product and differed by an ulp in 19 % of
        // the neurons).  The reference weights the local and excitatory
        // synapses by g_ampa and the inhibitory one by g_gaba; the whole-brain
        // variant sets them apart, hence g_local / g_exc.
        const float gna_m3h = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(p.gna, new_M), new_M), new_M), new_H);
        const float gk_n4 = __fmul_rn(p.gk, powf(new_N, 4));
        float G = __fadd_rn(__fadd_rn(gna_m3h, gk_n4), p.gl);
        G = __fadd_rn(G, __fmul_rn(p.g_local, new_local_Y));
        G = __fadd_rn(G, __fmul_rn(p.g_gaba, new_IY));
        G = __fadd_rn(G, __fmul_rn(p.g_exc, new_EY));
        float E = __fmaf_rn(gna_m3h, p.ena, __fmul_rn(gk_n4, p.ek));
        E = __fadd_rn(E, __fmul_rn(p.gl, p.el));
        E = __fadd_rn(E, __fmul_rn(__fmul_rn(p.g_local, new_local_Y), p.e_local));
        E = __fmaf_rn(__fmul_rn(p.g_gaba, new_IY), p.e_gaba, E);
        E = __fadd_rn(E, __fmul_rn(__fmul_rn(p.g_exc, new_EY), p.e_exc));

        const float white_noise = __fmaf_rn(p.noise_intensity, zi, p.noise_mean);
        const float half_dt = timestep / 2;
        float num = __fmaf_rn(E, timestep, __fmul_rn(__fadd_rn(white_noise, appcur), timestep));
        num = __fmaf_rn(__fmaf_rn(-half_dt, G, 1.0f), V, num);
        const float nV = __fdiv_rn(num, __fmaf_rn(half_dt, G, 1.0f));
        const float out = lf_sigmoid(p.Tmax, expf(-(nV - p.Vt) / p.Kp));
        if (!store) return;
        s.v[NN_HH_V][i] = nV;
        s.v[NN_HH_M][i] = new_M;
        s.v[NN_HH_N][i] = new_N;
        s.v[NN_HH_H][i] = new_H;
        s.v[NN_HH_LOCAL_Y][i] = new_local_Y;
        s.v[NN_HH_IY][i] = new_IY;
        s.v[NN_HH_EY][i] = new_EY;
        s.v[NN_HH_LOCAL_OUTPUT][i] = out;
        s.v[NN_HH_IOUTPUT][i] = out;
        s.v[NN_HH_EOUTPUT][i] = out;
    }
}

// A neuron per thread.  It draws its pair's two Box-Muller outputs and takes
// its own: the draw costs 6 % more instructions than a pair per thread would,
// and a network of 15k neurons has twice the warps to hide its latency with.
template <bool EXT_Z>
__global__ void __launch_bounds__(LF_THREADS) k_leapfrog(LFVars s, int n, float timestep, nn_leapfrog_params p,
                                                         uint64_t seed, uint64_t step, const float* __restrict__ z)
{
    const int lane = threadIdx.x & 31;
    const Pair tab = lf_exp_table[lane];
    const int first = blockIdx.x * blockDim.x + threadIdx.x - lane;
    // The step's kernels (this one, the coupling's two and the paracrine's) are
    // programmatic dependents of whatever is before them on the stream, which
    // hides their launches; the first noise needs no memory.  Ten steps of 14,638
    // neurons with a field solve: 289 -> 231 us; of a million 937 -> 861.
    nn_grid_dep_launch();
    const float z0 = EXT_Z ? 0.0f : nn_normal(seed, (uint32_t)min(first + lane, n - 1), step);
    nn_grid_dep_wait();
    // whole warps: lanes past the last neuron repeat it
    for (int i0 = first; i0 < n; i0 += gridDim.x * blockDim.x) {
        const int i = min(i0 + lane, n - 1);
        lf_neuron(s, i, timestep, p, EXT_Z ? z[i] : i0 == first ? z0 : nn_normal(seed, (uint32_t)i, step), tab,
                  i0 + lane < n);
    }
}

nn_status leapfrog_launch(nn_ctx* ctx, float* const* vars, int n, float dt, const nn_leapfrog_params* p,
                          uint64_t seed, uint64_t step, const float* d_z, const char* what)
{
    if (!ctx || !vars || !p || n < 0) return nn_fail(ctx, NN_ERR_INVALID_ARG, "%s: bad argument", what);
    if (n == 0) return NN_OK;
    LFVars s;
    for (int q = 0; q < NN_HH_NUM_VARS; ++q) {
        if (!vars[q]) return nn_fail(ctx, NN_ERR_INVALID_ARG, "%s: sim_vars[%d] is NULL", what, q);
        s.v[q] = vars[q];
    }
    const int grid = nn_grid_for(ctx, n, LF_THREADS, 64);
    NN_CUDA(ctx, nn_launch_pdl(d_z ? k_leapfrog<true> : k_leapfrog<false>, dim3(grid), dim3(LF_THREADS), 0, ctx->stream, s,
                               n, dt, *p, seed, step, d_z));
    NN_CHECK_LAUNCH(ctx, "k_leapfrog");
    return NN_OK;
}
}  // namespace

extern "C" nn_status nn_hh_leapfrog_step(nn_ctx* ctx, float* const* vars, int n, float dt,
                                         const nn_leapfrog_params* p, uint64_t seed, uint64_t step)
{
    return leapfrog_launch(ctx, vars, n, dt, p, seed, step, nullptr, "nn_hh_leapfrog_step");
}

extern "C" nn_status nn_hh_leapfrog_step_z(nn_ctx* ctx, float* const* vars, int n, float dt,
                                           const nn_leapfrog_params* p, const float* d_z)
{
    if (!d_z) return nn_fail(ctx, NN_ERR_INVALID_ARG, "nn_hh_leapfrog_step_z: d_z is NULL");
    return leapfrog_launch(ctx, vars, n, dt, p, 0, 0, d_z, "nn_hh_leapfrog_step_z");
}

// =============================================================== coupling ==

struct nn_coupling {
    nn_ctx* ctx = nullptr;
    int n = 0;
    int* firing = nullptr;       // n entries; first count ascending
    int* count = nullptr;        // device int
    int64_t* block_counts = nullptr;
    int* sub_before = nullptr;   // per sub-tile: firing neurons of its tile before it (behind block_counts)
    int nblocks = 0;
};

namespace {
constexpr int CMP_THREADS = 256;
constexpr int CMP_ITEMS = 8;
constexpr int CMP_TILE = CMP_THREADS * CMP_ITEMS;

// CheckFiringOperator (src/coupling.cu:103-109)
__device__ __forceinline__ int fires(float out) { return out > 0.1f ? 1 : 0; }

__global__ void __launch_bounds__(CMP_THREADS) k_cmp_count(const float* out, int n, int64_t* block_counts)
{
    const int base = blockIdx.x * CMP_TILE + threadIdx.x * CMP_ITEMS;
    int c = 0;
#pragma unroll
    for (int q = 0; q < CMP_ITEMS; ++q)
        if (base + q < n) c += fires(out[base + q]);
    __shared__ int tot;
    if (threadIdx.x == 0) tot = 0;
    __syncthreads();
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&tot, c);
    __syncthreads();
    if (threadIdx.x == 0) block_counts[blockIdx.x] = tot;
}

// single block: exclusive scan of the block counts, total -> *count
__global__ void __launch_bounds__(1024) k_cmp_scan(int64_t* bc, int nb, int* count)
{
    __shared__ int64_t carry_s;
    __shared__ int64_t warp_tot[32];
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (int off = 0; off < nb; off += 1024) {
        const int i = off + threadIdx.x;
        int64_t v = i < nb ? bc[i] : 0;
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        int64_t inc = v;
        for (int o = 1; o < 32; o <<= 1) {
            int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) warp_tot[w] = inc;
        __syncthreads();
        if (w == 0) {
            int64_t t = warp_tot[lane];
            for (int o = 1; o < 32; o <<= 1) {
                int64_t u = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += u;
            }
            warp_tot[lane] = t;
        }
        __syncthreads();
        const int64_t ex = carry_s + (w ? warp_tot[w - 1] : 0) + inc - v;
        if (i < nb) bc[i] = ex;
        __syncthreads();
        if (threadIdx.x == 0) carry_s += warp_tot[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) *count = (int)carry_s;
}

__global__ void __launch_bounds__(CMP_THREADS) k_cmp_write(const float* out, int n, const int64_t* block_off,
                                                           int* list)
{
    const int base = blockIdx.x * CMP_TILE + threadIdx.x * CMP_ITEMS;
    int f[CMP_ITEMS];
    int c = 0;
#pragma unroll
    for (int q = 0; q < CMP_ITEMS; ++q) {
        f[q] = base + q < n ? fires(out[base + q]) : 0;
        c += f[q];
    }
    // block exclusive scan of c
    __shared__ int wt[CMP_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = c;
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wt[w] = inc;
    __syncthreads();
    int wbase = 0;
    for (int q = 0; q < w; ++q) wbase += wt[q];
    int pos = (int)block_off[blockIdx.x] + wbase + inc - c;
#pragma unroll
    for (int q = 0; q < CMP_ITEMS; ++q)
        if (f[q]) list[pos++] = base + q;
}

// Threshold count of each tile with the tile's inputs zeroed (the first of
// the two launches of nn_coupling_run), and of the tile's sub-tiles the firing
// neurons before them, so that the second launch can use a block per sub-tile
// without summing the counts of thousands of blocks.
constexpr int CMP_SUB = 128;
constexpr int CMP_SUBS = CMP_TILE / CMP_SUB;

__global__ void __launch_bounds__(CMP_THREADS) k_cmp_count_zero(const float* out, int n, int64_t* block_counts,
                                                                int* sub_before, float* inputs)
{
    __shared__ int cnt[CMP_TILE / 32];  // firing neurons of 32 consecutive neurons
    nn_grid_dep_launch();
    nn_grid_dep_wait();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < CMP_ITEMS; ++q) {
        const int i = blockIdx.x * CMP_TILE + q * CMP_THREADS + threadIdx.x;
        const int f = i < n ? fires(out[i]) : 0;
        if (i < n) inputs[i] = 0.0f;
        const unsigned b = __ballot_sync(0xffffffffu, f);
        if (lane == 0) cnt[q * (CMP_THREADS / 32) + w] = __popc(b);
    }
    __syncthreads();
    if (w == 0) {
        constexpr int PER = CMP_SUB / 32;
        int c = 0;
        if (lane < CMP_SUBS)
            for (int q = 0; q < PER; ++q) c += cnt[lane * PER + q];
        int inc = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane < CMP_SUBS) sub_before[blockIdx.x * CMP_SUBS + lane] = inc - c;
        if (lane == 31) block_counts[blockIdx.x] = inc;
    }
}

// The second launch, a block for per_block consecutive stretches of SUB neurons:
// the stretch's offset in the ascending firing list (the earlier tiles' counts
// and the tile's own before it; later stretches go on from there), its entries
// written, the total stored by the last one, and its firing neurons scattered
// (signal_spikes_kernel), a warp per firing neuron with four targets per lane
// loaded before their reductions.
// Short stretches spread the scatter: with 2,048 neurons a block a network of
// 14,638 had 8 blocks whose warps scattered up to a dozen rows each in turn, 38
// us; with 128 115 blocks and 7.6 us.  Long ones save the fixed cost of a block.
// us of the two launches at 2 % firing with 10 targets / 50 % with 100, SUB = 128
// and 512: 300k neurons 8.4 / 82 and 7.6 / 119, 1M 18 / 240 and 11 / 254, 4M 60 /
// 912 and 28 / 931 (2,048: 39 / 1002).  So 512 from five waves of blocks of 128
// on.  The offset's sum costs more than the stretch from some 64 blocks an SM on:
// 16M neurons 152 us with a stretch a block, 133 with three.
template <int SUB>
__global__ void __launch_bounds__(CMP_THREADS) k_cmp_write_push(const float* out, int n, const int64_t* block_counts,
                                                                const int* sub_before, int per_block, int* list, int* count,
                                                                const int* indices, const int* offsets, float* inputs,
                                                                int signal_mode)
{
    __shared__ int64_t red[CMP_THREADS / 32];
    __shared__ int s_list[SUB];
    __shared__ int wt[SUB / 32];
    nn_grid_dep_launch();
    nn_grid_dep_wait();
    constexpr int ITEMS = SUB < CMP_THREADS ? 1 : SUB / CMP_THREADS, WARPS = CMP_THREADS / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int subs = (n - 1) / SUB + 1;
    int64_t boff = 0;
    const int s0 = blockIdx.x * (SUB == CMP_SUB ? 1 : per_block);
    for (int s = s0; s < (SUB == CMP_SUB ? s0 + 1 : min(s0 + per_block, subs)); ++s) {  // (short stretches: one a block)
        bool f[ITEMS];
        unsigned b[ITEMS];
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            const int i = s * SUB + q * CMP_THREADS + (int)threadIdx.x;
            f[q] = threadIdx.x < SUB && i < n && fires(out[i]);
            b[q] = __ballot_sync(0xffffffffu, f[q]);
            if (q * WARPS + w < SUB / 32 && lane == 0) wt[q * WARPS + w] = __popc(b[q]);
        }
        if (s == s0) {
            const int tile = (int)((int64_t)s * SUB / CMP_TILE);
            int64_t acc = 0;
            for (int q = threadIdx.x; q < tile; q += CMP_THREADS) acc += block_counts[q];
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) red[w] = acc;
            __syncthreads();
            boff = sub_before[s * (SUB / CMP_SUB)];
            for (int q = 0; q < WARPS; ++q) boff += red[q];
        } else {
            __syncthreads();
        }
        int nf = 0, before[ITEMS] = {};
#pragma unroll
        for (int q = 0; q < SUB / 32; ++q) {
#pragma unroll
            for (int r = 0; r < ITEMS; ++r)
                if (q < r * WARPS + w) before[r] += wt[q];
            nf += wt[q];
        }
        if (s == subs - 1 && threadIdx.x == 0) *count = (int)(boff + nf);
#pragma unroll
        for (int q = 0; q < ITEMS; ++q)
            if (f[q]) {
                const int pos = before[q] + __popc(b[q] & ((1u << lane) - 1u)), i = s * SUB + q * CMP_THREADS + (int)threadIdx.x;
                list[boff + pos] = i;
                s_list[pos] = i;
            }
        boff += nf;
        __syncthreads();
        for (int k = w; k < nf; k += CMP_THREADS / 32) {
            const int pre = s_list[k];
            const float sig = signal_mode ? out[pre] : 1.0f;
            const int beg = offsets[pre], end = offsets[pre + 1];
            for (int e0 = beg + lane; e0 < end; e0 += 128) {
                int post[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) post[u] = e0 + 32 * u < end ? indices[e0 + 32 * u] : -1;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if ((unsigned)post[u] < (unsigned)n) atomicAdd(inputs + post[u], sig);
            }
        }
        if (SUB != CMP_SUB) __syncthreads();
    }
}

// signal_spikes_kernel (src/coupling.cu:34-48; src_wholebrain/coupling.cu:12-33),
// a warp per firing presynaptic neuron with the lanes over its targets.
__global__ void __launch_bounds__(256) k_push_ref(const int* list, const int* count, const int* indices,
                                                  const int* offsets, float* inputs, const float* outputs,
                                                  int signal_mode, int n, int target_base)
{
    const int lane = threadIdx.x & 31;
    const int nf = *count;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int f = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); f < nf; f += warps) {
        const int pre = list[f];
        const float sig = signal_mode ? outputs[pre] : 1.0f;
        const int beg = offsets[pre], end = offsets[pre + 1];
        for (int e = beg + lane; e < end; e += 32) {
            const int post = target_base + indices[e];
            if ((unsigned)post < (unsigned)n) atomicAdd(inputs + post, sig);
        }
    }
}
}  // namespace

extern "C" nn_status nn_coupling_create(nn_ctx* ctx, int n, nn_coupling** out)
{
    if (!ctx || !out || n < 0) return nn_fail(ctx, NN_ERR_INVALID_ARG, "nn_coupling_create: bad argument");
    nn_coupling* c = new nn_coupling();
    c->ctx = ctx;
    nn_ctx_retain(ctx);
    c->n = n;
    c->nblocks = (n + CMP_TILE - 1) / CMP_TILE;
    if (c->nblocks < 1) c->nblocks = 1;
    nn_status st = nn_alloc(ctx, &c->firing, (size_t)(n > 0 ? n : 1));
    if (st == NN_OK) st = nn_alloc(ctx, &c->count, 1);
    if (st == NN_OK) st = nn_alloc(ctx, &c->block_counts, (size_t)c->nblocks * (1 + CMP_SUBS / 2));
    if (st == NN_OK) c->sub_before = reinterpret_cast<int*>(c->block_counts + c->nblocks);
    if (st != NN_OK) {
        nn_coupling_destroy(c);
        return st;
    }
    // firing_neurons(N_, 0) (src/coupling.cu:5-8 of the coupling constructor)
    cudaMemsetAsync(c->firing, 0, sizeof(int) * (size_t)(n > 0 ? n : 1), ctx->stream);
    cudaMemsetAsync(c->count, 0, sizeof(int), ctx->stream);
    *out = c;
    return nn_cuda_check(ctx, cudaGetLastError(), "nn_coupling_create");
}

extern "C" nn_status nn_coupling_destroy(nn_coupling* c)
{
    if (!c) return NN_OK;
    if (c->ctx) cudaStreamSynchronize(c->ctx->stream);
    nn_release(c->firing);
    nn_release(c->count);
    nn_release(c->block_counts);
    nn_ctx* ctx = c->ctx;
    delete c;
    nn_ctx_release(ctx);
    return NN_OK;
}

extern "C" const int* nn_coupling_firing_list(const nn_coupling* c) { return c ? c->firing : nullptr; }
extern "C" const int* nn_coupling_firing_count(const nn_coupling* c) { return c ? c->count : nullptr; }

static nn_status coupling_compact(nn_coupling* c, float* d_inputs, const float* d_outputs)
{
    nn_ctx* ctx = c->ctx;
    NN_CUDA(ctx, cudaMemsetAsync(d_inputs, 0, sizeof(float) * (size_t)c->n, ctx->stream));
    k_cmp_count<<<c->nblocks, CMP_THREADS, 0, ctx->stream>>>(d_outputs, c->n, c->block_counts);
    NN_CHECK_LAUNCH(ctx, "k_cmp_count");
    k_cmp_scan<<<1, 1024, 0, ctx->stream>>>(c->block_counts, c->nblocks, c->count);
    NN_CHECK_LAUNCH(ctx, "k_cmp_scan");
    k_cmp_write<<<c->nblocks, CMP_THREADS, 0, ctx->stream>>>(d_outputs, c->n, c->block_counts, c->firing);
    NN_CHECK_LAUNCH(ctx, "k_cmp_write");
    return NN_OK;
}

static nn_status coupling_readback(nn_coupling* c, int* num_firing)
{
    if (!num_firing) return NN_OK;
    NN_CUDA(c->ctx, cudaMemcpyAsync(num_firing, c->count, sizeof(int), cudaMemcpyDeviceToHost, c->ctx->stream));
    NN_CUDA(c->ctx, cudaStreamSynchronize(c->ctx->stream));
    return NN_OK;
}

extern "C" nn_status nn_coupling_run(nn_coupling* c, const int* d_indices, const int* d_offsets, float* d_inputs,
                                     const float* d_outputs, int signal_mode, int* num_firing)
{
    if (!c || !d_offsets || !d_inputs || !d_outputs) return nn_fail(c ? c->ctx : nullptr, NN_ERR_INVALID_ARG, "nn_coupling_run: bad argument");
    if (c->n == 0) { if (num_firing) *num_firing = 0; return NN_OK; }
    nn_ctx* ctx = c->ctx;
    // two launches: threshold counts with the inputs zeroed, then the ordered
    // list, the count and the scatter
    NN_CUDA(ctx, nn_launch_pdl(k_cmp_count_zero, dim3(c->nblocks), dim3(CMP_THREADS), 0, ctx->stream, d_outputs, c->n,
                               c->block_counts, c->sub_before, d_inputs));
    NN_CHECK_LAUNCH(ctx, "k_cmp_count_zero");
    const bool many = c->n > 5 * 8 * ctx->num_sms * CMP_SUB;
    const int subs = (c->n - 1) / (many ? 512 : CMP_SUB) + 1, per_block = std::max(1, subs / (64 * ctx->num_sms));
    NN_CUDA(ctx, nn_launch_pdl(many ? k_cmp_write_push<512> : k_cmp_write_push<CMP_SUB>, dim3((subs - 1) / per_block + 1),
                               dim3(CMP_THREADS), 0, ctx->stream, d_outputs, c->n, c->block_counts, c->sub_before,
                               per_block, c->firing, c->count, d_indices, d_offsets, d_inputs, signal_mode));
    NN_CHECK_LAUNCH(ctx, "k_cmp_write_push");
    return coupling_readback(c, num_firing);
}

extern "C" nn_status nn_coupling_run_chunked(nn_coupling* c, int nchunks, int n_per_chunk,
                                             const int* const* d_chunk_indices, const int* const* d_chunk_offsets,
                                             float* d_inputs, const float* d_outputs, int* num_firing)
{
    if (!c || nchunks <= 0 || n_per_chunk <= 0 || !d_chunk_indices || !d_chunk_offsets || !d_inputs || !d_outputs)
        return nn_fail(c ? c->ctx : nullptr, NN_ERR_INVALID_ARG, "nn_coupling_run_chunked: bad argument");
    if (c->n == 0) { if (num_firing) *num_firing = 0; return NN_OK; }
    nn_ctx* ctx = c->ctx;
    NN_TRY(coupling_compact(c, d_inputs, d_outputs));
    for (int ch = 0; ch < nchunks; ++ch) {
        k_push_ref<<<nn_grid_for(ctx, (int64_t)c->n * 32, 256, 4), 256, 0, ctx->stream>>>(
            c->firing, c->count, d_chunk_indices[ch], d_chunk_offsets[ch], d_inputs, d_outputs, NN_SIGNAL_COUNT, c->n,
            ch * n_per_chunk);
        NN_CHECK_LAUNCH(ctx, "k_push_ref(chunk)");
    }
    return coupling_readback(c, num_firing);
}

// ======================================================== network factory ==

namespace {
uint32_t minstd_next(uint32_t& s)
{
    s = (uint32_t)(((uint64_t)s * 16807u) % 2147483647u);
    return s;
}

// libstdc++ uniform_int_distribution<int>(a, b) over minstd_rand0 ([1, 2^31-2]):
// downscaling by rejection (scaling = range / (b - a + 1)).
int uniform_int(uint32_t& s, int a, int b)
{
    const uint64_t urngrange = 2147483646u - 1u;
    const uint64_t urange = (uint64_t)((int64_t)b - (int64_t)a);
    uint64_t ret;
    if (urngrange > urange) {
        const uint64_t uerange = urange + 1, scaling = urngrange / uerange, past = uerange * scaling;
        do ret = (uint64_t)minstd_next(s) - 1u;
        while (ret >= past);
        ret /= scaling;
    } else {
        ret = (uint64_t)minstd_next(s) - 1u;
    }
    return (int)(ret + (uint64_t)(int64_t)a);
}
}  // namespace

extern "C" nn_status nn_net_uniform_random(int n, int ncouple, uint32_t* engine_state, int* h_indices, int* h_offsets)
{
    // UniformRandomNetwork::Generate (src/network_factory.cu:96-131).  The
    // reference loops forever when ncouple > n; that is rejected here.
    if (n <= 0 || ncouple < 0 || ncouple > n || !engine_state || !h_offsets || (ncouple && !h_indices))
        return NN_ERR_INVALID_ARG;
    std::vector<char> used((size_t)n, 0);
    for (int i = 0; i < n; ++i) {
        int* row = h_indices + (int64_t)i * ncouple;
        for (int j = 0; j < ncouple; ++j) {
            int d;
            do d = uniform_int(*engine_state, 0, n - 1);
            while (used[(size_t)d]);
            row[j] = d;
            used[(size_t)d] = 1;
        }
        for (int j = 0; j < ncouple; ++j) used[(size_t)row[j]] = 0;
        h_offsets[i] = i * ncouple;
    }
    h_offsets[n] = n * ncouple;
    return NN_OK;
}

namespace {
__global__ void k_tcount(const int* idx, int64_t nnz, int n, float* tcount)
{
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nnz; e += (int64_t)gridDim.x * blockDim.x) {
        const int t = idx[e];
        if ((unsigned)t < (unsigned)n) atomicAdd(tcount + t, 1.0f);
    }
}

constexpr int MAX_CHUNKS = 64;
struct ChunkPtrs { int* p[MAX_CHUNKS]; };

// per row and chunk: number of targets in the chunk; written at [c][i + 1]
__global__ void k_chunk_count(const int* idx, const int* off, int n, int nchunks, int npc, int64_t* cnt)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        for (int c = 0; c < nchunks; ++c) cnt[(int64_t)c * (n + 1) + i] = 0;
        for (int e = off[i]; e < off[i + 1]; ++e) {
            const int c = idx[e] / npc;
            if (c >= 0 && c < nchunks) cnt[(int64_t)c * (n + 1) + i] += 1;
        }
    }
}

__global__ void k_chunk_fill(const int* idx, const int* off, int n, int nchunks, int npc, const int64_t* pos,
                             ChunkPtrs out_idx, ChunkPtrs out_off)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        int64_t cur[MAX_CHUNKS];
        for (int c = 0; c < nchunks; ++c) {
            cur[c] = pos[(int64_t)c * (n + 1) + i];
            out_off.p[c][i] = (int)cur[c];
        }
        if (i == n) continue;
        for (int e = off[i]; e < off[i + 1]; ++e) {
            const int t = idx[e];
            const int c = t / npc;
            if (c >= 0 && c < nchunks) out_idx.p[c][cur[c]++] = t % npc;
        }
    }
}
}  // namespace

extern "C" nn_status nn_net_tcount(nn_ctx* ctx, const int* d_indices, int64_t nnz, int n, float* d_tcount)
{
    // Tcount loop of Network::ToAdjacencyList (src/network_factory.cu:19-22)
    if (!ctx || n < 0 || nnz < 0 || (nnz && !d_indices) || (n && !d_tcount))
        return nn_fail(ctx, NN_ERR_INVALID_ARG, "nn_net_tcount: bad argument");
    if (n == 0) return NN_OK;
    NN_CUDA(ctx, cudaMemsetAsync(d_tcount, 0, sizeof(float) * (size_t)n, ctx->stream));
    if (nnz > 0) {
        k_tcount<<<nn_grid_for(ctx, nnz, 256, 16), 256, 0, ctx->stream>>>(d_indices, nnz, n, d_tcount);
        NN_CHECK_LAUNCH(ctx, "k_tcount");
    }
    return NN_OK;
}

extern "C" nn_status nn_net_to_chunked(nn_ctx* ctx, const int* d_indices, const int* d_offsets, int n, int nchunks,
                                       int n_per_chunk, int* const* d_chunk_indices, int* const* d_chunk_offsets,
                                       int64_t* chunk_nnz)
{
    // Network::ToChunkedAdjacencyList (src/network_factory.cu:29-85)
    if (!ctx || n <= 0 || nchunks <= 0 || nchunks > MAX_CHUNKS || n_per_chunk <= 0 || !d_offsets ||
        !d_chunk_indices || !d_chunk_offsets || !chunk_nnz)
        return nn_fail(ctx, NN_ERR_INVALID_ARG, "nn_net_to_chunked: bad argument");
    int64_t* cnt = nullptr;
    int64_t* pos = nullptr;
    const size_t stride = (size_t)n + 1;
    NN_TRY(nn_alloc(ctx, &cnt, stride * nchunks));
    NN_TRY(nn_alloc(ctx, &pos, stride * nchunks));
    k_chunk_count<<<nn_grid_for(ctx, n, 256, 16), 256, 0, ctx->stream>>>(d_indices, d_offsets, n, nchunks, n_per_chunk,
                                                                          cnt);
    NN_CHECK_LAUNCH(ctx, "k_chunk_count");
    for (int c = 0; c < nchunks; ++c) {
        NN_CUDA(ctx, cudaMemsetAsync(cnt + c * stride + n, 0, sizeof(int64_t), ctx->stream));
        NN_TRY(nn_scan_exclusive_i64(ctx, cnt + c * stride, pos + c * stride, (int64_t)stride));
    }
    ChunkPtrs oi, oo;
    for (int c = 0; c < nchunks; ++c) {
        oi.p[c] = d_chunk_indices[c];
        oo.p[c] = d_chunk_offsets[c];
    }
    k_chunk_fill<<<nn_grid_for(ctx, (int64_t)n + 1, 128, 16), 128, 0, ctx->stream>>>(d_indices, d_offsets, n, nchunks,
                                                                                     n_per_chunk, pos, oi, oo);
    NN_CHECK_LAUNCH(ctx, "k_chunk_fill");
    for (int c = 0; c < nchunks; ++c)
        NN_CUDA(ctx, cudaMemcpyAsync(&chunk_nnz[c], pos + c * stride + n, sizeof(int64_t), cudaMemcpyDeviceToHost,
                                     ctx->stream));
    NN_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    cudaFree(cnt);
    cudaFree(pos);
    return NN_OK;
}

// ============================================================== paracrine ==

struct nn_paracrine {
    nn_ctx* ctx = nullptr;
    nn_paracrine_ref_params p{};
    int n = 0;
    int64_t G = 0;
    int* idx8 = nullptr;
    float* w8 = nullptr;
    float* grids = nullptr;      // the allocation of the grids that follow
    float* u = nullptr;          // density
    float* Ax = nullptr;         // scatter accumulator
    float *un = nullptr, *x = nullptr, *b = nullptr, *r = nullptr, *p0 = nullptr, *p1 = nullptr, *Ap = nullptr;
    float* at_neurons = nullptr;    // density_at_neurons
    float* generated = nullptr;     // density_generated_at_neurons
    float* g_out = nullptr;         // d_g_paracrine (caller's)
    double* scal = nullptr;         // [0]=rr [1]=pAp [2]=rr_new
    double* partials = nullptr;     // [2][nparts]
    unsigned int* bar = nullptr;    // grid barrier of k_cn_solve
    int* done = nullptr;            // [0] outcome [1] iterations
    int* h_gave_up = nullptr;       // pinned, set by k_cn_solve: a wait gave up; cleared when reported
    int polls = 0;                  // limit of its waits
    int nparts = 0;                 // blocks of k_cn_solve
};

extern "C" void nn_paracrine_ref_params_default(nn_paracrine_ref_params* p)
{
    if (!p) return;
    // the SCN run of diekman_benchmark (src/main.cu:525) with its 32^3 grid
    p->nx = p->ny = p->nz = 32;
    p->h = 1.0f;
    p->D = 2e-5f;
    p->decay = 3e-4f;
    p->par_dt = 100.0f * 0.4f;
    p->coup_strength = 0.5f;
    p->max_iter = 20;
    p->abs_tol = 1e-6f;
    p->quirk_rhs = 1;
    p->quirk_firing_list = 1;
}

namespace {
struct Stencil27 { float k[27]; };

// Trilinear weights (src/paracrine.cu:136-270), written per neuron in the
// reference's corner order (:189-195) with the same float arithmetic.
__global__ void k_trilinear(int n, const float* x, const float* y, const float* z, int nx, int ny, int nz, float h,
                            int* idx8, float* w8)
{
    const float Lx = __fmul_rn((float)(nx - 1), h), Ly = __fmul_rn((float)(ny - 1), h), Lz = __fmul_rn((float)(nz - 1), h);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float xr = __fadd_rn(__fdiv_rn(x[i], Lx), 0.5f);
        const float yr = __fadd_rn(__fdiv_rn(y[i], Ly), 0.5f);
        const float zr = __fadd_rn(__fdiv_rn(z[i], Lz), 0.5f);
        const float sx = __fmul_rn((float)(nx - 1), xr), sy = __fmul_rn((float)(ny - 1), yr), sz = __fmul_rn((float)(nz - 1), zr);
        const int m = (int)sx, q = (int)sy, pz = (int)sz;
        const float fx = __fsub_rn(sx, (float)m), fy = __fsub_rn(sy, (float)q), fz = __fsub_rn(sz, (float)pz);
        const int base = m + q * nx + pz * nx * ny;
        const float kx0 = __fsub_rn(1.0f, fx), ky0 = __fsub_rn(1.0f, fy), kz0 = __fsub_rn(1.0f, fz);
        const float kx1 = __fsub_rn(1.0f, kx0), ky1 = __fsub_rn(1.0f, ky0), kz1 = __fsub_rn(1.0f, kz0);
        const float xy[4] = {__fmul_rn(kx0, ky0), __fmul_rn(kx1, ky0), __fmul_rn(kx0, ky1), __fmul_rn(kx1, ky1)};
        const int off[8] = {0, 1, nx, nx + 1, nx * ny, nx * ny + 1, nx * ny + nx, nx * ny + nx + 1};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            w8[8 * (int64_t)i + c] = __fmul_rn(xy[c], kz0);
            w8[8 * (int64_t)i + c + 4] = __fmul_rn(xy[c], kz1);
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) idx8[8 * (int64_t)i + c] = base + off[c];
    }
}

// scatter_to_grid (src/paracrine.cu:276-287): grid += G^T s
__global__ void k_scatter(int n, const int* idx8, const float* w8, const float* s, float* grid, int64_t G)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v = s[i];
        if (v == 0.0f) continue;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int g = idx8[8 * (int64_t)i + c];
            if ((uint64_t)g < (uint64_t)G) atomicAdd(grid + g, w8[8 * (int64_t)i + c] * v);
        }
    }
}

// interpolate_at_location (src/paracrine.cu:288-296)
__global__ void k_interp(int n, const int* idx8, const float* w8, const float* grid, int64_t G, float* out, float* out2)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float acc = 0.0f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int g = idx8[8 * (int64_t)i + c];
            if ((uint64_t)g < (uint64_t)G) acc += w8[8 * (int64_t)i + c] * grid[g];
        }
        out[i] = acc;
        if (out2) out2[i] = acc;
    }
}

// update_on_fine_timescale (src/paracrine.cuh:246-253)
__global__ void k_fine(int n, const int* list, const int* count, float* gen, float coup, int quirk)
{
    nn_grid_dep_launch();
    nn_grid_dep_wait();
    if (quirk) {
        // transform_if with the compacted index buffer as the stencil
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            if (list[i] != 0) gen[i] += coup;
    } else {
        const int nf = *count;
        for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) gen[list[f]] += coup;
    }
}

// The whole Crank-Nicolson solve (update_density, src/paracrine.cu:63-134) in
// one cooperative launch: density += deposits, right-hand side and initial
// guess from its Laplacian, up to max_iter CG iterations, commit.  As separate
// launches it was 106 kernels of 2.6-4 us each whatever the iteration count
// (about 4 are needed); here an iteration is two passes over the block's cells
// (vectors in L2) and two grid barriers.  The direction p = r + beta p is
// formed at the 27 neighbours as they are read (p alternates between two
// buffers), which saves a third barrier.
//
// Barrier: a counter that every block adds to, behind a fence; each block's
// first thread polls it (bounded), and its second fence lets the block's plain
// loads, L1 included, see what the others wrote.  Sums: FP64 per thread, block
// partials, added by every block in the same order after the barrier.
//
// Large grids are bound by the latency of the 27 x 2 loads a cell, small ones by
// the barriers, whose cost grows with the blocks.  us a solve by blocks a SM, 1 /
// 2 / 3: 48^3 83 / 93 / 93, 80^3 173 / 156 / 170, 100^3 246 / 204 / 218, 150^3
// 698 / 464 / 450, 300^3 6549 / 3611 / 3005 (with loads past L1 and one block
// 10190, as separate launches 4998).
constexpr int CN_THREADS = 512;
constexpr int CN_POLLS = 1 << 22;  // some seconds (NN_CN_POLLS sets another limit)

// Blocks a SM: by the cells of a thread at one.
int cn_blocks_per_sm(const nn_ctx* ctx, int64_t G)
{
    const int64_t cells = G / ((int64_t)ctx->num_sms * CN_THREADS);
    return cells < 5 ? 1 : cells < 25 ? 2 : 3;
}

struct CnArgs {
    int nx, ny, nz, max_iter;
    int64_t G;
    Stencil27 L, A;
    float a, bb, c, d;         // x0 = a u + bb lap, b = c u + d lap
    float tol;
    const float* dep;          // deposits
    float *u, *un, *x, *b, *r, *p0, *p1, *Ap;
    double* scal;              // out: [0] rr of the last direction [1] pAp [2] rr
    double* partials;          // [2][blocks]
    unsigned* bar;
    int* done;                 // out: [0] 1 converged, 2 nothing to do  [1] iterations
    int* gave_up;              // out (host memory): a wait gave up
    int polls;
};

template <class I>
__global__ void __launch_bounds__(CN_THREADS) k_cn_solve(CnArgs q)
{
    __shared__ double ws[CN_THREADS / 32];
    __shared__ double total;
    __shared__ int fail;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const I stride = (I)gridDim.x * CN_THREADS, c0 = (I)blockIdx.x * CN_THREADS + tid, G = (I)q.G;
    unsigned phase = 0;
    if (tid == 0) fail = 0;
    __syncthreads();
    // grid barrier; with sum set, the grid total of v in `total`
    auto barrier = [&](bool sum, double v) {
        double* part = q.partials + (phase & 1) * gridDim.x;
        if (sum) {
            v = nn_warp_sum(v);
            if (lane == 0) ws[w] = v;
        }
        __syncthreads();
        ++phase;
        if (tid == 0 && !fail) {  // (a block that gave up arrives nowhere any more)
            if (sum) {
                double s = 0.0;
                for (int k = 0; k < CN_THREADS / 32; ++k) s += ws[k];
                part[blockIdx.x] = s;
            }
            __threadfence();
            atomicAdd(q.bar, 1u);
            int n = 0;
            while (*(volatile unsigned*)q.bar < phase * gridDim.x)
                if (++n > q.polls) {
                    fail = 1;
                    break;
                }
            __threadfence();
        }
        __syncthreads();
        if (sum && w == 0) {
            double s = 0.0;
            for (unsigned k = lane; k < gridDim.x; k += 32) s += ((volatile double*)part)[k];
            s = nn_warp_sum(s);
            if (lane == 0) total = s;
        }
        __syncthreads();
    };
    // zero-padded 3x3x3 correlation (af::convolve3 with AF_CONV_DEFAULT), x fastest
    auto conv = [&](I c, const Stencil27& K, auto val) {
        const int i = (int)(c % (I)q.nx), j = (int)((c / (I)q.nx) % (I)q.ny), k = (int)(c / ((I)q.nx * (I)q.ny));
        float acc = 0.0f;
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                for (int dx = -1; dx <= 1; ++dx) {
                    const int ii = i + dx, jj = j + dy, kk = k + dz;
                    if (ii < 0 || ii >= q.nx || jj < 0 || jj >= q.ny || kk < 0 || kk >= q.nz) continue;
                    acc += K.k[(dx + 1) + 3 * (dy + 1) + 9 * (dz + 1)] * val((I)ii + (I)q.nx * ((I)jj + (I)q.ny * (I)kk));
                }
        return acc;
    };

    for (I c = c0; c < G; c += stride) {
        auto val = [&](I n) { return q.u[n] + q.dep[n]; };
        const float lap = conv(c, q.L, val), un = val(c);
        q.un[c] = un;
        q.x[c] = q.a * un + q.bb * lap;
        q.b[c] = q.c * un + q.d * lap;
    }
    barrier(false, 0.0);
    double acc = 0.0;
    for (I c = c0; c < G; c += stride) {
        const float rv = q.b[c] - conv(c, q.A, [&](I n) { return q.x[n]; });
        q.r[c] = rv;
        acc += (double)rv * rv;
    }
    barrier(true, acc);
    double rr = total, pap = 0.0, rr_new = 0.0;
    int done = rr < (double)q.tol ? 2 : 0, it = 0;
    float beta = 0.0f;
    float *p_old = q.p1, *p_new = q.p0;
    while (!done && it < q.max_iter && !fail) {
        acc = 0.0;
        for (I c = c0; c < G; c += stride) {
            auto val = [&](I n) { return it ? q.r[n] + beta * p_old[n] : q.r[n]; };
            const float pv = val(c), ap = conv(c, q.A, val);
            p_new[c] = pv;
            q.Ap[c] = ap;
            acc += (double)pv * ap;
        }
        barrier(true, acc);
        pap = total;
        const float alpha = (float)(rr / pap);
        acc = 0.0;
        for (I c = c0; c < G; c += stride) {
            q.x[c] += alpha * p_new[c];
            const float rv = q.r[c] - alpha * q.Ap[c];
            q.r[c] = rv;
            acc += (double)rv * rv;
        }
        barrier(true, acc);
        rr_new = total;
        ++it;
        if (rr_new < (double)q.tol) {
            done = 1;
        } else {
            beta = (float)(rr_new / rr);
            rr = rr_new;
            float* t = p_old;
            p_old = p_new;
            p_new = t;
        }
    }
    if (fail) {
        if (tid == 0) {
            *(volatile int*)q.gave_up = 1;
            __threadfence_system();
        }
        return;  // the block's cells keep their density
    }
    // density = x unless the initial residual already met the tolerance (src/paracrine.cu:114-116)
    for (I c = c0; c < G; c += stride) q.u[c] = done == 2 ? q.un[c] : q.x[c];
    if (tid == 0 && blockIdx.x == 0) {
        q.done[0] = done;
        q.done[1] = it;
        q.scal[0] = rr;
        q.scal[1] = pap;
        q.scal[2] = rr_new;
    }
}

const void* cn_kernel(int64_t G)
{
    return G <= INT32_MAX / 2 ? (const void*)k_cn_solve<int> : (const void*)k_cn_solve<int64_t>;
}
}  // namespace

extern "C" nn_status nn_paracrine_ref_create(nn_ctx* ctx, const nn_paracrine_ref_params* p, int n, const float* d_x,
                                             const float* d_y, const float* d_z, float* d_g_paracrine,
                                             nn_paracrine** out)
{
    if (!ctx || !p || !out || n < 0 || p->nx < 2 || p->ny < 2 || p->nz < 2 || (n && (!d_x || !d_y || !d_z)))
        return nn_fail(ctx, NN_ERR_INVALID_ARG, "nn_paracrine_ref_create: bad argument");
    nn_paracrine* pm = new nn_paracrine();
    pm->ctx = ctx;
    nn_ctx_retain(ctx);
    pm->p = *p;
    pm->n = n;
    pm->G = (int64_t)p->nx * p->ny * p->nz;
    pm->g_out = d_g_paracrine;
    const size_t G = (size_t)pm->G, N = (size_t)(n > 0 ? n : 1);
    // co-resident blocks only
    const void* cn = cn_kernel(pm->G);
    int per_sm = 0;
    nn_status st = nn_cuda_check(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cn, CN_THREADS, 0), "k_cn_solve");
    pm->nparts = nn_grid_for(ctx, pm->G, CN_THREADS, std::max(1, std::min(per_sm, cn_blocks_per_sm(ctx, pm->G))));
#define PM_ALLOC(ptr, cnt) if (st == NN_OK) st = nn_alloc(ctx, &pm->ptr, cnt)
    PM_ALLOC(idx8, 8 * N); PM_ALLOC(w8, 8 * N);
    const size_t V = (G + 63) / 64 * 64;
    PM_ALLOC(grids, 9 * V);
    if (st == NN_OK) {
        float* v = pm->grids;
        for (float** q : {&pm->u, &pm->Ax, &pm->un, &pm->x, &pm->b, &pm->r, &pm->p0, &pm->p1, &pm->Ap}) {
            *q = v;
            v += V;
        }
    }
    PM_ALLOC(at_neurons, N); PM_ALLOC(generated, N);
    PM_ALLOC(scal, 4); PM_ALLOC(partials, 2 * (size_t)pm->nparts); PM_ALLOC(bar, 1); PM_ALLOC(done, 2);
#undef PM_ALLOC
    if (st == NN_OK) st = nn_pinned_word(ctx, &pm->h_gave_up);
    if (st != NN_OK) {
        nn_paracrine_destroy(pm);
        return st;
    }
    const char* polls = std::getenv("NN_CN_POLLS");
    pm->polls = polls ? std::atoi(polls) : CN_POLLS;
    cudaStream_t s = ctx->stream;
    cudaMemsetAsync(pm->u, 0, sizeof(float) * G, s);
    cudaMemsetAsync(pm->generated, 0, sizeof(float) * N, s);
    cudaMemsetAsync(pm->at_neurons, 0, sizeof(float) * N, s);
    cudaMemsetAsync(pm->done, 0, 2 * sizeof(int), s);
    if (n > 0) {
        k_trilinear<<<nn_grid_for(ctx, n, 256, 16), 256, 0, s>>>(n, d_x, d_y, d_z, p->nx, p->ny, p->nz, p->h, pm->idx8,
                                                                  pm->w8);
        ctx->launches++;
        // constructor: interpolate the (zero) density and copy it out (src/paracrine.cuh:238-242)
        k_interp<<<nn_grid_for(ctx, n, 256, 16), 256, 0, s>>>(n, pm->idx8, pm->w8, pm->u, pm->G, pm->at_neurons,
                                                               pm->g_out);
        ctx->launches++;
    }
    st = nn_cuda_check(ctx, cudaGetLastError(), "nn_paracrine_ref_create");
    if (st != NN_OK) {
        nn_paracrine_destroy(pm);
        return st;
    }
    *out = pm;
    return NN_OK;
}

extern "C" nn_status nn_paracrine_destroy(nn_paracrine* pm)
{
    if (!pm) return NN_OK;
    if (pm->ctx) cudaStreamSynchronize(pm->ctx->stream);
    nn_release(pm->idx8); nn_release(pm->w8); nn_release(pm->grids);
    nn_release(pm->at_neurons); nn_release(pm->generated); nn_release(pm->scal); nn_release(pm->partials);
    nn_release(pm->bar); nn_release(pm->done);
    nn_pinned_release(pm->ctx, pm->h_gave_up);
    nn_ctx* ctx = pm->ctx;
    delete pm;
    nn_ctx_release(ctx);
    return NN_OK;
}

extern "C" float* nn_paracrine_density(nn_paracrine* pm) { return pm ? pm->u : nullptr; }
extern "C" float* nn_paracrine_sources(nn_paracrine* pm) { return pm ? pm->generated : nullptr; }

// Reports a solve whose wait gave up, once.
static nn_status cn_gave_up(nn_paracrine* pm)
{
    volatile int* f = pm->h_gave_up;
    if (!*f) return NN_OK;
    *f = 0;
    return nn_fail(pm->ctx, NN_ERR_TIMEOUT, "k_cn_solve: a grid barrier gave up");
}

extern "C" nn_status nn_paracrine_ref_fine(nn_paracrine* pm, const nn_coupling* c)
{
    if (!pm || !c || c->n != pm->n) return nn_fail(pm ? pm->ctx : nullptr, NN_ERR_INVALID_ARG, "nn_paracrine_ref_fine: bad argument");
    NN_TRY(cn_gave_up(pm));
    if (pm->n == 0) return NN_OK;
    nn_ctx* ctx = pm->ctx;
    NN_CUDA(ctx, nn_launch_pdl(k_fine, dim3(nn_grid_for(ctx, pm->n, 256, 16)), dim3(256), 0, ctx->stream, pm->n, c->firing,
                               c->count, pm->generated, pm->p.coup_strength, pm->p.quirk_firing_list));
    NN_CHECK_LAUNCH(ctx, "k_fine");
    return NN_OK;
}

extern "C" nn_status nn_paracrine_ref_own(nn_paracrine* pm, int* iters, float* final_rr)
{
    if (!pm) return NN_ERR_INVALID_ARG;
    NN_TRY(cn_gave_up(pm));
    nn_ctx* ctx = pm->ctx;
    cudaStream_t s = ctx->stream;
    const auto& p = pm->p;
    const int64_t G = pm->G;
    const int nb = nn_grid_for(ctx, pm->n, 256, 16);
    // scatter_to_grid: Ax = G^T generated; density += Ax (src/paracrine.cu:276-287)
    NN_CUDA(ctx, cudaMemsetAsync(pm->Ax, 0, sizeof(float) * (size_t)G, s));
    if (pm->n > 0) {
        k_scatter<<<nb, 256, 0, s>>>(pm->n, pm->idx8, pm->w8, pm->generated, pm->Ax, G);
        NN_CHECK_LAUNCH(ctx, "k_scatter");
    }
    // update_density (src/paracrine.cu:63-134)
    const double h = p.h, dt = p.par_dt;
    Stencil27 L, A;
    static const float st[27] = {1, 3, 1, 3, 14, 3, 1, 3, 1, 3, 14, 3, 14, -128, 14, 3, 14, 3,
                                 1, 3, 1, 3, 14, 3, 1, 3, 1};
    for (int q = 0; q < 27; ++q) {
        const double lq = st[q] * (1.0 / (h * h * 30.0));
        L.k[q] = (float)lq;
        A.k[q] = (float)(-0.5 * p.D * dt * lq);
    }
    A.k[13] = (float)((double)A.k[13] + 1.0 + 0.5 * dt * p.decay);
    const double c = p.quirk_rhs ? h : dt;
    CnArgs q{p.nx, p.ny, p.nz, p.max_iter, G, L, A};
    q.a = (float)(1.0 - dt * p.decay);
    q.bb = (float)(dt * p.D);
    q.c = (float)(1.0 - c * p.decay / 2.0);
    q.d = (float)(c * p.D / 2.0);
    q.tol = p.abs_tol;
    q.dep = pm->Ax;
    q.u = pm->u; q.un = pm->un; q.x = pm->x; q.b = pm->b; q.r = pm->r;
    q.p0 = pm->p0; q.p1 = pm->p1; q.Ap = pm->Ap;
    q.scal = pm->scal;
    q.partials = pm->partials;
    q.bar = pm->bar;
    q.done = pm->done;
    NN_CUDA(ctx, cudaHostGetDevicePointer((void**)&q.gave_up, pm->h_gave_up, 0));
    q.polls = pm->polls;
    NN_CUDA(ctx, cudaMemsetAsync(pm->bar, 0, sizeof(unsigned), s));
    void* args[] = {&q};
    NN_CUDA(ctx, cudaLaunchCooperativeKernel(cn_kernel(G), dim3(pm->nparts), dim3(CN_THREADS), args, 0, s));
    ctx->launches++;
    // interpolate, reset sources, copy out (src/paracrine.cuh:259-264)
    if (pm->n > 0) {
        k_interp<<<nb, 256, 0, s>>>(pm->n, pm->idx8, pm->w8, pm->u, G, pm->at_neurons, pm->g_out);
        NN_CHECK_LAUNCH(ctx, "k_interp");
        NN_CUDA(ctx, cudaMemsetAsync(pm->generated, 0, sizeof(float) * (size_t)pm->n, s));
    }
    if (std::getenv("NN_DEBUG_PARACRINE")) {
        int h_done[2];
        double h_scal[3];
        std::vector<float> hu((size_t)G), hx((size_t)G), hax((size_t)G);
        cudaMemcpyAsync(h_done, pm->done, sizeof h_done, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(h_scal, pm->scal, sizeof h_scal, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hu.data(), pm->u, sizeof(float) * (size_t)G, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hx.data(), pm->x, sizeof(float) * (size_t)G, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hax.data(), pm->Ax, sizeof(float) * (size_t)G, cudaMemcpyDeviceToHost, s);
        cudaStreamSynchronize(s);
        double su = 0, sx = 0, sa = 0;
        for (int64_t q = 0; q < G; ++q) { su += hu[(size_t)q]; sx += hx[(size_t)q]; sa += hax[(size_t)q]; }
        fprintf(stderr, "[paracrine] done=%d iters=%d rr0=%g pAp=%g rr=%g sum(u)=%.9g sum(x)=%.9g sum(Ax)=%.9g\n",
                h_done[0], h_done[1], h_scal[0], h_scal[1], h_scal[2], su, sx, sa);
    }
    if (iters || final_rr) {
        int h_done[2];
        double h_scal[3];
        NN_CUDA(ctx, cudaMemcpyAsync(h_done, pm->done, sizeof h_done, cudaMemcpyDeviceToHost, s));
        NN_CUDA(ctx, cudaMemcpyAsync(h_scal, pm->scal, 3 * sizeof(double), cudaMemcpyDeviceToHost, s));
        NN_CUDA(ctx, cudaStreamSynchronize(s));
        NN_TRY(cn_gave_up(pm));
        if (iters) *iters = h_done[1];
        if (final_rr) *final_rr = (float)(h_done[1] == 0 ? h_scal[0] : (h_done[0] == 1 ? h_scal[2] : h_scal[0]));
    }
    return NN_OK;
}
