// mfree_interact.cuh -- the pair loop and the fused per-particle rest of the step
// (kernel templates; mfree_interact.cu instantiates and launches them).
//
// Reference path replaced (src/leap_frog.cu:153-171):
//   do_interactions_monaghan  interactions_gpu.cu:152-471 (CSPM pre-pass, velocity
//                             gradient, stress divergence with artificial stress,
//                             artificial viscosity, XSPH, Brookshaw conduction)
//   do_interactions_heat      interactions_gpu.cu:89-150 (PSE conduction)
//   do_material_stress_rate_jaumann, do_contmech_continuity/momentum/advection
//                             actions_gpu.cu:134-300
//   correct                   leap_frog.cu:72-100
//   do_plasticity_johnson_cook actions_gpu.cu:371-449
//   do_reset_contact_forces, do_boundary_conditions(_thermal), do_move_tool_particles
//                             leap_frog.cu:102-119, actions_gpu.cu:55-68,451-487
//                             (particles inside a tool box defer these to kb_finalize)
//
// Work decomposition: a persistent block (one per SM) pulls tiles of 4 x 4 x D
// cells (D up to 8) of every scene of the table from one work
// counter (the tile list cuts the grid so that tiles are about equally full).
// The tile's particles are 16 contiguous ranges of the sorted order;
// the records their 5x5x5 stencils touch are the 64 contiguous column ranges
// of the 8 x 8 x (D+4)-cell halo, staged into shared memory with two bulk
// copies per column, its P records and the interleaved rest (TMA
// cp.async.bulk, completion counted on an mbarrier, bounded waits).
//
// Two lanes serve a target; the 480 compute threads hold up to 240 targets of
// a tile at once, each from its candidates to its new state without a block
// barrier in between.  The candidate pass walks the 25 stencil columns of the target's
// cell, the two lanes on alternate records, and puts the in-support neighbours
// into a queue that the lanes fill from its two ends.  The pair pass runs on
// the queue only -- the reference evaluates the pair body for every candidate,
// ~3.5x more work, and candidates outside the support contribute exact zeros
// there.  Four lanes share a target's queue there; their sums are joined by
// shuffles, then the first of its two lanes runs the fused rest of the step.  A producer warp builds the next tile's tables
// while the compute warps work, and issues its copies as soon as they have
// read the last record of the current tile, so that the copies land while the
// epilogue runs.
//
// What bounds it: instruction issue (52 % of the cycles) and shared-memory
// wavefronts (57 %), with 16 warps an SM -- the registers and the staged halo
// leave room for no more -- to hide latencies, and 25 % of warp time at the
// tile's barriers; FP32 pipe 34 %, DRAM 5 % (profiles/kb_interact_1m.md, 1M
// particles).  The split
// follows from the instructions it saves: eight lanes a target throughout (an
// earlier form) spent about 80 instruction slots a candidate on ballots and on
// walking columns that are about as long as the group is wide.  Pair kernel,
// us, that form -> this one: 1M with CSPM + PSE 1845 -> 1258, 1M with every
// temperature different 2062 -> 1396, 4.1M with Brookshaw 6646 -> 4575, 252,000
// 473 -> 323 (eager event times).
//
// Tried and slower: 2 or 3 candidates a lane at once (+2 %, +1 %); two queue
// entries a lane and iteration (+-0 with four lanes); 12 warps with 168 registers
// and no spills (+3 % at 1M, +8 % at 4.1M; -7 % at 30,000 particles); the
// epilogue's state prefetched into L2 by the producer warp (+11 %); compute warps
// polling the mbarrier themselves (+-0).
#pragma once

#include <type_traits>

#include "mfree_kernels.cuh"

namespace mfree {

// The CSPM matrix B = sum V_j (x_i - x_j) (x) grad W_ij is symmetric (grad W
// is parallel to x_i - x_j), and so is its inverse: both are kept as the six
// entries xx, yy, zz, xy, xz, yz.
__device__ __forceinline__ float det3s(const float *m) {
    return m[0] * (m[1] * m[2] - m[5] * m[5]) - m[3] * (m[3] * m[2] - m[4] * m[5]) + m[4] * (m[3] * m[5] - m[4] * m[1]);
}
// inverse by cofactors (cofactor(r, c) / det; symmetric)
__device__ __forceinline__ void inv3s(const float *m, float det, float *o) {
    const float id = 1.0f / det;
    o[0] = (m[1] * m[2] - m[5] * m[5]) * id;  // xx
    o[1] = (m[0] * m[2] - m[4] * m[4]) * id;  // yy
    o[2] = (m[0] * m[1] - m[3] * m[3]) * id;  // zz
    o[3] = (m[4] * m[5] - m[3] * m[2]) * id;  // xy
    o[4] = (m[3] * m[5] - m[4] * m[1]) * id;  // xz
    o[5] = (m[3] * m[4] - m[0] * m[5]) * id;  // yz
}

// ------------------------------------------------------ packed arithmetic --
// two FP32 operations per instruction (FADD2/FMUL2/FFMA2): the same IEEE
// results as two scalar ones, half the issue slots
__device__ __forceinline__ unsigned long long f2_bits(float2 v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
    return r;
}
__device__ __forceinline__ float2 f2_of(unsigned long long r) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(f2_bits(a)), "l"(f2_bits(b)), "l"(f2_bits(c)));
    return f2_of(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f2_bits(a)), "l"(f2_bits(b)));
    return f2_of(d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f2_bits(a)), "l"(f2_bits(b)));
    return f2_of(d);
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// -------------------------------------------------------------- pair body --
// the target's terms of the pair loop; its own sigma and R enter the stress
// divergence only through the sums (see finish_sums) and are read after the
// loop.  Differences and sums are packed with an addition each, so the
// target's values are kept with the sign they are added with.
struct Target {
    float2 nxy;       // -x, -y
    float nz;         // -z
    float2 nvxy;      // -vx, -vy
    float2 nvz_rho;   // -vz, rho
    float2 ch;        // c, h
    float T, tool, h1;
    float c_art;      // W(0-free part) factor / wdeltap: fab = (val c_art)^4
    bool art;
};
// the scene's constants of the pair body, in registers for a target's loop
struct PairConst {
    float eta2_4, alpha_2, beta_2;  // eta^2 / 4, -AV alpha / 2, AV beta / 2
};

// The sums of a target.  Every gradient sum is taken with the pair's unscaled
// factor g = (u^2 - t^2/4)/r (x_i - x_j), t = 2 - q, u = max(1 - q, 0), q = r/h:
// grad W = 3 fac/h g with fac = 1/(pi h^3), and W = fac (t^3/4 - u^3) (the two
// branches of cubic_spline, kernels.cuh:26-69, in one expression).  The factor
// and, with CSPM, the correction matrix are applied once after the loop: all
// terms are linear in the gradient.  So CSPM needs no pass of its own over the
// neighbours; the stress divergence then keeps sigma_j (x) g uncontracted.
template <bool CSPM, int COND> struct Sums {
    float2 Lx, Ly, Lz;       // sum vol dv_{x,y} g_x, g_y, g_z
    float2 Lw;               // sum vol dv_z g_{x,y}
    float Lzz;               // sum vol dv_z g_z
    float2 s0[3], s1[3], s2[3];  // CSPM: sum (t_xx, t_xy), (t_xz, t_yz), (t_yy, t_zz) times g_x, g_y, g_z
    float2 dx2;              // else: t_xx g_x, t_xy g_y (added: row x)
    float2 dz2;              //       t_xz g_x, t_yz g_y (added: row z)
    float2 dxy;              //       t_xz g_z, t_yz g_z (rows x and y)
    float dy, dz;            //       t_xy g_x + t_yy g_y, t_zz g_z
    float2 av; float avz;    // sum -pi_ij g
    float2 xs; float xsz;    // sum -W/(fac rho_ij) dv / 2 (factors after the loop)
    float2 g; float gz;      // sum g
    float2 f; float fz;      // sum fab g
    float2 b0; float2 b1; float bxz, bzz;  // CSPM: -sum vol d (x) g: (xx, xy), (yy, yz), xz, zz
    float2 h0; float2 h1; float hxz, hzz;  // CSPM + Brookshaw: the heat sum before its contraction
    float heat;              // Brookshaw without CSPM
    __device__ __forceinline__ void zero() {
        const float2 z = make_float2(0.f, 0.f);
        Lx = Ly = Lz = Lw = z; Lzz = 0.f;
#pragma unroll
        for (int k = 0; k < 3; k++) s0[k] = s1[k] = s2[k] = z;
        dx2 = dz2 = dxy = z; dy = dz = 0.f;
        av = xs = g = f = z; avz = xsz = gz = fz = 0.f;
        b0 = b1 = z; bxz = bzz = 0.f;
        h0 = h1 = z; hxz = hzz = 0.f;
        heat = 0.f;
    }
    // the sums as a list (zeros past COUNT), and back
    static constexpr int COUNT = CSPM ? (COND == MFREE_COND_BROOKSHAW ? 51 : 45) : (COND == MFREE_COND_BROOKSHAW ? 25 : 24);
    template <class F> __device__ __forceinline__ void each(F &&v) {
        auto v2 = [&](float2 &p) { v(p.x); v(p.y); };
        v2(Lx); v2(Ly); v2(Lz); v2(Lw); v(Lzz);
        v2(av); v(avz); v2(xs); v(xsz); v2(g); v(gz); v2(f); v(fz);
        if (CSPM) {
#pragma unroll
            for (int k = 0; k < 3; k++) { v2(s0[k]); v2(s1[k]); v2(s2[k]); }
            v2(b0); v2(b1); v(bxz); v(bzz);
        } else {
            v(dx2.x); v(dy); v(dz);
        }
        if (COND == MFREE_COND_BROOKSHAW) {
            if (CSPM) { v2(h0); v2(h1); v(hxz); v(hzz); }
            else v(heat);
        }
    }
    // without CSPM: the parts of the stress divergence in one value a row
    __device__ __forceinline__ void fold() {
        if (CSPM) return;
        dx2.x += dx2.y + dxy.x;
        dy += dxy.y;
        dz += dz2.x + dz2.y;
        dx2.y = dxy.x = dxy.y = dz2.x = dz2.y = 0.f;
    }
    // the sums over the LANES lanes of a group, left in row[0..COUNT) (shared
    // memory): a butterfly that halves the list at every step, so a lane ends
    // with a quarter of it.  Every lane of the warp calls it.
    template <int LANES> __device__ __forceinline__ void reduce_to(float *row, int l, bool store) {
        fold();
        constexpr int REST = COUNT % 8 <= 2 ? COUNT % 8 : 0;  // few left over: reduced in full
        constexpr int MAIN = (COUNT - REST + 7) / 8 * 8;
        float a[MAIN + 8];
#pragma unroll
        for (int k = 0; k < MAIN + 8; k++) a[k] = 0.f;
        int n = 0;
        each([&](float &v) { a[n++] = v; });
        constexpr int STEPS = LANES == 4 ? 2 : 1;
        int base = 0;
#pragma unroll
        for (int st = 0; st < STEPS; st++) {
            const int o = LANES >> (st + 1), half = MAIN >> (st + 1);
            const bool up = (l & o) != 0;
            if (up) base += half;
#pragma unroll
            for (int k = 0; k < half; k++) {
                const float send = up ? a[k] : a[k + half], keep = up ? a[k + half] : a[k];
                a[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
#pragma unroll
        for (int k = 0; k < REST; k++)
#pragma unroll
            for (int o = LANES / 2; o >= 1; o >>= 1) a[MAIN + k] += __shfl_xor_sync(0xffffffffu, a[MAIN + k], o);
        if (!store) return;
#pragma unroll
        for (int k = 0; k < (MAIN >> STEPS); k++)
            if (base + k < COUNT - REST) row[base + k] = a[k];
        if (l == 0)
#pragma unroll
            for (int k = 0; k < REST; k++) row[COUNT - REST + k] = a[MAIN + k];
    }
    __device__ __forceinline__ void load(const float *row) {
        int n = 0;
        each([&](float &v) { v = row[n++]; });
    }
};

// one neighbour: X points at its interleaved V, A, B, R, C records
template <bool CSPM, int COND>
__device__ __forceinline__ void pair_body(const PairConst &P, const Target &I, const float4 Pj, const float4 *X,
                                          Sums<CSPM, COND> &S) {
    const float4 Vj = X[REC_V - 1], Aj = X[REC_A - 1], Bj = X[REC_B - 1], Cj = X[REC_C - 1];
    const float2 nd = add2(lo2(Pj), I.nxy);  // -(x_i - x_j) in x, y
    const float ndz = Pj.z + I.nz;
    const float r2 = fmaf(ndz, ndz, fmaf(nd.y, nd.y, nd.x * nd.x));
    const float rinv = rsqrt_approx(r2);  // r2 >= 1e-8 here: never a denormal
    const float q = r2 * rinv * I.h1;
    const float2 tu = make_float2(2.f - q, fmaxf(1.f - q, 0.f));
    const float2 tu2 = mul2(tu, tu), tu3 = mul2(tu2, tu);
    const float val = fmaf(0.25f, tu3.x, -tu3.y);
    const float ng = fmaf(0.25f, tu2.x, -tu2.y) * rinv;  // -(u^2 - t^2/4)/r: g = ng * nd
    const float2 g = mul2(both(ng), nd);
    const float gz = ng * ndz;
    const float vol = Cj.w;
    if (!(I.tool == 1.f) && !(Pj.w == 1.f)) {
        const float2 dv = add2(lo2(Vj), I.nvxy);         // v_j - v_i
        const float2 zr = add2(hi2(Vj), I.nvz_rho);      // the z component; rho_i + rho_j
        const float2 gx2 = both(g.x), gy2 = both(g.y), gz2 = both(gz);
        {
            const float2 a = mul2(both(vol), dv);
            const float az = vol * zr.x;
            S.Lx = fma2(a, gx2, S.Lx);
            S.Ly = fma2(a, gy2, S.Ly);
            S.Lz = fma2(a, gz2, S.Lz);
            S.Lw = fma2(both(az), g, S.Lw);
            S.Lzz = fmaf(az, gz, S.Lzz);
        }
        // sum_j (sigma_i + sigma_j + fab (R_i + R_j)) g
        //   = sum_j (sigma_j + fab R_j) g + sigma_i sum_j g + R_i sum_j fab g
        float2 t0 = lo2(Aj), t1 = hi2(Aj), t2 = lo2(Bj);  // (xx, xy), (xz, yz), (yy, zz)
        if (I.art) {
            const float4 Rj = X[REC_R - 1];
            float fab = val * I.c_art;
            fab *= fab;
            fab *= fab;
            const float2 fab2 = both(fab);
            t0 = fma2(fab2, lo2(Rj), t0);
            t1 = fma2(fab2, hi2(Rj), t1);
            t2 = fma2(fab2, lo2(Cj), t2);
            S.f = fma2(fab2, g, S.f);
            S.fz = fmaf(fab, gz, S.fz);
        }
        S.g = add2(S.g, g);
        S.gz += gz;
        if (CSPM) {
            S.s0[0] = fma2(t0, gx2, S.s0[0]); S.s0[1] = fma2(t0, gy2, S.s0[1]); S.s0[2] = fma2(t0, gz2, S.s0[2]);
            S.s1[0] = fma2(t1, gx2, S.s1[0]); S.s1[1] = fma2(t1, gy2, S.s1[1]); S.s1[2] = fma2(t1, gz2, S.s1[2]);
            S.s2[0] = fma2(t2, gx2, S.s2[0]); S.s2[1] = fma2(t2, gy2, S.s2[1]); S.s2[2] = fma2(t2, gz2, S.s2[2]);
            // B = -sum V_j d (x) grad W with d = -nd
            const float2 w = mul2(both(vol), nd);
            S.b0 = fma2(both(w.x), g, S.b0);
            S.b1 = fma2(both(w.y), make_float2(g.y, gz), S.b1);
            S.bxz = fmaf(w.x, gz, S.bxz);
            S.bzz = fmaf(vol * ndz, gz, S.bzz);
        } else {
            S.dx2 = fma2(t0, g, S.dx2);
            S.dz2 = fma2(t1, g, S.dz2);
            S.dxy = fma2(t1, gz2, S.dxy);
            S.dy = fmaf(t0.y, g.x, fmaf(t2.x, g.y, S.dy));
            S.dz = fmaf(t2.y, gz, S.dz);
        }
        const float ir = rcp_approx(zr.y);  // 1 / (rho_i + rho_j)
        {   // artificial viscosity for approaching pairs, without a branch:
            // mu = h_ij v.r/(r2 + eta^2 h_ij^2), h_ij = hs/2 (m = 2 mu), c_ij = cs/2
            const float2 cs = add2(hi2(Bj), I.ch);
            const float vr = fminf(fmaf(zr.x, ndz, fmaf(dv.y, nd.y, dv.x * nd.x)), 0.f);
            const float m = vr * cs.y * rcp_approx(fmaf(P.eta2_4 * cs.y, cs.y, r2));
            const float npij = -m * fmaf(P.beta_2, m, P.alpha_2 * cs.x) * ir;
            S.av = fma2(both(npij), g, S.av);
            S.avz = fmaf(npij, gz, S.avz);
        }
        const float xw = val * ir;
        S.xs = fma2(both(xw), dv, S.xs);
        S.xsz = fmaf(xw, zr.x, S.xsz);
    }
    if (COND == MFREE_COND_BROOKSHAW) {
        // 2 (m/rho_j)(T_i - T_j) e.grad W / r = 2 V_j (T_i - T_j) (d.grad W)/r^2; factor 2 in the
        // epilogue.  Without CSPM d.g/r^2 is the pair's factor -ng.
        const float k = -vol * (I.T - Cj.z) * ng;
        if (CSPM) {
            const float w = k * rinv * rinv;
            const float2 v = mul2(both(w), nd);
            S.h0 = fma2(both(v.x), nd, S.h0);
            S.h1 = fma2(both(v.y), make_float2(nd.y, ndz), S.h1);
            S.hxz = fmaf(v.x, ndz, S.hxz);
            S.hzz = fmaf(w * ndz, ndz, S.hzz);
        } else {
            S.heat += k;
        }
    }
}

// the target's values from its records (h1, c_art and art are set apart)
template <bool CSPM, int COND> __device__ __forceinline__ void target_of(const float4 Pi, const float4 *X, Target &I) {
    const float4 Vi = X[REC_V - 1];
    I.nxy = make_float2(-Pi.x, -Pi.y);
    I.nz = -Pi.z;
    I.tool = Pi.w;
    I.nvxy = make_float2(-Vi.x, -Vi.y);
    I.nvz_rho = make_float2(-Vi.z, Vi.w);
    I.ch = hi2(X[REC_B - 1]);
    I.T = X[REC_C - 1].z;
}

// the joined sums as the epilogue takes them: 0-8 velocity gradient, 9-11
// stress divergence, 12-14 viscosity, 15-17 XSPH, 18 heat (Brookshaw)
template <bool CSPM, int COND>
__device__ __forceinline__ void finish_sums(const Sums<CSPM, COND> &S, const Target &I, float fac, const float4 Ai,
                                            const float4 Bi, const float4 Ri, const float4 Ci, float *o) {
    const float sc = 3.f * fac * I.h1;  // grad W = sc g
    // rows of the correction (times sc); the identity without CSPM
    float M[6] = {sc, sc, sc, 0.f, 0.f, 0.f};  // xx, yy, zz, xy, xz, yz
    if (CSPM) {
        float B[6] = {sc * S.b0.x, sc * S.b1.x, sc * S.bzz, sc * S.b0.y, sc * S.bxz, sc * S.b1.y}, inv[6];
        const float det = det3s(B);
        if (det > 9.99999994e-9f) {
            inv3s(B, det, inv);
#pragma unroll
            for (int k = 0; k < 6; k++) M[k] = sc * inv[k];
        }
    }
    auto corr = [&](float gx, float gy, float gz, float &x, float &y, float &z) {
        if (CSPM) {
            x = fmaf(M[0], gx, fmaf(M[3], gy, M[4] * gz));
            y = fmaf(M[3], gx, fmaf(M[1], gy, M[5] * gz));
            z = fmaf(M[4], gx, fmaf(M[5], gy, M[2] * gz));
        } else {
            x = sc * gx; y = sc * gy; z = sc * gz;
        }
    };
    corr(S.Lx.x, S.Ly.x, S.Lz.x, o[0], o[1], o[2]);
    corr(S.Lx.y, S.Ly.y, S.Lz.y, o[3], o[4], o[5]);
    corr(S.Lw.x, S.Lw.y, S.Lzz, o[6], o[7], o[8]);
    if (CSPM) {
        float a, b, c, x, y, z;
        corr(S.s0[0].x, S.s0[1].x, S.s0[2].x, x, y, z);  // t_xx
        a = x;
        corr(S.s0[0].y, S.s0[1].y, S.s0[2].y, x, y, z);  // t_xy
        a += y; b = x;
        corr(S.s1[0].x, S.s1[1].x, S.s1[2].x, x, y, z);  // t_xz
        a += z; c = x;
        corr(S.s1[0].y, S.s1[1].y, S.s1[2].y, x, y, z);  // t_yz
        b += z; c += y;
        corr(S.s2[0].x, S.s2[1].x, S.s2[2].x, x, y, z);  // t_yy
        b += y;
        corr(S.s2[0].y, S.s2[1].y, S.s2[2].y, x, y, z);  // t_zz
        c += z;
        o[9] = a; o[10] = b; o[11] = c;
    } else {
        o[9] = sc * S.dx2.x;
        o[10] = sc * S.dy;
        o[11] = sc * S.dz;
    }
    float gx, gy, gz, fx, fy, fz;
    corr(S.g.x, S.g.y, S.gz, gx, gy, gz);
    corr(S.f.x, S.f.y, S.fz, fx, fy, fz);
    // sigma_i sum g + R_i sum fab g; A = (xx, xy, xz, yz), B = (yy, zz, ..), R, C alike
    o[9] = fmaf(Ai.x, gx, fmaf(Ai.y, gy, fmaf(Ai.z, gz, o[9])));
    o[10] = fmaf(Ai.y, gx, fmaf(Bi.x, gy, fmaf(Ai.w, gz, o[10])));
    o[11] = fmaf(Ai.z, gx, fmaf(Ai.w, gy, fmaf(Bi.y, gz, o[11])));
    o[9] = fmaf(Ri.x, fx, fmaf(Ri.y, fy, fmaf(Ri.z, fz, o[9])));
    o[10] = fmaf(Ri.y, fx, fmaf(Ci.x, fy, fmaf(Ri.w, fz, o[10])));
    o[11] = fmaf(Ri.z, fx, fmaf(Ri.w, fy, fmaf(Ci.y, fz, o[11])));
    corr(S.av.x, S.av.y, S.avz, o[12], o[13], o[14]);
    const float xf = -2.f * fac;  // W/rho_ij (v_i - v_j) = -2 fac val/(rho_i + rho_j) dv
    o[15] = xf * S.xs.x; o[16] = xf * S.xs.y; o[17] = xf * S.xsz;
    if (COND == MFREE_COND_BROOKSHAW) {
        if (CSPM)
            o[18] = M[0] * S.h0.x + M[1] * S.h1.x + M[2] * S.hzz + 2.f * (M[3] * S.h0.y + M[4] * S.hxz + M[5] * S.h1.y);
        else
            o[18] = sc * S.heat;
    }
}

// ------------------------------------------------------------ epilogue --
template <bool PREC, int COND>
__device__ void epilogue(const StepArgs &a, int i, const float *res) {
    const Params &P = a.p;
    const State &S = a.b;
    float4 pos = S.pos4[i], vel = S.vel4[i], sa = S.sa4[i], sb = S.sb4[i];
    float4 da = S.da4[i], dv = S.dv4[i], dsa = S.dsa4[i], dsb = S.dsb4[i];
    float4 ft = S.ft4[i], fc = S.fc4[i];
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), lob = lo;
    if (PREC) {
        lo = S.lo4[i];
        lob = S.lo4b[i];
    }
    const float dt = P.dt;
    const HalfStep hs = half_step<PREC>(0.5f * dt, pos, vel, sa, sb, da, dv, dsa, dsb, lo, lob);
    const float tool_p = fc.w;
    const bool tool = tool_p == 1.f;
    const float fixed = dsb.w;
    // ---- rates
    float pt[3], vt[3], St[6], rho_t, T_t;
    if (!tool) {
        float L[9];
#pragma unroll
        for (int k = 0; k < 9; k++) L[k] = res[k];
        jaumann(L, hs.S, P.G, St);
        rho_t = -hs.rho * (L[0] + L[4] + L[8]);
        const float im = 1.0f / P.mass;
        vt[0] = P.mass * (res[12] + res[9]) + fc.x * im + ft.x * im;
        vt[1] = P.mass * (res[13] + res[10]) + fc.y * im + ft.y * im;
        vt[2] = P.mass * (res[14] + res[11]) + fc.z * im + ft.z * im;
        const float xf = -P.xspheps * P.mass;
        pt[0] = fmaf(xf, res[15], hs.vx);
        pt[1] = fmaf(xf, res[16], hs.vy);
        pt[2] = fmaf(xf, res[17], hs.vz);
    } else {
        pt[0] = pt[1] = pt[2] = 0.f;
        vt[0] = vt[1] = vt[2] = 0.f;
        St[0] = dsa.x; St[1] = dsa.y; St[2] = dsa.z; St[3] = dsa.w; St[4] = dsb.x; St[5] = dsb.y;
        rho_t = da.w;
    }
    T_t = dv.w;
    if (COND == MFREE_COND_BROOKSHAW) {
        const float al = tool_p == 0.f ? P.wp_alpha : P.tool_alpha;
        if (al != 0.f) T_t = al * (2.0f * res[18]);
    } else if (COND == MFREE_COND_PSE) {
        if (P.wp_alpha != 0.f) {
            const float al = tool ? P.tool_alpha : P.wp_alpha;
            const float h = pos.w, h2 = h * h;
            const float coef = 4.0f / (h2 * h2 * h * 5.5683279968317078f);  // pi^1.5
            T_t = al * coef * res[18];
        }
    }
    // ---- corrector x1 = x0 + dt * xdot (leap_frog.cu:72-100)
    if (PREC) {
        acc_comp(pos.x, lo.x, dt, pt[0]);
        acc_comp(pos.y, lo.y, dt, pt[1]);
        acc_comp(pos.z, lo.z, dt, pt[2]);
        acc_comp(vel.x, lo.w, dt, vt[0]);
        acc_comp(vel.y, lob.x, dt, vt[1]);
        acc_comp(vel.z, lob.y, dt, vt[2]);
    } else {
        pos.x = fmaf(dt, pt[0], pos.x);
        pos.y = fmaf(dt, pt[1], pos.y);
        pos.z = fmaf(dt, pt[2], pos.z);
        vel.x = fmaf(dt, vt[0], vel.x);
        vel.y = fmaf(dt, vt[1], vel.y);
        vel.z = fmaf(dt, vt[2], vel.z);
    }
    float s[6] = {fmaf(dt, St[0], sa.x), fmaf(dt, St[1], sa.y), fmaf(dt, St[2], sa.z),
                  fmaf(dt, St[3], sa.w), fmaf(dt, St[4], sb.x), fmaf(dt, St[5], sb.y)};
    vel.w = fmaf(dt, rho_t, vel.w);  // rho
    float T = fmaf(dt, T_t, sb.z);
    float eps = sb.w, epsd = dsb.z;
    // ---- Johnson-Cook radial return (actions_gpu.cu:371-449)
    if (P.plastic && !tool) {
        const float nS = sqrtf(s[0] * s[0] + s[1] * s[1] + s[2] * s[2] + 2.f * (s[3] * s[3] + s[5] * s[5] + s[4] * s[4]));
        float Tc = T;
        if (P.jc_clamp != 0.f) Tc = Tc > P.jc_Tmelt ? P.jc_Tmelt - 1.f : Tc;
        const float svm = 1.22474487139158905f * nS;
        if (jc_clearly_elastic(P, svm, eps, epsd, Tc) || svm < 0.99f * jc_yield_stress_screen(P, eps, epsd, Tc) ||
            svm < jc_yield_stress(P, eps, epsd, Tc)) {
            epsd = 0.f;  // elastic
        } else {
            // FP64 secant from FP32 inputs, the result stored as float
            int failed = 0;
            const double init = fmax((double)(epsd * dt) * 0.81649658092772603, 1e-8);
            const float dl = (float)jc_secant(P, init, nS, eps, Tc, dt, &failed);
            if (failed) atomicAdd(&a.clk->secant_failures, 1ull);
            const float s23 = 0.81649658092772603f;  // sqrtf(2/3)
            const float e1 = eps + s23 * fmaxf(dl, 0.f);
            const float ed1 = s23 * fmaxf(dl, 0.f) / dt;
            // S - S / |S| * dl * 2 * G: the quotient and the product with dl in
            // float, the rest in double (the literal 2. promotes it)
#pragma unroll
            for (int k = 0; k < 6; k++) s[k] = (float)((double)s[k] - (double)(s[k] / nS * dl) * 2.0 * (double)P.G);
            if (P.wp_tq != 0.f) {
                const float sY2 = jc_yield_stress(P, e1, ed1, Tc);
                T += P.wp_tq / (P.wp_cp * vel.w) * (e1 - eps) * sY2;
            }
            eps = e1;
            epsd = ed1;
        }
    }
    // ---- contact reset; particles inside a tool box finish in kb_finalize
    const bool deferred = !tool && contact_candidate(a, pos.x, pos.y, pos.z);
    if (deferred) atomicOr(&a.s.contact[i >> 5], 1u << (i & 31));
    fc.x = fc.y = fc.z = 0.f;  // w keeps tool_p
    ft.x = ft.y = ft.z = 0.f;  // w keeps blanked
    if (!deferred) {
        if (!tool && fixed != 0.f) {
            const float4 bc = S.bc4[i];
            vel.x = bc.x; vel.y = bc.y; vel.z = bc.z;
            if (PREC) { lo.w = 0.f; lob.x = lob.y = 0.f; }
            pt[0] = pt[1] = pt[2] = 0.f;
            vt[0] = vt[1] = vt[2] = 0.f;
        }
        if (P.thermal && fixed == 1.f) T = P.wp_Tinit;
        if (P.diagnostics) a.s.nrm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tool) {  // do_move_tool_particles
        if (PREC) {
            acc_comp(pos.x, lo.x, dt, P.tool0_vel[0]);
            acc_comp(pos.y, lo.y, dt, P.tool0_vel[1]);
            acc_comp(pos.z, lo.z, dt, P.tool0_vel[2]);
        } else {
            pos.x = fmaf(P.tool0_vel[0], dt, pos.x);
            pos.y = fmaf(P.tool0_vel[1], dt, pos.y);
            pos.z = fmaf(P.tool0_vel[2], dt, pos.z);
        }
    }
    S.pos4[i] = pos;
    S.vel4[i] = vel;
    S.sa4[i] = make_float4(s[0], s[1], s[2], s[3]);
    S.sb4[i] = make_float4(s[4], s[5], T, eps);
    S.da4[i] = make_float4(pt[0], pt[1], pt[2], rho_t);
    S.dv4[i] = make_float4(vt[0], vt[1], vt[2], T_t);
    S.dsa4[i] = make_float4(St[0], St[1], St[2], St[3]);
    S.dsb4[i] = make_float4(St[4], St[5], epsd, fixed);
    S.fc4[i] = fc;
    S.ft4[i] = ft;
    if (PREC) {
        S.lo4[i] = lo;
        S.lo4b[i] = lob;
    }
    if (P.diagnostics) a.s.nnb[i] = __float_as_int(res[19]);
}

// ---------------------------------------------------------- pair kernel --
// Tile = TX x TY x D cells of the cell grid; its particles are 16 contiguous
// column ranges of the sorted order.  Their 5x5x5 stencils lie in the halo of
// HX x HY x (D+4) cells: 64 contiguous column ranges of the P records and of the
// interleaved rest, which two bulk copies per column (cp.async.bulk,
// completion counted on an mbarrier) stage into shared memory in the same
// layout.  A tile whose halo exceeds the staging capacity reads the same
// records from global memory instead.
constexpr int HX = TX + 4, HY = TY + 4;
constexpr int CSROW = TILE_Z_MAX + 5;  // cell starts kept per halo column
constexpr int NHC = HX * HY;           // halo columns
constexpr int NTC = TX * TY;           // target columns
constexpr int LPT = 2;                 // lanes per target
constexpr int PPT = 4;                 // lanes per target in the pair pass
constexpr int TPR = 32 / PPT;          // targets of a warp at a time there
constexpr int NCOMP = 480;             // compute threads
constexpr int NTHREADS = NCOMP + 32;   // and the producer warp: 16 warps, 128 registers a thread
constexpr int TCAP = NCOMP / LPT;      // targets per pass of a tile
constexpr int QCAP = 96;               // in-support queue per target before the rescan path
constexpr int CH = 4;                  // candidates a lane tests at once
constexpr int QROW = 102;              // 204 bytes a target: the rows of a warp on different banks, and room for its sums

constexpr int SMEM_LIMIT = 232448;     // per-block shared memory of sm_100
constexpr long long WAIT_CYCLES = 1ll << 30;  // bound of a staging wait (~0.5 s of SM clock)

// a tile's tables, built by the producer warp one tile ahead (two buffers)
struct TileTab {
    int cs[NHC][CSROW];   // record index (staged) or sorted index of the cell starts of each halo column
    int shift[NHC];       // record index minus sorted index of each halo column (staged)
    int trec[NTC];        // record index of each target column's first target
    int tsrt[NTC];        // its sorted index
    int tpref[NTC + 1];   // targets before the column
    float4 org;           // stencil pruning: grid origin, w = margin in cells (0: off)
    int tile, depth, scene, args, total, staged;  // scene < 0: no tile left; args: slot of the scene's arguments
    int nzr, rec0;        // cell starts in use per halo column; a target's record
};
struct BlockSmem {
    TileTab tab[2];
    unsigned long long bar;
    int fail;
};
__host__ __device__ constexpr size_t round128(size_t b) { return (b + 127) / 128 * 128; }
// shared memory: the tables, the arguments of two scenes, the queues, the staged records
constexpr size_t ARGS_OFFSET = round128(sizeof(BlockSmem));
constexpr size_t ARGS_SIZE = round128(sizeof(StepArgs));
constexpr size_t QUEUE_OFFSET = ARGS_OFFSET + 2 * ARGS_SIZE;
constexpr size_t REC_OFFSET = round128(QUEUE_OFFSET + size_t(TCAP) * QROW * sizeof(unsigned short));
constexpr int REC_CAP = int((SMEM_LIMIT - REC_OFFSET) / (REC_N * sizeof(float4)));
// a tile read from global memory keeps 32-bit queue entries in the idle staging area
static_assert(size_t(TCAP) * QROW * sizeof(int) <= size_t(REC_CAP) * REC_N * sizeof(float4), "queue in the staging area");
static_assert(CH * LPT <= REC_CAP, "reads past a column stay in the staging area");
static_assert(QROW * sizeof(unsigned short) >= 51 * sizeof(float) && QROW >= QCAP, "a target's sums fit its queue row");
static_assert(TILE_HALO_MAX + NHC <= REC_CAP, "the estimated halo and its parity gaps fit the staging area");
static_assert(REC_CAP < 65536, "16-bit queue entries");

__device__ __forceinline__ unsigned smem_u32(const void *p) { return unsigned(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(unsigned long long *b, unsigned n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long *b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned long long *b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_to_smem(void *dst, const void *src, unsigned bytes, unsigned long long *b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(b))
                 : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Named barriers, each passed once per tile (a warp that waits at one takes no
// issue slots; fifteen warps polling the mbarrier took a third of them):
//   BAR_FULL   everybody: the tile's records have landed and its tables are
//              built, and the compute warps are done with the tile before
//   BAR_READ   the compute warps (which only arrive) have read their last
//              record of the tile; the producer waits for it
// and one among the compute warps alone, with an AND of a predicate.
constexpr int BAR_FULL = 1, BAR_READ = 2, BAR_COMPUTE = 3;
// (the aligned forms: a warp's lanes arrive together)
template <int ID> __device__ __forceinline__ void bar_arrive() {
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(NTHREADS) : "memory");
}
template <int ID> __device__ __forceinline__ void bar_wait() {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(NTHREADS) : "memory");
}
__device__ __forceinline__ bool compute_and(bool v) {
    unsigned r;
    __syncwarp();
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(r)
                 : "r"(unsigned(v)), "n"(BAR_COMPUTE), "n"(NCOMP)
                 : "memory");
    return r != 0;
}

__device__ __forceinline__ int warp_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// One pass over the targets of a tile: lane pair (tt, sl) serves target tt
// from its candidates to its reduced sums.  Returns the target's sorted index
// (-1: none) and its results in res[0..19] (19: neighbours in support).
template <bool CSPM, int COND, bool STAGED>
__device__ __forceinline__ int process_target(const StepArgs &a, const TileTab &tab, unsigned short *queue,
                                              float4 *sarr, int ntg, int tt, int sl, int rounds, float *res) {
    const Params &P = a.p;
    using Q = typename std::conditional<STAGED, unsigned short, int>::type;
    // the records: P at RF, V, A, B, R, C interleaved from RF + rn
    const float4 *__restrict__ RF = STAGED ? sarr : a.r.f[REC_P];
    const int rn = STAGED ? REC_CAP : P.n_init;
    const float4 *__restrict__ X = RF + rn;
    const bool valid = tt < ntg;
    const TileGeo G = tile_geo(P, tab.tile, tab.depth);
    // the target: its column, sorted index, record and cell
    int i = -1, si = 0, c = 0, gk = G.Z0;
    if (valid) {
#pragma unroll
        for (int k = NTC / 2; k >= 1; k >>= 1)
            if (tab.tpref[c + k] <= tt) c += k;
        i = tab.tsrt[c] + (tt - tab.tpref[c]);
        si = tab.trec[c] + (tt - tab.tpref[c]);
        if (!bounds_ok(a.clk, i, P.n_init)) i = 0;
        if (!bounds_ok(a.clk, si, rn)) si = 0;
        const int *cs = tab.cs[(c / TY + 2) * HY + (c % TY + 2)];
        int k = G.Z0 - G.zl;
        while (k < G.nzr - 2 && cs[k + 1] <= si) k++;
        gk = G.zl + k;
    }
    Target I;
    float h, fac;
    {
        target_of<CSPM, COND>(RF[si], X + si * REC_X, I);
        h = I.ch.y;
        I.h1 = 1.0f / h;
        fac = 0.31830988618379067f * I.h1 * I.h1 * I.h1;
        I.art = P.wdeltap > 0.f;
        I.c_art = fac * P.inv_wdeltap;
    }
    // ---- the candidates: lane sl takes the records of parity sl of each
    // stencil column.  Without PSE (which sums every candidate of the 5x5x5 cells) the
    // cells that lie wholly beyond the target's support radius are left out
    // (org.w = the margin in cells, 0 = off; org.xyz = the grid origin of this
    // step's hash): in cell units, a column's x-y box and a cell's z extent,
    // each widened by the margin, against the sphere of radius 2h around the
    // target.  Only out-of-support candidates go, in the same order, so the
    // queue and every sum over it are unchanged.  Cell 0 of an axis also holds
    // positions up to one cell below the origin (the hash truncates toward 0).
    constexpr bool PRUNE = COND != MFREE_COND_PSE;
    const float4 org = tab.org;
    const bool prune = PRUNE && org.w != 0.f;
    const int klo = max(gk - 2, 0), khi = min(gk + 2, P.gnz - 1);
    const int *cs0 = tab.cs[(c / TY) * HY + (c % TY)];  // the stencil's first column
    auto scan = [&](auto &&fn) {
        if (!valid) return;
        const int gi = G.X0 + c / TY, gj = G.Y0 + c % TY;
        float ux = 0.f, uy = 0.f, uz = 0.f, rc2 = 0.f;
        if (prune) {
            const float ic = 1.0f / P.gdx;
            ux = (-I.nxy.x - org.x) * ic;
            uy = (-I.nxy.y - org.y) * ic;
            uz = (-I.nz - org.z) * ic;
            const float rc = 2.0f * h * ic;
            rc2 = rc * rc;
        }
#pragma unroll 1
        for (int ca = 0; ca < 5; ca++) {
            const int cx = gi + ca - 2;
            const float ex = fmaxf(0.f, fmaxf((cx == 0 ? -1.f : float(cx)) - org.w - ux, ux - (float(cx + 1) + org.w)));
            const float rx2 = rc2 - ex * ex;
            const int *row = cs0 + ca * (HY * CSROW) - G.zl;
            // the record ranges of five columns at once: their latencies overlap
            int js[5], je[5];
#pragma unroll
            for (int cb = 0; cb < 5; cb++) {
                int k0 = klo, k1 = khi;
                if (prune) {
                    const int cy = gj + cb - 2;
                    const float ey = fmaxf(0.f, fmaxf((cy == 0 ? -1.f : float(cy)) - org.w - uy, uy - (float(cy + 1) + org.w)));
                    const float rz2 = rx2 - ey * ey;
                    float z;
                    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(z) : "f"(fmaxf(rz2, 0.f)));  // the margin covers its error
                    const float zr = z + org.w;
                    int z1 = __float2int_rd(uz + zr);
                    if (z1 < 0 && uz + zr > -1.f) z1 = 0;
                    k0 = max(k0, __float2int_rd(uz - zr));
                    k1 = rz2 > 0.f ? min(k1, z1) : -1;
                }
                const bool some = k1 >= k0;
                const int j0 = row[cb * CSROW + (some ? k0 : klo)], j1 = row[cb * CSROW + (some ? k1 : klo) + 1];
                js[cb] = j0 + ((j0 ^ sl) & 1);
                je[cb] = some ? j1 : 0;
            }
#pragma unroll
            for (int cb = 0; cb < 5; cb++) fn(js[cb], je[cb]);
        }
    };
    // ---- support test, PSE, queue (filled by lane 0 from its start, by lane 1 from its end)
    const float pse_k = -1.44269504088896341f * I.h1 * I.h1;  // exp(-r^2/h^2) = 2^(pse_k r^2)
    const float four_h2 = __fmul_rn(__fmul_rn(4.0f, h), h);
    Q *const qrow = (STAGED ? reinterpret_cast<Q *>(queue) : reinterpret_cast<Q *>(sarr)) + (threadIdx.x / LPT) * QROW;
    Q *qp = sl == 0 ? qrow : qrow + (QCAP - 1);
    const int qstep = sl == 0 ? 1 : -1;
    int qn = 0;
    float pse = 0.f;
    // the in-support test of the reference's neighbour count (kernels.cuh:41): the
    // unfused sum of squares, 1e-8 <= r^2 < 4 h^2, the lower bound a double
    // there: r^2 > 9.99999994e-9f, the largest float below it
    auto dist2 = [&](const float4 Pj) {
        const float2 d = add2(lo2(Pj), I.nxy);
        const float dz = Pj.z + I.nz;
        const float2 m = mul2(d, d);
        return __fadd_rn(__fadd_rn(m.x, m.y), __fmul_rn(dz, dz));
    };
    scan([&](int j, int je) {
        // CH candidates a lane at once, without a branch: records past the
        // column's end are read (they lie inside the record arrays) and masked
#pragma unroll 1
        for (; j < je; j += CH * LPT) {
            if (!bounds_ok(a.clk, j, rn)) continue;
            float4 p[CH];
            float2 tv[CH];
#pragma unroll
            for (int k = 0; k < CH; k++) {
                p[k] = RF[j + k * LPT];
                if (COND == MFREE_COND_PSE) tv[k] = hi2(X[min(j + k * LPT, rn - 1) * REC_X + (REC_C - 1)]);
            }
            const bool room = qn <= QCAP - CH;
#pragma unroll
            for (int k = 0; k < CH; k++) {
                const float r2 = dist2(p[k]);
                const bool have = j + k * LPT < je;
                if (COND == MFREE_COND_PSE) {
                    float e;
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(pse_k * r2));
                    const float v = fmaf((tv[k].x - I.T) * tv[k].y, e, pse);
                    pse = have ? v : pse;
                }
                const bool in = have && !(r2 >= four_h2) && r2 > 9.99999994e-9f;
                if (in && room) *qp = Q(j + k * LPT);
                if (in) qp += qstep;
                qn += in ? 1 : 0;
            }
        }
    });
    __syncwarp();
    const int qo = __shfl_xor_sync(0xffffffffu, qn, 1);  // the other lane's neighbours
    const int nq = qn + qo;
    const bool queued = nq <= QCAP && max(qn, qo) <= QCAP - CH;
    if (COND == MFREE_COND_PSE) pse += __shfl_xor_sync(0xffffffffu, pse, 1);
    // ---- pair body over the in-support neighbours: four lanes a target, eight
    // targets of the warp at a time; lanes 0 and 1 take the queue's front part,
    // lanes 2 and 3 its back part.  A target's entries are mostly neighbouring
    // records, which lie on different banks, so more lanes a target mean fewer
    // conflicts, and a longer reduction with more idle lanes at the end: pair
    // kernel on the 1M step 1288 / 1258 / 1314 us with two / four / eight.
    // A target's sums replace its queue row.
    const int lane = threadIdx.x & 31;
    const PairConst PC{0.25f * P.av_eta * P.av_eta, -0.5f * P.av_alpha, 0.5f * P.av_beta};
    {
        const int l = lane % PPT, back = l >= PPT / 2, lh = l % (PPT / 2);
        Q *const wrow = qrow - size_t(lane / LPT) * QROW;  // the warp's first row
#pragma unroll 1
        for (int rd = 0; rd < rounds; rd++) {
            const int tl = rd * TPR + lane / PPT, own = tl * LPT;
            const int n_f = __shfl_sync(0xffffffffu, queued && valid ? qn : 0, own);
            const int n_b = __shfl_sync(0xffffffffu, queued && valid ? qn : 0, own + 1);
            const int sj = __shfl_sync(0xffffffffu, si, own);
            const unsigned busy = __ballot_sync(0xffffffffu, n_f + n_b > 0);
            if (busy == 0) continue;
            Target J;
            J.h1 = __shfl_sync(0xffffffffu, I.h1, own);
            J.c_art = __shfl_sync(0xffffffffu, I.c_art, own);
            J.art = I.art;
            target_of<CSPM, COND>(RF[sj], X + sj * REC_X, J);
            Q *const row = wrow + tl * QROW;
            const Q *qe = back ? row + (QCAP - 1) - lh : row + lh;
            const int qd = back ? -(PPT / 2) : PPT / 2, cnt = back ? n_b : n_f;
            Sums<CSPM, COND> S;
            S.zero();
            // the next entry's index and position are read ahead
            int m = lh;
            int j = m < cnt ? int(*qe) : sj;
            float4 Pj = RF[j];
            int jn = m + PPT / 2 < cnt ? int(qe[qd]) : j;
#pragma unroll 1
            for (; m < cnt; m += PPT / 2) {
                const float4 Pc = Pj;
                const int jc = j;
                j = jn;
                Pj = RF[j];
                qe += qd;
                jn = m + PPT < cnt ? int(qe[qd]) : j;
                pair_body<CSPM, COND>(PC, J, Pc, X + jc * REC_X, S);
            }
            __syncwarp();
            S.template reduce_to<PPT>(reinterpret_cast<float *>(row), l, n_f + n_b > 0);
        }
    }
    __syncwarp();
    Sums<CSPM, COND> S;
    S.zero();
    float *const srow = reinterpret_cast<float *>(qrow);
    if (__any_sync(0xffffffffu, !queued)) {  // queues that overflowed: the neighbours are found again by the same scan
        if (!queued)
            scan([&](int j, int je) {
#pragma unroll 1
                for (; j < je; j += LPT) {
                    if (!bounds_ok(a.clk, j, rn)) continue;
                    const float4 Pj = RF[j];
                    const float r2 = dist2(Pj);
                    if (!(r2 >= four_h2) && r2 > 9.99999994e-9f) pair_body<CSPM, COND>(PC, I, Pj, X + j * REC_X, S);
                }
            });
        __syncwarp();
        S.template reduce_to<LPT>(srow, sl, !queued);
        __syncwarp();
    }
    if (nq > 0 && valid) S.load(srow);
    const float4 Ai = X[si * REC_X + (REC_A - 1)], Bi = X[si * REC_X + (REC_B - 1)], Ri = X[si * REC_X + (REC_R - 1)],
                 Ci = X[si * REC_X + (REC_C - 1)];
    finish_sums<CSPM, COND>(S, I, fac, Ai, Bi, Ri, Ci, res);
    if (COND == MFREE_COND_PSE) res[18] = pse;
    if (COND == MFREE_COND_NONE) res[18] = 0.f;
    res[19] = __int_as_float(nq);
    return i;
}

// The producer warp: takes the entries of the tile list (the non-empty tiles
// of every scene) one after the other; for each it builds the tables in the
// buffer that the compute warps have left, waits until they have read the last
// record of the tile before, and issues the staging copies.  The next entry
// is claimed after the copies, so its round trip is hidden.
__device__ __forceinline__ void produce(const BatchTable &T, BlockSmem &sm, StepArgs *sa, float4 *sarr, int lane) {
    int slot_scene[2] = {-1, -1};  // scenes whose arguments the two slots hold
    int slot = 0;
    int2 e = make_int2(0, -1);
    // the first entry is the block's own, the others are claimed
    const int list_n = min(*T.tile_count, T.tile_max);
    if (lane == 0 && int(blockIdx.x) < list_n) e = T.tile_list[blockIdx.x];
    auto claim = [&] {
        if (lane == 0) {
            const int k = atomicAdd(T.tile_next, 1) + int(gridDim.x);
            e = k < list_n ? T.tile_list[k] : make_int2(0, -1);
        }
    };
#pragma unroll 1
    for (int n = 0;; n++) {
        const int t = __shfl_sync(0xffffffffu, e.x, 0), sd = __shfl_sync(0xffffffffu, e.y, 0);
        const int s = sd < 0 ? -1 : sd >> 4, depth = sd & 15;
        TileTab &tab = sm.tab[n & 1];
        if (s < 0) {
            if (n > 0) bar_wait<BAR_READ>();
            if (lane == 0) tab.scene = -1;
            bar_wait<BAR_FULL>();
            return;
        }
        if (s != slot_scene[slot]) {  // the other slot: the compute warps still use this one
            slot ^= 1;
            if (s != slot_scene[slot]) {
                const StepArgs *a0 = T.args + 2 * s;
                const int4 *src = reinterpret_cast<const int4 *>(a0 + (a0->clk->parity & 1));
                int4 *d = reinterpret_cast<int4 *>(reinterpret_cast<char *>(sa) + slot * ARGS_SIZE);
                for (int k = lane; k < int(sizeof(StepArgs) / 16); k += 32) d[k] = src[k];
                __syncwarp();
                slot_scene[slot] = s;
            }
        }
        const StepArgs &a = *reinterpret_cast<const StepArgs *>(reinterpret_cast<char *>(sa) + slot * ARGS_SIZE);
        const Params &P = a.p;
        const int nx = P.gnx, ny = P.gny, nz = P.gnz;
        const TileGeo G = tile_geo(P, t, depth);
        const int *__restrict__ first = a.s.first;
        // halo cell starts (sorted indices), each lane's loads in flight together
        constexpr int NCS = NHC * CSROW / 32;
        static_assert(NHC * CSROW % 32 == 0, "whole warps of cell starts");
        int csv[NCS];
        {
#pragma unroll
            for (int r = 0; r < NCS; r++) {
                const int x = lane + r * 32;
                const int c = x / CSROW, k = x - c * CSROW;
                const int cx = G.X0 - 2 + c / HY, cy = G.Y0 - 2 + c % HY;
                csv[r] = 0;
                if (k < G.nzr && cx >= 0 && cx < nx && cy >= 0 && cy < ny) {
                    const int fi = (cx * ny + cy) * nz + G.zl + k;
                    if (bounds_ok(a.clk, fi, (long long)P.num_cell + 1)) csv[r] = first[fi];
                }
            }
#pragma unroll
            for (int r = 0; r < NCS; r++) (&tab.cs[0][0])[lane + r * 32] = csv[r];
        }
        __syncwarp();
        // the halo columns (lane l: columns 2 l and 2 l + 1), their staged offsets
        int hs[2], hl[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int c = 2 * lane + k;
            hs[k] = tab.cs[c][0];
            hl[k] = tab.cs[c][G.nzr - 1] - hs[k];
            // bounds-checked build: a column whose range lies outside the
            // record arrays is counted and left out
            if (!range_ok(a.clk, hs[k], hl[k], P.n_init)) {
                hl[k] = 0;
                for (int q = 0; q < CSROW; q++) tab.cs[c][q] = 0;
                hs[k] = 0;
            }
        }
        // a record's staged index has the parity of its sorted index (the lanes
        // of a target share its candidates by that parity, so its sums depend
        // neither on the tile it falls in nor on the pruning): a column takes
        // an even number of slots and starts at its own parity
        const int w0 = (hl[0] + (hs[0] & 1) + 1) & ~1, w1 = (hl[1] + (hs[1] & 1) + 1) & ~1;
        const int inc = warp_scan(w0 + w1, lane);
        const int ho[2] = {inc - w0 - w1 + (hs[0] & 1), inc - w1 + (hs[1] & 1)};
        const bool staged = __shfl_sync(0xffffffffu, inc, 31) <= REC_CAP;
        const int total = __reduce_add_sync(0xffffffffu, hl[0] + hl[1]);  // records to copy
        __syncwarp();
        // the target columns: cells Z0 .. Z0 + depth - 1
        int len = 0;
        if (lane < NTC) {
            const int cx = G.X0 + lane / TY, cy = G.Y0 + lane % TY;
            const int *cs = tab.cs[(lane / TY + 2) * HY + (lane % TY + 2)];
            int s0 = 0;
            if (cx < nx && cy < ny && G.Z0 < nz) {
                s0 = cs[G.Z0 - G.zl];
                len = cs[min(G.Z0 + depth - 1, nz - 1) + 1 - G.zl] - s0;
            }
            tab.tsrt[lane] = s0;
        }
        const int ti = warp_scan(len, lane);
        const int c0 = max(__ffs(__ballot_sync(0xffffffffu, len > 0)) - 1, 0);  // first column with a target
        if (lane < NTC) tab.tpref[lane] = ti - len;
        if (lane == 31) tab.tpref[NTC] = ti;
        __syncwarp();
        if (staged) {  // the cell starts as record indices: every lane shifts those it holds
#pragma unroll
            for (int k = 0; k < 2; k++) tab.shift[2 * lane + k] = hl[k] > 0 ? ho[k] - hs[k] : int(0x80000000);
            __syncwarp();
#pragma unroll
            for (int r = 0; r < NCS; r++) {
                const int x = lane + r * 32, d = tab.shift[x / CSROW];
                if (d != int(0x80000000)) (&tab.cs[0][0])[x] = csv[r] + d;
            }
        }
        __syncwarp();
        if (lane < NTC) tab.trec[lane] = tab.cs[(lane / TY + 2) * HY + (lane % TY + 2)][max(0, min(G.Z0 - G.zl, CSROW - 1))];
        if (lane == 0) {
            tab.tile = t;
            tab.depth = depth;
            tab.scene = s;
            tab.args = slot;
            tab.total = total;
            tab.staged = staged ? 1 : 0;
            tab.nzr = G.nzr;
            tab.rec0 = tab.cs[(c0 / TY + 2) * HY + (c0 % TY + 2)][G.Z0 - G.zl];
            float4 org = make_float4(0.f, 0.f, 0.f, 0.f);
            const float md = __uint_as_float(a.clk->max_disp);
            if (!P.full_stencil && md <= PRUNE_DISP_MAX) {
                const float *gm = P.grid_moving ? a.clk->grid_min : P.grid_min0;
                org = make_float4(gm[0], gm[1], gm[2], md + PRUNE_SLACK);
            }
            tab.org = org;
        }
        if (n > 0) bar_wait<BAR_READ>();
        const bool copy = staged && total > 0;
        if (lane == 0)
            mbar_expect(&sm.bar, copy ? unsigned(total) * unsigned(REC_N * sizeof(float4)) + unsigned(P.stage_extra) : 0u);
        __syncwarp();
        if (copy) {
            // two copies a column: its P records to sarr, the interleaved rest
            // to sarr + REC_CAP (the record arrays are one allocation: P from
            // f[REC_P], the rest from f[REC_P] + n_init)
            const float4 *gbase = a.r.f[REC_P];
#pragma unroll
            for (int k = 0; k < 2; k++)
                if (hl[k] > 0) {
                    bulk_to_smem(sarr + ho[k], gbase + hs[k], unsigned(hl[k]) * unsigned(sizeof(float4)), &sm.bar);
                    bulk_to_smem(sarr + REC_CAP + ho[k] * REC_X, gbase + size_t(P.n_init) + size_t(hs[k]) * REC_X,
                                 unsigned(hl[k] * REC_X) * unsigned(sizeof(float4)), &sm.bar);
                }
        }
        claim();
        bool ok = true;
        auto landed = [&] {
            const long long t_wait = clock64();
            while (!mbar_try(&sm.bar, unsigned(n & 1)))
                if (clock64() - t_wait > WAIT_CYCLES) return false;
            return true;
        };
        ok = __all_sync(0xffffffffu, landed());
        if (!ok && lane == 0) {
            // the copies did not complete in time: count it (the host reports
            // MFREE_ERR_TIMEOUT); everybody leaves the kernel
            atomicAdd(&a.clk->staging_timeouts, 1);
            sm.fail = 1;
        }
        bar_wait<BAR_FULL>();
        if (!ok) {
            landed();  // wait once more (bounded) for the copies in flight to land
            return;
        }
    }
}

// Persistent (one block per SM) over the tiles of every scene of the table
// (one queue).
template <bool CSPM, int COND, bool PREC>
__global__ void __launch_bounds__(NTHREADS, 1) kb_interact(BatchTable T) {
    extern __shared__ __align__(128) unsigned char dyn[];
    BlockSmem &sm = *reinterpret_cast<BlockSmem *>(dyn);
    StepArgs *sa = reinterpret_cast<StepArgs *>(dyn + ARGS_OFFSET);
    unsigned short *queue = reinterpret_cast<unsigned short *>(dyn + QUEUE_OFFSET);
    float4 *sarr = reinterpret_cast<float4 *>(dyn + REC_OFFSET);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    begin_after();
    if (threadIdx.x == 0) {
        sm.fail = 0;
        mbar_init(&sm.bar, 1);
    }
    fence_proxy_async();
    __syncthreads();
    if (warp == NCOMP / 32) {
        produce(T, sm, sa, sarr, lane);
        return;
    }
    const int sl = lane % LPT;
#pragma unroll 1
    for (int n = 0;; n++) {
        bar_wait<BAR_FULL>();
        const TileTab &tab = sm.tab[n & 1];
        if (tab.scene < 0 || sm.fail) return;
        mbar_try(&sm.bar, unsigned(n & 1));  // the phase is complete: each thread observes the copies itself
        const StepArgs &a = *reinterpret_cast<const StepArgs *>(reinterpret_cast<char *>(sa) + tab.args * ARGS_SIZE);
        const int ntg = tab.tpref[NTC];
        const bool staged = tab.staged != 0;
        // PSE: every term carries T_j - T_i, so when all staged records of the
        // tile hold the same temperature (and finite positions and volumes)
        // each term is exactly +0 and so is every target's sum; such a tile runs
        // the variant without conduction terms, on the pruned stencil, with the
        // same results.
        bool pse_zero = false;
        if (COND == MFREE_COND_PSE && staged && tab.total > 0 && !a.p.full_stencil) {
            const float4 *rc = sarr + REC_CAP + (REC_C - 1);
            const float T0 = rc[tab.rec0 * REC_X].z;
            bool u = true;
            for (int hc = warp; hc < NHC; hc += NCOMP / 32)
                for (int k = tab.cs[hc][0] + lane; k < tab.cs[hc][tab.nzr - 1]; k += 32) {
                    const float4 c = rc[k * REC_X], p = sarr[k];
                    u = u && c.z == T0 && isfinite(c.w) && isfinite(p.x) && isfinite(p.y) && isfinite(p.z);
                }
            pse_zero = compute_and(u);
            if (pse_zero && threadIdx.x == 0) atomicAdd(&a.clk->pse_zero_targets, (unsigned long long)ntg);
        }
#pragma unroll 1
        for (int t0 = 0;; t0 += TCAP) {
            float res[NRES];
            int i = -1;
            // targets a warp: its rounds of the pair pass (eight targets each) are
            // what a tile waits for, so few targets are spread over all warps
            const int rounds = min(32 / LPT / TPR, (min(ntg - t0, TCAP) + NCOMP / PPT - 1) / (NCOMP / PPT));
            const int tw = t0 + warp * (TPR * rounds);  // the warp's first target
            if (tw < min(ntg, t0 + TCAP)) {
                const int tt = lane / LPT < TPR * rounds ? tw + lane / LPT : ntg;
                if (staged && COND == MFREE_COND_PSE && pse_zero)
                    i = process_target<CSPM, MFREE_COND_NONE, true>(a, tab, queue, sarr, ntg, tt, sl, rounds, res);
                else if (staged)
                    i = process_target<CSPM, COND, true>(a, tab, queue, sarr, ntg, tt, sl, rounds, res);
                else
                    i = process_target<CSPM, COND, false>(a, tab, queue, sarr, ntg, tt, sl, rounds, res);
            }
            const bool last = t0 + TCAP >= ntg;
            if (last) {
                // the last reads of the staged halo: order them before the next
                // tile's bulk writes, which the producer issues after this barrier
                fence_proxy_async();
                bar_arrive<BAR_READ>();
            }
            if (i >= 0 && sl == 0) epilogue<PREC, COND>(a, i, res);
            if (last) break;
        }
    }
}

// ------------------------------------------------------------ dispatch --
template <bool CSPM, int COND, bool PREC> struct Variant {
    static cudaError_t batch(const BatchTable &T, int grid, cudaStream_t s) {
        auto kern = kb_interact<CSPM, COND, PREC>;
        if (grid <= 0)  // prepare only: raise the shared-memory limit (outside any graph capture)
            return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
        return launch_after(kern, grid, NTHREADS, SMEM_LIMIT, s, T);
    }
};

// calls fn(Variant<...>{}) for the variant of the options
template <class F> static cudaError_t with_variant(bool cspm, int cond, bool prec, F &&fn) {
#define MFREE_CASE(C, CO, PR) \
    if (cspm == C && cond == CO && prec == PR) return fn(Variant<C, CO, PR>{});
    MFREE_CASE(false, MFREE_COND_NONE, false)
    MFREE_CASE(false, MFREE_COND_BROOKSHAW, false)
    MFREE_CASE(false, MFREE_COND_PSE, false)
    MFREE_CASE(true, MFREE_COND_NONE, false)
    MFREE_CASE(true, MFREE_COND_BROOKSHAW, false)
    MFREE_CASE(true, MFREE_COND_PSE, false)
    MFREE_CASE(false, MFREE_COND_NONE, true)
    MFREE_CASE(false, MFREE_COND_BROOKSHAW, true)
    MFREE_CASE(false, MFREE_COND_PSE, true)
    MFREE_CASE(true, MFREE_COND_NONE, true)
    MFREE_CASE(true, MFREE_COND_BROOKSHAW, true)
    MFREE_CASE(true, MFREE_COND_PSE, true)
#undef MFREE_CASE
    return cudaErrorInvalidValue;
}

}  // namespace mfree
