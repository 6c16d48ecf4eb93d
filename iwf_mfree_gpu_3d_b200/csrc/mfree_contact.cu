// mfree_contact.cu -- end of the step: rigid-tool contact and the work that
// follows it for the particles inside a tool box.
//
// Reference path replaced (src/leap_frog.cu:173-188):
//   tool_3d_gpu::update_tool + do_update_tool   tool_3d_gpu.cu:74-99,907-948 (vertices
//                                               p_init + v t are formed on the fly)
//   do_compute_contact_forces (spatial hashing, safe) tool_3d_gpu.cu:585-681
//       establish_contact_by_ray / _by_normal, comp_closest_point,
//       triangle_ray_intersect                  tool_3d_gpu.cu:101-444
//   do_compute_contact_forces_n2 (exhaustive)   tool_3d_gpu.cu:455-583
//   tool_forces (atomicAdd)                     tool_3d_gpu.cu:30-69 -- here a
//                                               fixed-order block reduction
//   do_material_fric_heat_gen                   actions_gpu.cu:192-220
//   do_boundary_conditions(_thermal)            actions_gpu.cu:451-487
//   do_move_tool_particles (blanked tail)       actions_gpu.cu:55-68
//
// The pair kernel's epilogue has finished every particle outside the tool
// boxes and marked the others in a bitmap; here each of those is taken by a
// group of 2, 8 or 32 lanes, which share the triangles of the ray test and of
// the closest-point search.  These are chains of dependent loads.  One thread
// per particle walked some hundred triangles of a 1,280-triangle mesh one
// after the other: 500 us a step with five of them on 10,000 particles.  The
// bitmap's words are dealt to the blocks in turn, so that neighbouring
// particles, which are in contact together, spread over the SMs; and it takes
// the place of a pass over the positions (4.1M particles: 120 us).
#include "mfree_geom.h"
#include "mfree_kernels.cuh"

namespace mfree {

namespace {

// vector algebra of the contact code on the shared float 3-vector
using V3 = Vec3f;
__device__ __forceinline__ V3 v3(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return vadd(a, b); }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return vsub(a, b); }
__device__ __forceinline__ V3 operator*(float s, V3 a) { return vscale(s, a); }
__device__ __forceinline__ float dot(V3 a, V3 b) { return vdot(a, b); }
__device__ __forceinline__ V3 cross(V3 a, V3 b) { return vcross(a, b); }
__device__ __forceinline__ float len(V3 a) { return vlength(a); }
__device__ __forceinline__ V3 ld(const float4 *p, int i) {
    float4 v = p[i];
    return {v.x, v.y, v.z};
}

// current vertex p_init + v t (do_update_tool)
__device__ __forceinline__ V3 vert(const ToolDev &T, const float4 *p, int i, float t) {
    float4 v = p[i];
    return {v.x + T.vel[0] * t, v.y + T.vel[1] * t, v.z + T.vel[2] * t};
}

// closest point on triangle k and the normal of the feature it lies on
// (comp_closest_point, tool_3d_gpu.cu:141-212; the geometry is shared with the
// host setup in mfree_geom.h)
__device__ void closest_point(const ToolDev &T, int k, float t, V3 qp, V3 &cp, V3 &np) {
    switch (closest_on_triangle(vert(T, T.p1, k, t), vert(T, T.p2, k, t), vert(T, T.p3, k, t), qp, cp)) {
        case TF_V1: np = ld(T.np1, k); break;
        case TF_V2: np = ld(T.np2, k); break;
        case TF_V3: np = ld(T.np3, k); break;
        case TF_E12: np = ld(T.ne1, k); break;
        case TF_E23: np = ld(T.ne2, k); break;
        case TF_E31: np = ld(T.ne3, k); break;
        default: np = ld(T.n, k); break;
    }
}

// Moller-Trumbore along +z (triangle_ray_intersect, tool_3d_gpu.cu:248-280)
__device__ bool ray_z(const ToolDev &T, int k, float t, V3 o, float &tt) {
    const float EPS = 0.0000001f;
    V3 v0 = vert(T, T.p1, k, t), v1 = vert(T, T.p2, k, t), v2 = vert(T, T.p3, k, t);
    V3 e1 = v1 - v0, e2 = v2 - v0;
    V3 dir = v3(0.f, 0.f, 1.f);
    V3 h = cross(dir, e2);
    float a = dot(e1, h);
    if (a > -EPS && a < EPS) return false;
    float f = 1.f / a;
    V3 s = o - v0;
    float u = f * dot(s, h);
    if (u < 0.f || u > 1.f) return false;
    V3 q = cross(s, e1);
    float v = f * dot(dir, q);
    if (v < 0.f || u + v > 1.f) return false;
    tt = f * dot(e2, q);
    return tt > EPS;
}

__device__ __forceinline__ void unhash(const ToolDev &T, const ToolClock &B, V3 p, int &ix, int &iy, int &iz) {
    // (unsigned int) cast of unhash_pos (tool_3d_gpu.cu:101-107), kept inside the grid
    ix = int(min((unsigned)((p.x - B.bbmin[0]) / T.dx), unsigned(T.nx - 1)));
    iy = int(min((unsigned)((p.y - B.bbmin[1]) / T.dx), unsigned(T.ny - 1)));
    iz = int(min((unsigned)((p.z - B.bbmin[2]) / T.dx), unsigned(T.nz - 1)));
}

// A group of G neighbouring lanes of a warp that serves one particle
template <int G> struct Group {
    static constexpr int SIZE = G;
    int l;          // the lane within the group
    unsigned mask;  // the group's lanes
    __device__ __forceinline__ Group(int lane)
        : l(lane % G), mask(G == 32 ? 0xffffffffu : ((1u << (G % 32)) - 1u) << (lane / G * G)) {}
    template <class F> __device__ __forceinline__ unsigned fold(unsigned v, F &&f) const {
#pragma unroll
        for (int o = G / 2; o >= 1; o >>= 1) v = f(v, __shfl_xor_sync(mask, v, o, G));
        return v;
    }
    __device__ __forceinline__ unsigned least(unsigned v) const {
        return fold(v, [](unsigned a, unsigned b) { return min(a, b); });
    }
    __device__ __forceinline__ unsigned sum(unsigned v) const {
        return fold(v, [](unsigned a, unsigned b) { return a + b; });
    }
    __device__ __forceinline__ int from(int v, int lane) const { return __shfl_sync(mask, v, lane, G); }
};

// +z ray parity over the tri-grid column (establish_contact_by_ray, :382-444),
// a group per particle.  A column's cells are consecutive, so its triangles from
// the particle's cell up are one range; the hit's cell is looked up on a hit only.
template <int G> __device__ bool inside_by_ray(const ToolDev &T, const ToolClock &B, float t, V3 qp, const Group<G> &g) {
    int ix, iy, iz;
    unhash(T, B, qp, ix, iy, iz);
    const int *cells = T.cells + (ix * T.ny + iy) * T.nz;
    const int k0 = cells[iz], k1 = cells[T.nz];
    unsigned ni = 0;
    for (int k = k0 + g.l; k < k1; k += G) {
        float tt;
        if (ray_z(T, k, t, qp, tt)) {
            V3 ip = qp + tt * v3(0.f, 0.f, 1.f);
            int cz = iz;
            while (cells[cz + 1] <= k) cz++;
            float lox = B.bbmin[0] + ix * T.dx, loy = B.bbmin[1] + iy * T.dx, loz = B.bbmin[2] + cz * T.dx;
            float hix = B.bbmin[0] + (ix + 1) * T.dx, hiy = B.bbmin[1] + (iy + 1) * T.dx,
                  hiz = B.bbmin[2] + (cz + 1) * T.dx;
            if (lox <= ip.x && ip.x < hix && loy <= ip.y && ip.y < hiy && loz <= ip.z && ip.z < hiz) ni++;
        }
    }
    __syncwarp(g.mask);
    return (g.sum(ni) % 2) != 0;
}

// the closest triangle so far of a lane, and of the group: the smallest squared
// distance, the earliest in visiting order (seq) where distances are equal --
// the triangle that a serial search with "closer than" keeps
struct Closest {
    float dd;
    int k;
    unsigned seq;  // 0: earlier than whatever is visited next
    __device__ __forceinline__ void test(const ToolDev &T, int kk, unsigned sq, float t, V3 qp) {
        V3 c, n;
        closest_point(T, kk, t, qp, c, n);
        V3 d = c - qp;
        const float x = dot(d, d);
        if (x < dd) { dd = x; k = kk; seq = sq; }
    }
    template <int G> __device__ __forceinline__ void join(const Group<G> &g) {
        __syncwarp(g.mask);
        // (distances are never negative: their bits order as values)
        const unsigned m = g.least(__float_as_uint(dd));
        const unsigned s = g.least(__float_as_uint(dd) == m ? seq : 0xffffffffu);
        // lanes that agree in both hold the same triangle
        const unsigned kk = g.least(__float_as_uint(dd) == m && seq == s ? unsigned(k) : 0xffffffffu);
        k = int(kk);
        dd = __uint_as_float(m);
        seq = 0;
    }
};

// closest triangle by expanding shells until one is non-empty, plus one more
// shell (establish_contact_by_normal, :282-380); bounded by the grid size.  A
// group per particle: a shell is searched as the whole cube around the home
// cell, whose cells are runs along z and so ranges of triangles.  Cells of
// earlier shells cannot win again.  Eight and more lanes share the triangles of
// G runs at a time; two take a run each.
template <int G>
__device__ void closest_by_shells(const ToolDev &T, const ToolClock &B, float t, V3 qp, V3 &cp, V3 &nrm, DevClock *clk,
                                  const Group<G> &g) {
    int ix, iy, iz;
    unhash(T, B, qp, ix, iy, iz);
    Closest best{__int_as_float(0x7f800000), -1, 0xffffffffu};  // DBL_MAX stored in a float
    cp = qp;
    nrm = v3(0.f, 0.f, 0.f);
    bool empty_so_far = true;
    const int cap = max(T.nx, max(T.ny, T.nz)) + 2;
    bool all_done = false;
    int off = 0;
    for (; off <= cap;) {
        const int li = max(ix - off, 0), lj = max(iy - off, 0), lk = max(iz - off, 0);
        const int hi = min(ix + off + 1, T.nx), hj = min(iy + off + 1, T.ny), hk = min(iz + off + 1, T.nz);
        const int nj = hj - lj, runs = (hi - li) * nj;
        unsigned seq0 = 1;  // visiting order: run after run
        bool found = false;
        for (int r0 = 0; r0 < runs; r0 += G) {
            const int r = r0 + g.l;
            int s0 = 0, len = 0;
            if (r < runs) {
                const int *c = T.cells + ((li + r / nj) * T.ny + lj + r % nj) * T.nz;
                s0 = c[lk];
                len = c[hk] - s0;
                if (len > 0 && !bounds_ok(clk, s0 + len - 1, T.num_tris)) len = 0;
            }
            int inc = len;
#pragma unroll
            for (int o = 1; o < G; o <<= 1) {
                const int y = __shfl_up_sync(g.mask, inc, o, G);
                if (g.l >= o) inc += y;
            }
            const int total = g.from(inc, G - 1);
            found |= total > 0;
            if (G >= 8) {
                for (int x0 = 0; x0 < total; x0 += G) {
                    const int x = x0 + g.l;
                    int run = 0;  // the first run that ends beyond x
#pragma unroll
                    for (int o = G / 2; o >= 1; o >>= 1)
                        if (g.from(inc, run + o - 1) <= x) run += o;
                    const int rs = g.from(s0, run), re = g.from(inc, run), rl = g.from(len, run);
                    if (x < total) best.test(T, rs + (x - (re - rl)), seq0 + unsigned(x), t, qp);
                    __syncwarp(g.mask);
                }
            } else {
                for (int x = 0; x < len; x++) best.test(T, s0 + x, seq0 + unsigned(inc - len + x), t, qp);
                __syncwarp(g.mask);
            }
            seq0 += unsigned(total);
        }
        if (found) {
            empty_so_far = false;
            best.join(g);
        }
        if (off == 0) {  // the home cell alone is not a shell
            off = 1;
            continue;
        }
        if (all_done) break;
        off++;
        if (!empty_so_far) all_done = true;
    }
    if (best.k >= 0) closest_point(T, best.k, t, qp, cp, nrm);
    if (off > cap && g.l == 0) atomicAdd(&clk->contact_cap, 1ull);
}

}  // namespace

// contact, friction heat and boundary conditions of particle i, which lies in
// a tool box: by a group (every lane computes the same, the first writes).
// force: where the particle's tool forces go when they are recorded, a stride
// of 3 * FIN_BLOCK floats between tools.
template <int G> __device__ void contact_particle(const StepArgs &a, int i, const Group<G> &g, bool rec, float *force) {
    const Params &P = a.p;
    const State &S = a.b;
    const float4 pos = S.pos4[i];
    float4 fc = S.fc4[i];
    const float t = a.clk->t;
    const float dt = P.dt;
    float4 vel = S.vel4[i], ft = S.ft4[i];
    V3 qp = v3(pos.x, pos.y, pos.z);
    V3 n_last = v3(0.f, 0.f, 0.f);
    for (int k = 0; k < P.num_tools; k++) {
        if (!in_tool_box(a, k, pos.x, pos.y, pos.z)) continue;
        const ToolDev &T = a.tools[k];
        const ToolClock &B = a.clk->tool[k];
        V3 cp, n;
        if (T.hashed) {
            if (!inside_by_ray(T, B, t, qp, g)) continue;
            closest_by_shells(T, B, t, qp, cp, n, a.clk, g);
        } else {
            Closest best{3.402823466e+38f, -1, 0xffffffffu};  // FLT_MAX
            cp = qp;
            n = v3(0.f, 0.f, 0.f);
            for (int kk = g.l; kk < T.num_tris; kk += G) best.test(T, kk, unsigned(kk), t, qp);
            best.join(g);
            if (best.k >= 0) closest_point(T, best.k, t, qp, cp, n);
            if (dot(cp - qp, n) > 0.f) continue;
        }
        // the reference's operation order, divisions included
        // (tool_3d_gpu.cu:630-661): fN = ((-m gN) n) / dt^2 * alpha,
        // kdeltae = ((alpha m) vr) / dt, fT = (fy fstar) / |fstar|
        const float gN = dot(qp - cp, n);
        const float dt2 = dt * dt;
        const V3 mgn = (-P.mass * gN) * n;
        V3 fN = v3(mgn.x / dt2 * T.alpha, mgn.y / dt2 * T.alpha, mgn.z / dt2 * T.alpha);
        V3 fT = v3(0.f, 0.f, 0.f);
        if (T.mu != 0.f) {
            V3 vm = P.friction_tool_vel ? v3(T.vel[0], T.vel[1], T.vel[2]) : v3(0.f, 0.f, 0.f);
            V3 v = v3(vel.x, vel.y, vel.z) - vm;
            V3 vr = v3(v.x - v.x * n.x, v.y - v.y * n.y, v.z - v.z * n.z);
            const V3 amv = (T.alpha * P.mass) * vr;
            V3 kde = v3(amv.x / dt, amv.y / dt, amv.z / dt);
            float fy = T.mu * len(fN);
            V3 fs = v3(ft.x, ft.y, ft.z) - kde;
            float lfs = len(fs);
            if (lfs > fy) {
                const V3 ffs = fy * fs;
                fT = v3(ffs.x / lfs, ffs.y / lfs, ffs.z / lfs);
            } else {
                fT = fs;
            }
        }
        fc.x = fN.x; fc.y = fN.y; fc.z = fN.z;
        ft.x = fT.x; ft.y = fT.y; ft.z = fT.z;
        n_last = n;
        if (rec && g.l == 0) {
            float *f = force + k * (3 * FIN_BLOCK);
            f[0] = fN.x + fT.x;
            f[1] = fN.y + fT.y;
            f[2] = fN.z + fT.z;
        }
    }
    // friction heat (do_material_fric_heat_gen) with the first tool's velocity
    float4 sb = S.sb4[i];
    float T = sb.z;
    if (P.fric_heat) {
        const float fm = sqrtf(ft.x * ft.x + ft.y * ft.y + ft.z * ft.z);
        if (fm != 0.f) {
            const float dx = vel.x - P.tool0_vel[0], dy = vel.y - P.tool0_vel[1], dz = vel.z - P.tool0_vel[2];
            const float dn = dx * n_last.x + dy * n_last.y + dz * n_last.z;
            const float rx = dx - dn, ry = dy - dn, rz = dz - dn;
            const float vm = sqrtf(rx * rx + ry * ry + rz * rz);
            T += P.wp_eta * dt * fm * vm / (P.wp_cp * P.mass);
        }
    }
    // boundary conditions
    const float fixed = S.dsb4[i].w;
    __syncwarp(g.mask);  // every lane has read the state before the first writes it
    if (g.l == 0) {
        if (fixed != 0.f) {
            const float4 bc = S.bc4[i];
            vel.x = bc.x; vel.y = bc.y; vel.z = bc.z;
            fc.x = fc.y = fc.z = 0.f;
            float4 da = S.da4[i], dv = S.dv4[i];
            da.x = da.y = da.z = 0.f;
            dv.x = dv.y = dv.z = 0.f;
            S.da4[i] = da;
            S.dv4[i] = dv;
            if (P.precision) {
                float4 lo = S.lo4[i], lob = S.lo4b[i];
                lo.w = 0.f; lob.x = lob.y = 0.f;
                S.lo4[i] = lo;
                S.lo4b[i] = lob;
            }
        }
        if (P.thermal && fixed == 1.f) T = P.wp_Tinit;
        sb.z = T;
        S.sb4[i] = sb;
        S.vel4[i] = vel;
        S.fc4[i] = fc;
        S.ft4[i] = ft;
        if (P.diagnostics) a.s.nrm[i] = make_float4(n_last.x, n_last.y, n_last.z, 0.f);
    }
}

// Block bid of the scene's nb takes words bid, bid + nb, ... of the contact
// bitmap, eight at a time, and its share of the blanked tail, whose tool
// particles only translate.
__device__ __forceinline__ void finalize_body(const StepArgs &a, int bid) {
    __shared__ int list[FIN_BLOCK], listed;
    __shared__ float force[MAX_TOOLS][FIN_BLOCK][3], red[FIN_BLOCK / 32][3 * MAX_TOOLS];
    const Params &P = a.p;
    const int N = a.clk->n_active;
    const bool rec = a.clk->record != 0;
    const State &S = a.b;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = finalize_blocks(P.n_init), words = (P.n_init + 31) / 32;
    if (bid >= nb) return;
    for (int i = N + bid * FIN_BLOCK + threadIdx.x; i < P.n_init; i += nb * FIN_BLOCK) {
        if (S.fc4[i].w == 1.f) {
            float4 pos = S.pos4[i];
            if (P.precision) {
                float4 lo = S.lo4[i];
                acc_comp(pos.x, lo.x, P.dt, P.tool0_vel[0]);
                acc_comp(pos.y, lo.y, P.dt, P.tool0_vel[1]);
                acc_comp(pos.z, lo.z, P.dt, P.tool0_vel[2]);
                S.lo4[i] = lo;
            } else {
                pos.x = fmaf(P.tool0_vel[0], P.dt, pos.x);
                pos.y = fmaf(P.tool0_vel[1], P.dt, pos.y);
                pos.z = fmaf(P.tool0_vel[2], P.dt, pos.z);
            }
            S.pos4[i] = pos;
        }
    }
    float fsum = 0.f;  // thread 3 k + d: the block's force on tool k in direction d
    for (int w0 = bid; w0 < words; w0 += nb * (FIN_BLOCK / 32)) {
        const int w = w0 + warp * nb;  // the warp's word
        unsigned bits = 0;
        if (w < words) bits = a.s.contact[w];
        __syncwarp();
        if (bits && lane == 0) a.s.contact[w] = 0u;  // for the next step
        const bool contact = (bits >> lane) & 1u;
        if (!__syncthreads_or(contact)) continue;
        if (threadIdx.x == 0) listed = 0;
        if (rec)
            for (int k = threadIdx.x; k < P.num_tools * FIN_BLOCK * 3; k += FIN_BLOCK) (&force[0][0][0])[k] = 0.f;
        __syncthreads();
        // (which group takes which particle shows in no result)
        const unsigned m = __ballot_sync(0xffffffffu, contact);
        int base = 0;
        if (lane == 0 && m) base = atomicAdd(&listed, __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (contact) list[base + __popc(m & ((1u << lane) - 1u))] = threadIdx.x;
        __syncthreads();
        const int n = listed;
        auto take = [&](auto g) {
            constexpr int G = decltype(g)::SIZE;
            for (int c = threadIdx.x / G; c < n; c += FIN_BLOCK / G) {
                const int l = list[c];
                contact_particle<G>(a, (w0 + (l >> 5) * nb) * 32 + (l & 31), g, rec, &force[0][l][0]);
            }
        };
        // Few triangles: as wide a group as lets the block take all its
        // particles at once (8,000 particles and a wedge, a step's contact:
        // 2 lanes 15 us, 32 lanes 32 us).  Many: narrow groups read unrelated
        // triangles and wait for the longest of sixteen searches.  num_tris counts
        // a hashed mesh's triangles once for every cell that holds them.  us by
        // count / 32 lanes, on five small grains, one deep grain (some 500
        // particles in contact) and a large one (some 2,000): 291 triangles
        // 53/30, 54/74, 106/106; 1,345 66/33, 65/81, 128/124; 5,720 87/48,
        // 110/81, 154/124; 320 exhaustive 41/31, 83/71.
        bool many = false;
        for (int k = 0; k < P.num_tools; k++) many |= a.tools[k].num_tris > 512;
        if (many || n <= FIN_BLOCK / 32) take(Group<32>(lane));
        else if (n <= FIN_BLOCK / 8) take(Group<8>(lane));
        else take(Group<2>(lane));
        __syncthreads();
        if (!rec) continue;
        // fixed-order block reduction of the tool forces
        for (int k = 0; k < P.num_tools; k++)
            for (int d = 0; d < 3; d++) {
                float v = force[k][threadIdx.x][d];
                for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) red[warp][3 * k + d] = v;
            }
        __syncthreads();
        if (threadIdx.x < 3 * P.num_tools)
            for (int q = 0; q < FIN_BLOCK / 32; q++) fsum += red[q][threadIdx.x];
    }
    if (rec && threadIdx.x < 3 * P.num_tools) a.s.force_part[size_t(bid) * (3 * MAX_TOOLS) + threadIdx.x] = fsum;
}

// sum of the per-block partials: thread t adds blocks t, t+256, ... in order,
// then a fixed tree over the 256 threads (deterministic for a given grid)
__device__ __forceinline__ void force_final_body(const StepArgs &a, int num_blocks, float *out) {
    if (!a.clk->record) return;
    __shared__ float red[256];
    for (int c = 0; c < 3 * a.p.num_tools; c++) {
        float s = 0.f;
        for (int b = threadIdx.x; b < num_blocks; b += 256) s += a.s.force_part[size_t(b) * (3 * MAX_TOOLS) + c];
        red[threadIdx.x] = s;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) out[c] = red[0];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) kb_finalize(BatchTable T) {
    begin_after();
    const int s = find_scene(T.pblk, T.nscenes, blockIdx.x);
    finalize_body(scene_args(T, s), int(blockIdx.x) - T.pblk[s]);
}
// one block per scene
__global__ void __launch_bounds__(256) kb_force_final(BatchTable T) {
    begin_after();
    __shared__ StepArgs sa;
    load_scene_args(sa, T, blockIdx.x);
    __syncthreads();
    if (sa.p.num_tools > 0) force_final_body(sa, finalize_blocks(sa.p.n_init), sa.s.forces);
}

}  // namespace mfree
