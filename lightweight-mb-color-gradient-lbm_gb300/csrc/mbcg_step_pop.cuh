// mbcg_step_pop.cuh -- the step by populations: of lattices in BF16 storage without an inlet, and of fully
// periodic unforced ones in FP16 storage.
//
// step_tile() (mbcg_step.cuh) is faster (1.3x on a 192^3 drop, 1.07x on small walled ones) and nearer to the
// exact step.  These lattices keep this kernel for what they store.  The density slot of a drop in
// equal-density fluids holds (rho - 1) / 0.01 with rho - 1 around 1e-6, so the FP32 rounding of the density
// sum, 1e-7, is 1 to 7 % of the slot (64^3 to 200^3), and another order of summation changes stored states by
// that much.  With a density ratio a last bit of FP32 now and then rounds a colour slot the other way (three
// nodes in 10^6); beside such a node the stress of the next step is up to 1.7 times the field's mean away
// in BF16, 0.3 times in FP16 (RTI).  With an inlet states agree to 6e-4 (BF16) after two steps.
// For the same reason the server and the plain-load path step them by populations too: served by step_tile
// their states differed from a case's by up to a unit of the form after the first step (served alone, D3Q27 drop
// 61^3 in FP16 41 us a step against 31 by step_tile, in BF16 46 against 31; RTI 31^2x64 in BF16 26 against 41).
//
// Each source evaluates all Q populations of its coefficient tensor with a separable inverse transform (x, y,
// then z); they stream to the neighbouring lanes by shuffles, to the neighbouring rows through shared memory and
// along z by the march, and are projected onto the destination's moments by the separable forward transform.  A
// CTA is 32 lanes x W warps, one node a thread, 30 x (W-2) destination columns; staging as in step_tile.
#pragma once

#include "mbcg_step.cuh"

namespace mbcg {

namespace {

namespace pop {

constexpr int kNSTAGE = 4; // planes staged: k, k+1, and k+2, k+3 in flight

// shared-memory carve-up (see Geo in mbcg_step.cuh)
template <typename S, int W>
struct Geo {
    static constexpr int RBY = W + 2;
    static constexpr int MY = W;
    static constexpr int rb_field = align128(RBY * kRBX * (int)sizeof(S));
    static constexpr int m_field = align128(MY * kMX * (int)sizeof(S));
    static constexpr int stage = 2 * rb_field + 9 * m_field;
    static constexpr int tx = 2 * RBY * kRBX * (int)sizeof(S) + 9 * MY * kMX * (int)sizeof(S);
    static constexpr int psi_plane = RBY * kPSX;           // floats
    static constexpr int psi = kNSTAGE * psi_plane * 4;    // bytes (ring slot = stage slot)
    static constexpr int xbuf_floats = 3 * 2 * 4 * W * 32; // float4 [class][slot][row][lane]
    static constexpr int xbuf = xbuf_floats * 4;
    static constexpr int off_bar = 0;
    static constexpr int off_stage = 128;
    static constexpr int off_psi = off_stage + kNSTAGE * stage;
    static constexpr int off_xbuf = off_psi + psi;
    static constexpr int smem = off_xbuf + xbuf + 128;
};

struct Coef {
    float p000, p100, p010, p001, p200, p020, p002, p110, p101, p011;
    float p210, p201, p120, p102, p021, p012, p111;
    float r0; // extra on the rest population (density ratio)
};

// Equilibrium (pdf.cuh:16-36) + oms * regularised non-equilibrium (pdf.cuh:38-79) + 1/2 Guo force
// (pdf.cuh:94-136) + density-ratio rest term, as the coefficients of a polynomial in c (w_i factored out).
template <int kFeat>
__device__ __forceinline__ void build_coef(const StepParams& P, Coef& c, float rho, float rr, float rb, float ux,
                                           float uy, float uz, float pxx, float pxy, float pyy, float pyz, float pzz,
                                           float pxz) {
    const float vx = ux, vy = uy, vz = uz;
    float oms = P.oms;
    if constexpr ((kFeat & F_FORCE) != 0)
        if (P.tau_var) oms = 1.0f - 1.0f / tau_eff_of(P, rr, rb);
    const float usq = ux * ux + uy * uy + uz * uz;
    const float rux = rho * ux, ruy = rho * uy, ruz = rho * uz;
    const float t1 = 3.0f - 4.5f * usq;
    const float a3xxy = pxx * vy + 2.0f * pxy * vx;
    const float a3xxz = pxx * vz + 2.0f * pxz * vx;
    const float a3xyy = pyy * vx + 2.0f * pxy * vy;
    const float a3xzz = pzz * vx + 2.0f * pxz * vz;
    const float a3yyz = pyy * vz + 2.0f * pyz * vy;
    const float a3yzz = pzz * vy + 2.0f * pyz * vz;
    const float a3xyz = pxy * vz + pxz * vy + pyz * vx;
    const float o45 = 4.5f * oms, o9 = 9.0f * oms, o135 = 13.5f * oms;
    // p000 holds only the small isotropic part; rho itself is added to every direction last
    // (see emit), so the rounding of rho + small treats rest and moving populations alike
    c.p000 = -1.5f * (rho * usq + oms * (pxx + pyy + pzz));
    c.p100 = rux * t1 + 4.5f * rux * ux * ux - o45 * (a3xyy + a3xzz);
    c.p010 = ruy * t1 + 4.5f * ruy * uy * uy - o45 * (a3xxy + a3yzz);
    c.p001 = ruz * t1 + 4.5f * ruz * uz * uz - o45 * (a3xxz + a3yyz);
    c.p200 = 4.5f * rux * ux + o45 * pxx;
    c.p020 = 4.5f * ruy * uy + o45 * pyy;
    c.p002 = 4.5f * ruz * uz + o45 * pzz;
    c.p110 = 9.0f * rux * uy + o9 * pxy;
    c.p101 = 9.0f * rux * uz + o9 * pxz;
    c.p011 = 9.0f * ruy * uz + o9 * pyz;
    c.p210 = 13.5f * rux * ux * uy + o135 * a3xxy;
    c.p201 = 13.5f * rux * ux * uz + o135 * a3xxz;
    c.p120 = 13.5f * rux * uy * uy + o135 * a3xyy;
    c.p102 = 13.5f * rux * uz * uz + o135 * a3xzz;
    c.p021 = 13.5f * ruy * uy * uz + o135 * a3yyz;
    c.p012 = 13.5f * ruy * uz * uz + o135 * a3yzz;
    c.p111 = 27.0f * rux * uy * uz + 2.0f * o135 * a3xyz;
    c.r0 = 0.0f;
    if constexpr ((kFeat & F_FORCE) == 0) return;
    if (P.forced) {
        const float Fx = rho * P.g[0], Fy = rho * P.g[1], Fz = rho * P.g[2];
        const float Gxxy = Fx * ux * uy + 0.5f * Fy * ux * ux;
        const float Gxxz = Fx * ux * uz + 0.5f * Fz * ux * ux;
        const float Gxyy = Fy * ux * uy + 0.5f * Fx * uy * uy;
        const float Gxzz = Fz * ux * uz + 0.5f * Fx * uz * uz;
        const float Gyyz = Fy * uy * uz + 0.5f * Fz * uy * uy;
        const float Gyzz = Fz * uy * uz + 0.5f * Fy * uz * uz;
        const float Gxyz = Fx * uy * uz + Fy * ux * uz + Fz * ux * uy;
        c.p000 -= 1.5f * (Fx * ux + Fy * uy + Fz * uz);
        c.p100 += 1.5f * Fx - 4.5f * (Gxyy + Gxzz);
        c.p010 += 1.5f * Fy - 4.5f * (Gxxy + Gyzz);
        c.p001 += 1.5f * Fz - 4.5f * (Gxxz + Gyyz);
        c.p200 += 4.5f * Fx * ux;
        c.p020 += 4.5f * Fy * uy;
        c.p002 += 4.5f * Fz * uz;
        c.p110 += 4.5f * (Fx * uy + Fy * ux);
        c.p101 += 4.5f * (Fx * uz + Fz * ux);
        c.p011 += 4.5f * (Fy * uz + Fz * uy);
        c.p210 += 13.5f * Gxxy;
        c.p201 += 13.5f * Gxxz;
        c.p120 += 13.5f * Gxyy;
        c.p102 += 13.5f * Gxzz;
        c.p021 += 13.5f * Gyyz;
        c.p012 += 13.5f * Gyzz;
        c.p111 += 13.5f * Gxyz;
    }
    if (P.ratio) {
        const float K = rr * P.kappa_r + rb * P.kappa_b;
        c.p000 += K;
        c.r0 -= K;
    }
}

// ------------------------------------------------------------------ accumulators
// (rho, red) and (jx, xx) are packed pairs: they always take the same operations, which then
// issue as one f32x2 instruction (add/fma.f32x2, sm_100 and later) instead of two.
struct Acc {
    float2 rr, jxx;
    float jy, jz, xy, yy, yz, zz, xz;
    __device__ __forceinline__ void zero() {
        rr = jxx = make_float2(0.0f, 0.0f);
        jy = jz = xy = yy = yz = zz = xz = 0.0f;
    }
};

// a + f b on both halves (f = 1: a plain add, as fmaf(1, b, a) would round)
template <int F>
__device__ __forceinline__ float2 acc2(float2 a, float2 b) {
    if constexpr (F == 1) return __fadd2_rn(a, b);
    else return __ffma2_rn(pair(static_cast<float>(F)), b, a);
}
// A quantity over the three x velocities of one (cy, cz): `o` = (cx = -1, cx = +1) as an f32x2
// pair, `c` = cx = 0.  The two outer values always take the same operations.
struct Tri {
    float2 o;
    float c;
};
__device__ __forceinline__ Tri tri(float base, float odd, float centre) {
    return Tri{make_float2(base - odd, base + odd), centre};
}
__device__ __forceinline__ Tri operator+(Tri a, Tri b) { return Tri{__fadd2_rn(a.o, b.o), a.c + b.c}; }
__device__ __forceinline__ Tri operator-(Tri a, Tri b) { return Tri{mbcg::operator-(a.o, b.o), a.c - b.c}; }
__device__ __forceinline__ Tri operator+(Tri a, float s) { return Tri{__fadd2_rn(a.o, pair(s)), a.c + s}; }

// add one population of velocity (ex, ey, ez) to a destination's moment sums
__device__ __forceinline__ void add_pop(Acc& a, float g, float r, int ex, int ey, int ez) {
    a.rr.x += g;
    a.rr.y += r;
    if (ex) { a.jxx.x += ex * g; a.jxx.y += g; }
    if (ey) { a.jy += ey * g; a.yy += g; }
    if (ez) { a.jz += ez * g; a.zz += g; }
    if (ex && ey) a.xy += ex * ey * g;
    if (ey && ez) a.yz += ey * ez * g;
    if (ex && ez) a.xz += ex * ez * g;
}

// one tile (30 columns x (W-2) rows x zchunk planes), arguments as step_tile's
template <int Q, typename S, int W, bool kTMA, int kFeat>
__device__ __forceinline__ bool tile(const StepParams& P, const CUtensorMap* maps, int bx, int by, int bz, long long step,
                                     unsigned char* smem, uint32_t& phase) {
    using G = Geo<S, W>;
    float* psi_ring = reinterpret_cast<float*>(smem + G::off_psi);
    float4* xbuf = reinterpret_cast<float4*>(smem + G::off_xbuf);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + G::off_bar);

    const int lane = threadIdx.x;
    const int w = threadIdx.y;
    const int tid = w * 32 + lane;
    const int nx = P.nx, ny = P.ny, nz = P.nz;

    const int xb = kTX * bx;     // source column of lane 0
    const int yb = (W - 2) * by; // source row of warp 0
    const int xs = xb + lane, ys = yb + w;
    const int zd0 = 1 + P.zchunk * bz;
    const int zd1 = min(zd0 + P.zchunk, nz - 1);
    const int kfirst = zd0 - 2;

    const int xr0 = floor8(xb - 1); // first staged column of rhor/rhob
    const int xm0 = floor8(xb);     // first staged column of the other fields
    const int offRB = xb - xr0;
    const int offM = xb - xm0;
    const int bR = (w + 1) * kRBX + lane + offRB; // this node in the rhor/rhob boxes
    const int bM = w * kMX + lane + offM;         // this node in the other boxes

    const bool dest_thread = lane >= 1 && lane <= kTX && w >= 1 && w <= W - 2 && xs <= nx - 2 && ys <= ny - 2;
    const int rx = axis_role<kFeat>(P, 0, xs, nx);
    const int ry = axis_role<kFeat>(P, 1, ys, ny);
    const bool in_xy = rx != R_OUT && ry != R_OUT;
    // the node's role, given the role of its plane
    auto role_of = [&](int rz) -> int {
        if (rx == R_OUT || ry == R_OUT || rz == R_OUT) return R_OUT;
        if ((kFeat & F_WALL) && (rx == R_WALL || ry == R_WALL || rz == R_WALL)) return R_WALL;
        return R_FLUID;
    };
    const int role_xy = role_of(R_FLUID); // on fluid planes
    // stochastic rounding of the 16-bit stores: key base of this step
    const unsigned key_base = round_key_base(P.seed, step);
    // periodic images of this column's store (x = 1 / nx-2, y = 1 / ny-2 on a periodic axis)
    const int img_x = P.bc[0] == MBCG_BC_PERIODIC ? (xs == 1 ? nx - 1 : (xs == nx - 2 ? 0 : -1)) : -1;
    const int img_y = P.bc[1] == MBCG_BC_PERIODIC ? (ys == 1 ? ny - 1 : (ys == ny - 2 ? 0 : -1)) : -1;

    // psi fill: each thread owns <= kPsiPer ring elements; their mapping never changes along z.
    // Each element reads the staged box at the node whose stored value equals psi there (the
    // periodic ghost frame holds images), or, for the periodic images two layers out that the
    // box cannot hold, a global load issued one plane ahead into registers.
    constexpr int kPsiPer = (G::psi_plane + 32 * W - 1) / (32 * W);
    int psi_box[kPsiPer];      // box index, -1: prefetched global load, -2: no element
    long long psi_g[kPsiPer];  // mapped (x, y) offset in global memory
    float pf0[kPsiPer], pf1[kPsiPer];
#pragma unroll
    for (int j = 0; j < kPsiPer; ++j) {
        const int e = tid + j * 32 * W;
        psi_box[j] = -2;
        psi_g[j] = 0;
        pf0[j] = pf1[j] = 0.0f;
        if (e < G::psi_plane) {
            const int r = e / kPSX, c = e % kPSX;
            const int gx = xb - 1 + c, gy = yb - 1 + r;
            if (gx < -1 || gx > nx || gy < -1 || gy > ny) {
                // beyond the ghost frame and its one-node halo: read only by the colour gradient of
                // sources outside the lattice, whose populations reach no destination of the tile,
                // so any staged element serves (no global load)
                psi_box[j] = 0;
                continue;
            }
            const int mx = psi_coord(P, 0, gx, nx), my = psi_coord(P, 1, gy, ny);
            const bool px = P.bc[0] == MBCG_BC_PERIODIC, py = P.bc[1] == MBCG_BC_PERIODIC;
            const int dx = (px && gx >= 0 && gx <= nx - 1) ? gx : mx;
            const int dy = (py && gy >= 0 && gy <= ny - 1) ? gy : my;
            const int bc_ = dx - xr0, br_ = dy - (yb - 1);
            psi_box[j] = (bc_ >= 0 && bc_ < kRBX && br_ >= 0 && br_ < G::RBY) ? br_ * kRBX + bc_ : -1;
            psi_g[j] = static_cast<long long>(my) * P.pitch + mx;
        }
    }

    // periodic images two layers out are read from global memory; most tiles have none
    bool far_any = false;
#pragma unroll
    for (int j = 0; j < kPsiPer; ++j) far_any = far_any || psi_box[j] == -1;
    far_any = __syncthreads_or(far_any) != 0;

    // Plane k lives in stage slot (k - kfirst) mod 3, and its psi in the ring slot of the same
    // index; the z loop advances the slot incrementally.
    auto nxt = [](int sl) -> int { return sl == kNSTAGE - 1 ? 0 : sl + 1; };
    auto prv = [](int sl) -> int { return sl == 0 ? kNSTAGE - 1 : sl - 1; };
    auto stage_at = [&](int sl) -> unsigned char* { return smem + G::off_stage + sl * G::stage; };
    auto rb_box = [&](unsigned char* st, int f) -> S* { return reinterpret_cast<S*>(st + f * G::rb_field); };
    auto m_box = [&](unsigned char* st, int f) -> S* {
        return reinterpret_cast<S*>(st + 2 * G::rb_field + (f - 2) * G::m_field);
    };
    auto zload = [&](int k) -> int { return data_coord(P, 2, k, nz); };

    // ---- stage loader -------------------------------------------------------------
    auto issue = [&](int k, int sl) {
        unsigned char* st = stage_at(sl);
        const int kz = zload(k);
        if constexpr (kTMA) {
            if (tid == 0) {
                uint64_t* bar = &bars[sl];
                fence_proxy_async();
                mbar_expect_tx(bar, G::tx);
                tma_load_3d(rb_box(st, 0), &maps[0], xr0, yb - 1, kz, bar);
                tma_load_3d(rb_box(st, 1), &maps[1], xr0, yb - 1, kz, bar);
#pragma unroll
                for (int f = 2; f < NF; ++f) tma_load_3d(m_box(st, f), &maps[f], xm0, yb, kz, bar);
            }
        } else {
            // plain loads, for layouts TMA cannot describe: whole boxes, zeros outside the lattice
            const long long zo = static_cast<long long>(kz) * P.plane;
            auto box = [&](int f, S* dst, int x0, int y0, int width, int rows) {
                for (int e = tid; e < rows * width; e += 32 * W) {
                    const int gx = x0 + e % width, gy = y0 + e / width;
                    const bool in = gx >= 0 && gx < nx && gy >= 0 && gy < ny;
                    dst[e] = in ? static_cast<const S*>(P.a[f])[zo + gy * P.pitch + gx] : Codec<S>::from_f(0.0f);
                }
            };
            for (int f = 0; f < 2; ++f) box(f, rb_box(st, f), xr0, yb - 1, kRBX, G::RBY);
            for (int f = 2; f < NF; ++f) box(f, m_box(st, f), xm0, yb, kMX, G::MY);
        }
    };
    constexpr long long kWaitLimit = 4000000000LL; // ~2 s at 2 GHz
    // Expected parity of the next phase of each slot's mbarrier; every completed wait flips it.
    // It starts from the parities the previous tile of this CTA left.
    uint32_t par = phase;
    int k_waited = kfirst - 1; // last plane whose load was waited for
    auto wait_slot = [&](int k, int sl) -> bool {
        bool ok = true;
        if constexpr (kTMA) ok = mbar_wait_bounded(&bars[sl], (par >> sl) & 1u, kWaitLimit);
        if (ok) {
            par ^= 1u << sl;
            k_waited = k;
        }
        return ok;
    };
    // on a failed wait (see step_tile)
    auto bail = [&](int k_issued) {
        if (tid == 0 && P.status) atomicOr(P.status, 1);
        for (int k = k_waited + 1; kTMA && k <= k_issued; ++k) {
            const int sl = (k - kfirst) % kNSTAGE;
            mbar_wait_bounded(&bars[sl], (par >> sl) & 1u, kWaitLimit / 4);
        }
    };

    // ---- psi ring: psi = (rhor - rhob)/rho (mathUtilities.cuh:12-19) of plane k over
    // columns xb-1..xb+32 and rows yb-1..yb+W, colour-gradient neighbour rule applied
    auto prefetch_psi = [&](int mz) {
        const long long zo = static_cast<long long>(mz) * P.plane;
#pragma unroll
        for (int j = 0; j < kPsiPer; ++j)
            if (psi_box[j] == -1) {
                pf0[j] = Codec<S>::to_f(static_cast<const S*>(P.a[0])[zo + psi_g[j]]);
                pf1[j] = Codec<S>::to_f(static_cast<const S*>(P.a[1])[zo + psi_g[j]]);
            }
    };
    // mz: the plane the colour-gradient rule maps k to; plane_in_box: it is the staged plane
    auto fill_psi = [&](int mz, bool plane_in_box, int sl, bool prefetched) {
        float* ring = psi_ring + sl * G::psi_plane;
        if (plane_in_box && !far_any) {
            // every element of this tile is in the staged box (the first one of each thread
            // always exists: the ring plane has at least 32 W elements)
            unsigned char* st = stage_at(sl);
            const S* r0b = rb_box(st, 0);
            const S* r1b = rb_box(st, 1);
            ring[tid] = psi_of<S>(P, r0b[psi_box[0]], r1b[psi_box[0]]);
#pragma unroll
            for (int j = 1; j < kPsiPer; ++j)
                if (psi_box[j] >= 0) ring[tid + j * 32 * W] = psi_of<S>(P, r0b[psi_box[j]], r1b[psi_box[j]]);
            return;
        }
        const long long zo = static_cast<long long>(mz) * P.plane;
        unsigned char* st = stage_at(sl);
        const S* r0b = rb_box(st, 0);
        const S* r1b = rb_box(st, 1);
#pragma unroll
        for (int j = 0; j < kPsiPer; ++j) {
            if (psi_box[j] == -2) continue;
            float v;
            if (plane_in_box && psi_box[j] >= 0) {
                v = psi_of<S>(P, r0b[psi_box[j]], r1b[psi_box[j]]);
            } else if (prefetched && psi_box[j] == -1) {
                v = psi_of_slots<S>(pf0[j], pf1[j]);
            } else {
                const long long o = zo + psi_g[j];
                v = psi_of<S>(P, static_cast<const S*>(P.a[0])[o], static_cast<const S*>(P.a[1])[o]);
            }
            ring[tid + j * 32 * W] = v;
        }
    };

    // ---- set-up ------------------------------------------------------------------
    // every thread is done with the previous tile's shared memory before it is refilled
    __syncthreads();
    int k_issued = kfirst + kNSTAGE - 1;
    for (int k = kfirst; k <= k_issued; ++k) issue(k, k - kfirst);
    if constexpr (!kTMA) __syncthreads();
    {
        // the first wait (wait_test_cycles: see step_tile)
        bool ok = true;
        if constexpr (kTMA) {
            const bool test = P.wait_test_cycles > 0;
            ok = mbar_wait_bounded(test ? &bars[kMaxStages] : &bars[0], test ? 0u : (par & 1u),
                                   test ? static_cast<long long>(P.wait_test_cycles) : kWaitLimit);
            if (ok) {
                par ^= 1u;
                k_waited = kfirst;
            }
        }
        ok = ok && wait_slot(kfirst + 1, 1);
        if (__syncthreads_or(!ok)) {
            bail(k_issued);
            return false;
        }
    }
    {
        const int m0 = psi_coord(P, 2, kfirst, nz), m1 = psi_coord(P, 2, kfirst + 1, nz);
        fill_psi(m0, m0 == zload(kfirst), 0, false);
        fill_psi(m1, m1 == zload(kfirst + 1), 1, false);
    }
    if (far_any) prefetch_psi(psi_coord(P, 2, kfirst + 2, nz));

    Acc accP, accC, accN; // destination planes k-1, k, k+1
    accP.zero();
    accC.zero();
    accN.zero();

    constexpr float cs2 = 1.0f / 3.0f;
    float4* xb_self = xbuf + w * 32 + lane; // (X0, XR, X1, X2) of one exported row

    int sl = 1; // slot of plane k (k starts at kfirst + 1)
    int k = zd0 - 1;
    // One plane of the z-march with the feature set kFB: the tile's own, or, between the walls of a z
    // axis, the same set without their part.  Returns false after a bail.
    auto plane = [&](auto featc) -> bool {
        constexpr int kFB = decltype(featc)::value;
        const int sl_next = nxt(sl), sl_prev = prv(sl);
        // (1) psi of plane k+1; one barrier both publishes the ring and makes the bail decision
        // uniform (a plane that never arrived leaves garbage in the ring, which nobody reads)
        // Plane coordinates: every mapping (staging, colour-gradient rule, node role) is the
        // identity while planes k .. k+3 are fluid planes, which is almost every plane.
        const bool zid = k >= 1 && k + kNSTAGE - 1 <= nz - 2;
        int mz1 = k + 1, mz2 = k + 2, rz = R_FLUID;
        bool inbox1 = true;
        if (!zid) {
            mz1 = psi_coord(P, 2, k + 1, nz);
            inbox1 = mz1 == zload(k + 1);
            mz2 = psi_coord(P, 2, k + 2, nz);
            rz = axis_role<kFB>(P, 2, k, nz);
        }
        {
            const bool ok = wait_slot(k + 1, sl_next);
            if (ok) fill_psi(mz1, inbox1, sl_next, true);
            if (__syncthreads_or(!ok)) {
                bail(k_issued);
                return false;
            }
        }
        if (far_any && k + 2 <= zd1 + 1) prefetch_psi(mz2);
        // (2) prefetch plane k+3 into the slot plane k-1 used
        if (k + kNSTAGE - 1 <= zd1 + 1 && k + kNSTAGE - 1 > k_issued) {
            issue(k + kNSTAGE - 1, sl_prev);
            k_issued = k + kNSTAGE - 1;
        } else {
            launch_dependents(); // nothing more to stage
        }

        // (3) this thread's source node at plane k
        const int role = zid ? role_xy : role_of(rz);
        // Sources outside the lattice (lanes / rows past the last ghost layer) only ever stream
        // into nodes that are not destinations of this tile, so without walls every source is
        // processed branch-free; wall ghost layers hold data and must not emit.
        const bool active = ((kFB & F_WALL) == 0) || role == R_FLUID;

        unsigned char* st = stage_at(sl);
        Node<S> nd{};
        if (active) {
            float v[NF];
            v[0] = Codec<S>::to_f(rb_box(st, 0)[bR]);
            v[1] = Codec<S>::to_f(rb_box(st, 1)[bR]);
#pragma unroll
            for (int f = 2; f < NF; ++f) v[f] = Codec<S>::to_f(m_box(st, f)[bM]);
            decode<S>(P, v, nd);
        }

        // coefficient tensor and colour split; inactive sources keep all-zero coefficients
        Coef cf{};
        float aR = 0.0f, dcoef = 0.0f, Fx = 0.0f, Fy = 0.0f, Fz = 0.0f, omega2_rest = 0.0f;
        bool iface = false;
        if (active) {
            const float rho = nd.rr + nd.rb;
            const float inv = fast_rcp(rho);
            // colour fraction as a correctly rounded quotient (one residual correction): a
            // product with a rounded reciprocal is biased (aR rho - rr averages +2.5e-10 per
            // mixed node), which would move colour mass the same way every step
            const float q0 = nd.rr * inv;
            const float q1 = fmaf(fmaf(-q0, rho, nd.rr), inv, q0);
            aR = nd.rb == 0.0f ? 1.0f : (nd.rr == 0.0f ? 0.0f : q1);
            iface = (4.0f * nd.rr * nd.rb * inv * inv) > 1.0e-4f; // lbm.cuh:181,187
            // zero-filled staging outside the lattice decodes to a mixed node: off the interface path
            iface = iface && in_xy;
            build_coef<kFB>(P, cf, rho, nd.rr, nd.rb, nd.ux, nd.uy, nd.uz, nd.pxx, nd.pxy, nd.pyy, nd.pyz, nd.pzz, nd.pxz);
        }
        const bool any_iface = __any_sync(kFull, iface);
        if (any_iface && iface) {
            // colour gradient at the source (forces.cuh:20-60) from the psi ring
            const float* rm = psi_ring + sl_prev * G::psi_plane;
            const float* r0p = psi_ring + sl * G::psi_plane;
            const float* rp = psi_ring + sl_next * G::psi_plane;
            float sx = 0.0f, sy = 0.0f, sz = 0.0f;
#pragma unroll
            for (int dz = -1; dz <= 1; ++dz) {
                const float* ring = dz < 0 ? rm : (dz == 0 ? r0p : rp);
#pragma unroll
                for (int dy = -1; dy <= 1; ++dy) {
#pragma unroll
                    for (int dx = -1; dx <= 1; ++dx) {
                        if (dx == 0 && dy == 0 && dz == 0) continue;
                        if (!Stencil<Q>::has(dx, dy, dz)) continue;
                        const float ps = ring[(w + 1 + dy) * kPSX + lane + 1 + dx];
                        const float wp = weight<Q>(dx, dy, dz) * ps;
                        if (dx) sx += dx * wp;
                        if (dy) sy += dy * wp;
                        if (dz) sz += dz * wp;
                    }
                }
            }
            Fx = 3.0f * sx;
            Fy = 3.0f * sy;
            Fz = 3.0f * sz;
            const float absF = sqrtf(Fx * Fx + Fy * Fy + Fz * Fz);
            // Omega2 (collisionOperators.cuh:16-25) folded into the coefficients
            float Aeff = P.A; // A_calculation (forces.cuh:114-117) at the node's relaxation time
            if constexpr ((kFB & F_FORCE) != 0)
                if (P.tau_var) Aeff = P.s4 / tau_eff_of(P, nd.rr, nd.rb);
            float hA = (P.omega2_conservative && !(absF > 1.0e-4f)) ? 0.0f : 0.5f * Aeff * absF;
            if (absF > 1.0e-4f) {
                const float ia_ = fast_rcp(absF);
                const float qf = 0.5f * Aeff * ia_;
                // isotropic part from the same q |F|^2 as the anisotropic part, so Omega2 sums
                // to zero over the directions in floating point too
                hA = qf * (Fx * Fx + Fy * Fy + Fz * Fz);
                cf.p200 += qf * Fx * Fx;
                cf.p020 += qf * Fy * Fy;
                cf.p002 += qf * Fz * Fz;
                cf.p110 += 2.0f * qf * Fx * Fy;
                cf.p101 += 2.0f * qf * Fx * Fz;
                cf.p011 += 2.0f * qf * Fy * Fz;
                // recolouring (collisionOperators.cuh:60-80): beta rr rb / (rho^2 |F|) * feq0, where
                // the rest equilibrium of moving directions is w rho (w (rho + K) with a density ratio)
                const float rho = nd.rr + nd.rb;
                const float feq0 = ((kFB & F_FORCE) && P.ratio) ? rho + nd.rr * P.kappa_r + nd.rb * P.kappa_b : rho;
                const float irho = fast_rcp(rho);
                dcoef = P.beta * (nd.rr * nd.rb) * irho * irho * ia_ * feq0;
            }
            cf.p000 -= hA;
            omega2_rest = hA; // rest-population part, -hA (B0 - w0) = +2/3 hA, added below in exact units
        }
        const float rho_src = active ? nd.rr + nd.rb : 0.0f;
        const float rr_src = active ? nd.rr : 0.0f;
        // colour fractions of the x neighbours (lane -1 and lane +1)
        float2 aRlr;
        aRlr.x = __shfl_up_sync(kFull, aR, 1);
        aRlr.y = __shfl_down_sync(kFull, aR, 1);

        // separable inverse transform, x-pass: t_bc(cx) for the monomials cy^b cz^c
        const Tri t00 = tri(cf.p000 + cf.p200, cf.p100, cf.p000);
        const Tri t10 = tri(cf.p010 + cf.p210, cf.p110, cf.p010);
        const Tri t01 = tri(cf.p001 + cf.p201, cf.p101, cf.p001);
        const Tri t20 = tri(cf.p020, cf.p120, cf.p020);
        const Tri t02 = tri(cf.p002, cf.p102, cf.p002);
        const Tri t11 = tri(cf.p011, cf.p111, cf.p011);
        const float2 rho2 = pair(rho_src);
        // Populations are carried scaled by S = 216 (D3Q27) or 36 (D3Q19), where the weights
        // are small integers that sum to S exactly: float-rounded weights do not sum to 1, and
        // that error would scale every node's mass each step (about 1.5e-8 per step for D3Q19).
        // D3Q27 weights are also separable, S w(c) = prod over axes of (4 if c_a = 0 else 1):
        // populations are carried unweighted and the factors 4 are applied inside the forward
        // passes.  D3Q19 weights 12, 2, 1 are applied per population.  Each destination
        // divides its sums by S once, the mass sums with a correctly rounded quotient.
        constexpr bool kSepW = (Q == 27);
        const float dk1 = kSepW ? dcoef : 2.0f * dcoef;
        const float dk2 = dcoef * 0.7071067811865475f;
        const float dk3 = kSepW ? dcoef * 0.5773502691896258f : 0.0f;
        // rest-population correction (density-ratio K and the Omega2 rest term), with the Omega2
        // part in exact units so that Omega2 sums to zero over the directions (B0 - w0 = -2/3
        // for both lattices)
        // in value units before the rest weight (64 of 216, or 12 of 36): S r0 / W_0 and
        // S (w0 - B0) hA / W_0 = (2/3) S hA / W_0, i.e. 3.375 r0 + 2.25 hA or 3 r0 + 2 hA
        const float rc0 = kSepW ? fmaf(cf.r0, 3.375f, 2.25f * omega2_rest) : fmaf(cf.r0, 3.0f, 2.0f * omega2_rest);

        // wall bounce-back of this node's own populations (destination = this node, plane k)
        const bool wx0 = P.bc[0] == MBCG_BC_WALL && xs == 1, wx1 = P.bc[0] == MBCG_BC_WALL && xs == nx - 2;
        const bool wy0 = P.bc[1] == MBCG_BC_WALL && ys == 1, wy1 = P.bc[1] == MBCG_BC_WALL && ys == ny - 2;
        const bool wz0 = P.bc[2] == MBCG_BC_WALL && k == 1, wz1 = P.bc[2] == MBCG_BC_WALL && k == nz - 2;
        const bool reflect = (kFB & F_WALL) && role == R_FLUID && dest_thread && (wx0 | wx1 | wy0 | wy1 | wz0 | wz1);
        const bool any_reflect = (kFB & F_WALL) ? __any_sync(kFull, reflect) : false;

        // ---- emit: populations of the rows this warp exports, x streaming, own-row moments,
        // y exchange.  Halo rows export one population row (cy = +1 for warp 0, -1 for warp W-1).
        auto emit = [&](auto rowsc) {
            constexpr int ROWS = decltype(rowsc)::value;
            // y-pass per exported row j (cy = j - 1): s0 (cz^0), s1 (cz^1), e2 (cz^0 + cz^2)
            Tri s0[3], s1[3], e2[3];
            {
                const Tri e0 = t00 + t20;
                const Tri e1 = t01 + cf.p021;
                if (ROWS & 2) {
                    s0[1] = t00;
                    s1[1] = t01;
                    e2[1] = t00 + t02;
                }
                if (ROWS & 4) {
                    s0[2] = e0 + t10;
                    s1[2] = e1 + t11;
                    e2[2] = s0[2] + (t02 + cf.p012);
                }
                if (ROWS & 1) {
                    s0[0] = e0 - t10;
                    s1[0] = e1 - t11;
                    e2[0] = s0[0] + (t02 + (-cf.p012));
                }
            }
            auto do_class = [&](auto czc, Acc& acc) {
                constexpr int cz = decltype(czc)::value;
                // populations of row j: rho + the small part (rho last, see above); sm keeps the
                // small parts (value units, before the D3Q19 weight) for the red populations
                Tri g[3], sm[3];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const int cy = j - 1;
                    g[j].o = sm[j].o = make_float2(0.0f, 0.0f);
                    g[j].c = sm[j].c = 0.0f;
                    if (!(ROWS & (1 << j))) continue;
                    Tri small = cz == 0 ? s0[j] : (cz > 0 ? e2[j] + s1[j] : e2[j] - s1[j]);
                    if (cy == 0 && cz == 0) small.c += rc0;
                    const int shc = cy * cy + cz * cz; // |c|^2 of the centre; the outer ones have shc + 1
                    if (Stencil<Q>::has(1, cy, cz)) {
                        sm[j].o = small.o;
                        const float2 vv = __fadd2_rn(rho2, small.o);
                        g[j].o = (kSepW || shc != 0) ? vv : __fadd2_rn(vv, vv);
                    }
                    if (Stencil<Q>::has(0, cy, cz)) {
                        sm[j].c = small.c;
                        const float vv = rho_src + small.c;
                        g[j].c = kSepW ? vv : (shc == 0 ? 12.0f * vv : (shc == 1 ? vv + vv : vv));
                    }
                }
                // recolouring part Delta_i of the red populations (interface sources only; the
                // red population is aR g_i + Delta_i, collisionOperators.cuh:60-80)
                auto delta = [&](int i, int j) -> float {
                    const int cx = i - 1, cy = j - 1, sh = cx * cx + cy * cy + cz * cz;
                    if (!(ROWS & (1 << j)) || !Stencil<Q>::has(cx, cy, cz) || sh == 0) return 0.0f;
                    const float dks = sh == 1 ? dk1 : (sh == 2 ? dk2 : dk3);
                    const float fc = (cx ? cx * Fx : 0.0f) + (cy ? cy * Fy : 0.0f) + (cz ? cz * Fz : 0.0f);
                    return dks * fc;
                };
                // Red population of direction (cx, cy, cz) = (i - 1, j - 1, cz) of a source with
                // density rho, red density rr, colour fraction aR = rr / rho, population
                // g = W (rho + sm) and recolouring part Delta.  On interface warps it is formed
                // as W (rr + aR sm) + Delta, which is aR g + Delta in exact arithmetic, but the
                // red populations of a source then sum to S rr + aR sum(W sm) (sm sums to zero)
                // whatever the rounding of aR, where aR g emits S aR rho: in a near-steady state
                // the quotient's rounding error repeats step after step and its sum over the
                // interface moved the 64^3 D3Q19 bubble's red mass by 7e-6 in 10^4 steps
                // (3.5e-7 with this form).  Elsewhere aR is within 2.5e-5 of 0 or 1 and the
                // populations are aR g.
                auto red_pop = [&](float rr_, float smv, float gv, float dl, int i, int j, bool withd) -> float {
                    if (!withd) return aR * gv;
                    const int cy = j - 1, shc = cy * cy + cz * cz + (i != 1 ? 1 : 0);
                    const float b = fmaf(aR, smv, rr_);
                    // D3Q19 weight of the population: 12 (rest), 2 (|c|^2 = 1), 1 (|c|^2 = 2)
                    if (kSepW || shc == 2) return b + dl;
                    if (shc == 1) return fmaf(2.0f, b, dl);
                    return fmaf(12.0f, b, dl);
                };
                if constexpr (ROWS == 7 && (kFB & F_WALL) != 0) {
                    if (any_reflect && reflect) {
#pragma unroll
                        for (int i = 0; i < 3; ++i)
#pragma unroll
                            for (int j = 0; j < 3; ++j) {
                                const int cx = i - 1, cy = j - 1;
                                if (!Stencil<Q>::has(cx, cy, cz)) continue;
                                const bool into = (wx0 && cx < 0) || (wx1 && cx > 0) || (wy0 && cy < 0) ||
                                                  (wy1 && cy > 0) || (wz0 && cz < 0) || (wz1 && cz > 0);
                                if (!into) continue;
                                const float f = kSepW ? static_cast<float>((cx == 0 ? 4 : 1) * (cy == 0 ? 4 : 1) *
                                                                           (cz == 0 ? 4 : 1))
                                                      : 1.0f;
                                const float gv = i == 0 ? g[j].o.x : (i == 2 ? g[j].o.y : g[j].c);
                                const float smv = i == 0 ? sm[j].o.x : (i == 2 ? sm[j].o.y : sm[j].c);
                                const float rr_ = red_pop(rr_src, smv, gv, any_iface ? delta(i, j) : 0.0f, i, j, any_iface);
                                add_pop(accC, f * gv, f * rr_, -cx, -cy, -cz);
                            }
                    }
                }
                // x streaming: destination x receives cx=+1 from lane-1 and cx=-1 from lane+1.
                // The populations cross lanes; on interface warps the source forms its red
                // populations (red_pop) and they cross too, elsewhere the destination forms them
                // as aR g from the source's colour fraction (shuffled once per plane).
                float X0[3], X1[3], X2[3], XR[3];
                auto xstream = [&](auto ifc) {
                    constexpr bool kIf = decltype(ifc)::value;
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const int cy = j - 1;
                        X0[j] = X1[j] = X2[j] = XR[j] = 0.0f;
                        if (!(ROWS & (1 << j))) continue;
                        const float r1 = red_pop(rr_src, sm[j].c, g[j].c, kIf ? delta(1, j) : 0.0f, 1, j, kIf);
                        if (Stencil<Q>::has(1, cy, cz)) {
                            float2 glr; // (from lane - 1, from lane + 1)
                            glr.x = __shfl_up_sync(kFull, g[j].o.y, 1);
                            glr.y = __shfl_down_sync(kFull, g[j].o.x, 1);
                            X2[j] = glr.x + glr.y;
                            X0[j] = kSepW ? fmaf(4.0f, g[j].c, X2[j]) : X2[j] + g[j].c;
                            X1[j] = glr.x - glr.y;
                            float2 rlr;
                            if constexpr (kIf) {
                                // red_pop of this lane's cx = -1 / +1 populations, paired
                                const bool w2 = !kSepW && cy == 0 && cz == 0; // D3Q19 weight 2
                                float2 ro = __ffma2_rn(pair(aR), sm[j].o, pair(rr_src));
                                const float2 dl = make_float2(delta(0, j), delta(2, j));
                                ro = w2 ? __ffma2_rn(pair(2.0f), ro, dl) : __fadd2_rn(ro, dl);
                                rlr.x = __shfl_up_sync(kFull, ro.y, 1);
                                rlr.y = __shfl_down_sync(kFull, ro.x, 1);
                            } else {
                                rlr = __fmul2_rn(aRlr, glr);
                            }
                            XR[j] = kSepW ? fmaf(4.0f, r1, rlr.x + rlr.y) : (rlr.x + rlr.y) + r1;
                        } else {
                            X0[j] = g[j].c;
                            XR[j] = r1;
                        }
                    }
                };
                if (any_iface) xstream(std::true_type{});
                else xstream(std::false_type{});
                if constexpr ((ROWS & 2) != 0) {
                    // cy = 0 row stays in this column: add to the destination's sums now.  Plane
                    // k+1 (cz = +1) receives its first contributions here: they are assigned, so
                    // its sums need no clearing.
                    constexpr int fi = kSepW ? (cz == 0 ? 16 : 4) : 1;
                    constexpr float f = static_cast<float>(fi);
                    if constexpr (cz == 1) {
                        acc.rr = fi == 1 ? make_float2(X0[1], XR[1]) : __fmul2_rn(pair(f), make_float2(X0[1], XR[1]));
                        acc.jxx = fi == 1 ? make_float2(X1[1], X2[1]) : __fmul2_rn(pair(f), make_float2(X1[1], X2[1]));
                        acc.jz = f * X0[1];
                        acc.xz = f * X1[1];
                        acc.zz = f * X0[1];
                    } else {
                        acc.rr = acc2<fi>(acc.rr, make_float2(X0[1], XR[1]));
                        acc.jxx = acc2<fi>(acc.jxx, make_float2(X1[1], X2[1]));
                        if (cz != 0) {
                            acc.jz = fmaf(cz * f, X0[1], acc.jz);
                            acc.xz = fmaf(cz * f, X1[1], acc.xz);
                            acc.zz = fmaf(f, X0[1], acc.zz);
                        }
                    }
                }
                // cy = +1 goes to row w+1 (slot 0), cy = -1 to row w-1 (slot 1)
                constexpr int cls = cz + 1;
                if constexpr ((ROWS & 4) != 0) {
                    xb_self[(cls * 2 + 0) * (W * 32)] = make_float4(X0[2], XR[2], X1[2], X2[2]);
                }
                if constexpr ((ROWS & 1) != 0) {
                    xb_self[(cls * 2 + 1) * (W * 32)] = make_float4(X0[0], XR[0], X1[0], X2[0]);
                }
            };
            do_class(std::integral_constant<int, -1>{}, accP);
            do_class(std::integral_constant<int, 0>{}, accC);
            do_class(std::integral_constant<int, 1>{}, accN);
        };
        if (w == 0) emit(std::integral_constant<int, 4>{});
        else if (w == W - 1) emit(std::integral_constant<int, 1>{});
        else emit(std::integral_constant<int, 7>{});
        __syncthreads();

        // (4) y streaming into destination rows
        auto gather = [&](auto czc, Acc& acc) {
            constexpr int cz = decltype(czc)::value;
            constexpr int cls = cz + 1;
            constexpr int fi = (kSepW && cz == 0) ? 4 : 1;
            constexpr float f = static_cast<float>(fi);
            const float4 pv = xb_self[(cls * 2 + 0) * (W * 32) - 32]; // row w-1 exported cy = +1
            const float4 mv = xb_self[(cls * 2 + 1) * (W * 32) + 32]; // row w+1 exported cy = -1
            // slots (X0, XR, X1, X2)
            const float2 s0r = __fadd2_rn(make_float2(pv.x, pv.y), make_float2(mv.x, mv.y)); // (s00, red)
            const float2 s12 = __fadd2_rn(make_float2(pv.z, pv.w), make_float2(mv.z, mv.w)); // (s10, s20)
            const float d00 = pv.x - mv.x;
            acc.rr = acc2<fi>(acc.rr, s0r);
            acc.jxx = acc2<fi>(acc.jxx, s12);
            if constexpr (cz == 1) {
                // first contributions to jy, xy, yy, yz of plane k+1 (f = 1)
                acc.jy = d00;
                acc.xy = pv.z - mv.z;
                acc.yy = s0r.x;
                acc.yz = d00;
            } else {
                acc.jy = fmaf(f, d00, acc.jy);
                acc.xy = fmaf(f, pv.z - mv.z, acc.xy);
                acc.yy = fmaf(f, s0r.x, acc.yy);
                if (cz != 0) acc.yz += cz * d00;
            }
            if (cz != 0) {
                acc.jz += cz * s0r.x;
                acc.xz += cz * s12.x;
                acc.zz += s0r.x;
            }
        };
        const bool dest_row = (w >= 1 && w <= W - 2);
        if (dest_row) gather(std::integral_constant<int, -1>{}, accP);

        // (5) destination plane k-1 is complete: moments (lbm.cuh:239-261), store, boundary
        const int d = k - 1;
        if (dest_thread && d >= zd0 && d < zd1) {
            {
                constexpr float kS = kSepW ? 216.0f : 36.0f;
                constexpr float sc = 1.0f / kS;
                // correctly rounded mass quotients (no systematic bias), plain scaling for the rest
                const float2 q = __fmul2_rn(accP.rr, pair(sc));
                const float2 e = __ffma2_rn(make_float2(-q.x, -q.y), pair(kS), accP.rr);
                accP.rr = __ffma2_rn(e, pair(sc), q);
                // xx stays a scalar here: xx sc - rho/3 below then contracts to one fma, which
                // keeps Pi's bits through the cancellation
                accP.jxx.x *= sc; accP.jxx.y *= sc;
                accP.jy *= sc; accP.jz *= sc;
                accP.xy *= sc; accP.yy *= sc; accP.yz *= sc; accP.zz *= sc; accP.xz *= sc;
            }
            const float rho = accP.rr.x;
            const float rr = accP.rr.y;
            const float rb = rho - rr;
            const float inv = fast_rcp(rho);
            float Fbx = 0.0f, Fby = 0.0f, Fbz = 0.0f;
            constexpr bool kF = (kFB & F_FORCE) != 0;
            if (kF && P.forced) {
                Fbx = rho * P.g[0];
                Fby = rho * P.g[1];
                Fbz = rho * P.g[2];
            }
            const float ux = (accP.jxx.x + 0.5f * Fbx) * inv;
            const float uy = (accP.jy + 0.5f * Fby) * inv;
            const float uz = (accP.jz + 0.5f * Fbz) * inv;
            const float ctr = cs2 * rho;
            float pi[6];
            pi[0] = (accP.jxx.y - ctr) - rho * ux * ux;
            pi[1] = accP.xy - rho * ux * uy;
            pi[2] = (accP.yy - ctr) - rho * uy * uy;
            pi[3] = accP.yz - rho * uy * uz;
            pi[4] = (accP.zz - ctr) - rho * uz * uz;
            pi[5] = accP.xz - rho * ux * uz;
            if (kF && P.forced) {
                pi[0] += ux * Fbx;
                pi[1] += 0.5f * (ux * Fby + uy * Fbx);
                pi[2] += uy * Fby;
                pi[3] += 0.5f * (uy * Fbz + uz * Fby);
                pi[4] += uz * Fbz;
                pi[5] += 0.5f * (ux * Fbz + uz * Fbx);
            }
            if (kF && P.ratio) {
                const float Kc = (rr * P.kappa_r + rb * P.kappa_b) * cs2;
                pi[0] -= Kc;
                pi[2] -= Kc;
                pi[4] -= Kc;
            }
            const long long at = static_cast<long long>(d) * P.plane + static_cast<long long>(ys) * P.pitch + xs;
            finalize_store<S>(P, at * static_cast<int>(sizeof(S)), 0U, xs, ys, d, rr, rb, ux, uy, uz, pi, img_x, img_y,
                              key_base);
        }
        if (dest_row) {
            gather(std::integral_constant<int, 0>{}, accC);
            gather(std::integral_constant<int, 1>{}, accN);
        }
        accP = accC;
        accC = accN; // accN is assigned before it is added to again
            return true;
    };
    auto run = [&](auto featc, int kend) -> bool {
        for (; k <= kend; ++k, sl = nxt(sl))
            if (!plane(featc)) return false;
        return true;
    };
    if constexpr ((kFeat & F_WALL) != 0) {
        // walls on the z axis: planes 2 .. nz-5 need none of their part (fluid sources with identity
        // mappings, no wall-adjacent source)
        if (P.bc[2] == MBCG_BC_WALL) {
            const int k0 = max(zd0 - 1, 2), k1 = min(zd1, nz - 5);
            if (k1 >= k0) {
                if (!run(std::integral_constant<int, kFeat>{}, k0 - 1)) return false;
                if (!run(std::integral_constant<int, kFeat & ~F_WALL>{}, k1)) return false;
            }
        }
    }
    if (!run(std::integral_constant<int, kFeat>{}, zd1)) return false;
    // every load of this tile was waited for: carry the parities over to the next tile
    phase = par;
    return true;
}

// the features of the lattices that step by populations in this storage (uses_pop)
template <typename S>
constexpr int pop_features() {
    return std::is_same<S, __nv_bfloat16>::value ? F_WALL | F_FORCE : 0;
}

template <int Q, typename S, int W, bool kTMA, int kFeat>
__global__ void __launch_bounds__(32 * W, W <= 8 ? 2 : 1) step_kernel(const __grid_constant__ StepParams P,
                                                                      const __grid_constant__ TensorMaps T) {
    unsigned char* smem = aligned_smem_base();
    init_barriers<0>(smem);
    wait_prior_grid();
    uint32_t phase = 0;
    tile<Q, S, W, kTMA, kFeat>(P, T.m, blockIdx.x, blockIdx.y, blockIdx.z, P.step, smem, phase);
}

template <int Q, typename S, int W, bool kTMA, int kFeat>
cudaError_t launch_one(const StepParams& P, const TensorMaps& T, cudaStream_t s) {
    auto kern = step_kernel<Q, S, W, kTMA, kFeat>;
    static std::atomic<unsigned long long> configured{0};
    if (cudaError_t e = configure_once(kern, Geo<S, W>::smem, configured)) return e;
    const dim3 grid((P.nx - 2 + kTX - 1) / kTX, (P.ny - 2 + W - 3) / (W - 2), (P.nz - 2 + P.zchunk - 1) / P.zchunk);
    return launch_pdl(kern, grid, dim3(32, W, 1), Geo<S, W>::smem, s, P, T);
}

template <int Q, typename S, int W>
cudaError_t launch_w(bool tma, const StepParams& P, const TensorMaps& T, cudaStream_t s) {
    constexpr int kAll = pop_features<S>();
    if (!tma) return launch_one<Q, S, W, false, kAll>(P, T, s);
    if constexpr (kAll != 0)
        if (features_of(P) != 0) return launch_one<Q, S, W, true, kAll>(P, T, s);
    return launch_one<Q, S, W, true, 0>(P, T, s);
}
template <int Q, typename S>
cudaError_t launch(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s) {
    return w == kStepWSmall ? launch_w<Q, S, kStepWSmall>(tma, P, T, s) : launch_w<Q, S, kStepW>(tma, P, T, s);
}

} // namespace pop

} // namespace

} // namespace mbcg
