// mbcg_step.cuh -- fused moment-based colour-gradient time step for sm_103a (GB300).
//
// step_tile() advances one tile (30 columns x (W-2) rows x a chunk of planes) of one lattice by one
// time step of the reference's main loop (main.cu:41-45):
//   RCS (lbm.cuh:20-262)  +  jet inlet/outlet functors (kernels.cu:102-114)  [+ swap by the host]
// The plain step kernel runs one tile per CTA over a grid covering the lattice; the batch
// kernels (mbcg_batch_kernel.cuh) run tiles of many lattices from a queue in persistent CTAs.  The
// translation units mbcg_step_q{19,27}_{f32,f16,bf16}.cu instantiate the plain kernel.
//
// Formulation.  The reference pulls, for every destination node and direction i, the post-
// collision population of the source node x - c_i and rebuilds it from the source's 11
// moments (feq + oms*fneqr, Omega2 and recolouring at interfaces).  Every one of those
// populations is w_i times a polynomial in c_i (powers a, b, c <= 2 of cx, cy, cz; 17 coefficients)
// that depends only on the source node, and a destination needs only the moments of order <= 2 of what
// it receives.  So each source is visited once and populations are never formed: one axis at a time,
// the polynomial is evaluated at c_a = -1, 0, +1, the outer two values stream to the neighbours along
// that axis, and the receiver sums its moments along it:
//   x: the 8 coefficients (in cy^b cz^c) at cx = -1 and +1 cross to the neighbouring lanes (8 shuffles
//      each way); the column keeps order 0, 1, 2 in x of each,
//   y: those at cy = -1 and +1 go to the neighbouring warps' rows through shared memory (12 values each
//      way for D3Q27, 8 for D3Q19),
//   z: the CTA marches along z; what plane k sends with cz = -1, 0, +1 joins the sums of the destination
//      planes k-1, k, k+1.
// Red populations are the total's times the source's colour fraction plus the recolouring term, itself
// a polynomial whose coefficients are multiples of one vector: an interface source sends three more
// values along x.  The colour gradient F (forces.cuh:20-60) is evaluated once per interface source
// from a ring of psi = (rhor - rhob)/rho planes kept in shared memory.
//
// Two nodes a thread.  A warp holds two rows of the tile, w from below and w from above, one in each
// half of f32x2 registers, the upper one in a frame with y mirrored: both halves take the same
// operations throughout, and every arithmetic instruction does two nodes' work.  The kernel is bound by
// instruction issue and latency, not by HBM (D3Q27 jet 256x256x1024, FP32): 663 warp instructions per 32
// node updates and 12 warps per SM, against 971 and 16 for one node a thread with all 27 populations
// formed and crossing lanes; 2.72 ms -> 1.90 ms a step (24.7 -> 35.4 GLUPS).
//
// Tiling.  A CTA is 32 lanes (x) x W rows (y), W/2 warps.  Lanes 0 and 31 and rows 0 and W-1 are
// halo sources; the CTA writes the 30 x (W-2) destination columns in between, for a chunk of
// planes.  W = 24 (12 warps, one CTA per SM) is the tallest that leaves a thread the 168 registers the
// body needs: W = 16 with 8 warps and 220 registers took 2.69 ms on that jet.  Each source plane arrives
// in shared memory through TMA (cp.async.bulk.tensor.3d, one box per field, 3- or 4-slot ring tracked by
// mbarriers).  The ghost frame of a periodic x / y axis holds the periodic image of the opposite fluid
// layer (every store writes it through), so every source a tile needs is inside its staged box
// (bounds.cuh:34-77 wraps on read instead); the periodic images two layers out that the colour
// gradient needs come from global memory by cp.async.  Warp 0 holds the two halo rows, so it has no
// sums to finish: it issues the copies and prepares the psi elements around the tile meanwhile.
//
// Boundary kinds: periodic; inlet/outlet (the reference's ghost-source branch,
// lbm.cuh:79-151, plus the inlet and outlet functors fused into the store of the first and
// last fluid layer); wall (halfway bounce-back).
//
// Feature sets.  kFeat selects at compile time which optional parts a tile carries:
// F_WALL (bounce-back walls), F_FORCE (body force and density-ratio rest term), F_INOUT (an
// inlet/outlet axis).  A lattice runs on any instantiation whose set covers its parameters;
// the smaller sets leave out code, registers and branches the lattice never uses, and tiles clear of
// the non-periodic axis leave out its parts.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "mbcg_lattice.cuh"
#include "mbcg_internal.h"

namespace mbcg {

namespace {

constexpr int kTX = kStepTileX; // destination columns per CTA (30)
constexpr int kRBX = kStepRBX;   // staged width of rhor/rhob rows (34 needed + 16-byte alignment slack)
constexpr int kMX = kStepMX;     // staged width of the other 9 fields (32 needed + slack)
constexpr int kPSX = 34;   // psi ring width (32 sources + 1 on each side)
constexpr int kMaxStages = 4; // planes staged at most: k, k+1, and k+2, k+3 in flight
constexpr int kPlaneBar = kMaxStages + 1; // the warps' barrier of a plane (after the stages' and the test's)
constexpr int kYBar = kPlaneBar + 1;      // and one for each warp
constexpr unsigned kFull = 0xffffffffu;

constexpr int align128(int b) { return (b + 127) / 128 * 128; }

// Shared-memory carve-up of one tile: the mbarriers in the first 256 bytes, then the staged
// planes, the psi ring and the y-exchange buffer.  `smem` is the dynamic size to request (it
// includes 128 bytes of slack for aligning the base).
template <typename S, int W>
struct Geo {
    // planes staged: k, k+1, and two more in flight, or one where the tile leaves no room for two
    static constexpr int NST = W > 16 && sizeof(S) == 4 ? 3 : kMaxStages;
    static constexpr int RBY = W + 2;
    static constexpr int MY = W;
    static constexpr int rb_field = align128(RBY * kRBX * (int)sizeof(S));
    static constexpr int m_field = align128(MY * kMX * (int)sizeof(S));
    static constexpr int stage = 2 * rb_field + 9 * m_field;
    static constexpr int tx = 2 * RBY * kRBX * (int)sizeof(S) + 9 * MY * kMX * (int)sizeof(S);
    static constexpr int psi_plane = RBY * kPSX;           // floats
    static constexpr int psi = NST * psi_plane * 4;    // bytes (ring slot = stage slot)
    static constexpr int H = W / 2;                        // warps: two rows each
    static constexpr int xbuf = 25 * (H + 1) * 32 * 8;     // float2 [quantity][warp, one more][lane]
    // psi elements beside the source nodes inside the lattice: the frame around the tile, and the
    // column nx and row ny where the lattice ends inside it
    static constexpr int frame = 2 * kPSX + 2 * W + (W + 2) + kPSX;
    static constexpr int ftab = align128(frame * 8 + 8);   // int2 [element], then the two list lengths
    static constexpr int fbuf = align128(frame * 8);       // uint2 [far element]: words of fields 0 and 1
    static constexpr int off_bar = 0;
    static constexpr int off_stage = 256;
    static constexpr int off_psi = off_stage + NST * stage;
    static constexpr int off_xbuf = off_psi + psi;
    static constexpr int off_ftab = off_xbuf + xbuf;
    static constexpr int off_fbuf = off_ftab + ftab;
    static constexpr int smem = off_fbuf + fbuf + 128;
};

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after ~limit clock cycles instead of spinning forever.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, long long limit) {
    if (mbar_try_wait(bar, parity)) return true; // the usual case: the plane is already there
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > limit) return false;
    }
    return true;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
// (zeros, without reading src, if not `valid`)
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid = true) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)),
                 "l"(__cvta_generic_to_global(src)), "r"(valid ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Programmatic dependent launch: lets the next kernel of the stream start its set-up once every CTA of
// this one has said so or is done, and waits for the kernel before this one to be complete.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ int floor8(int v) { return v & ~7; }

// ------------------------------------------------------------------ coordinate roles
enum Role : int { R_FLUID = 0, R_IMAGE = 1, R_GHOST = 2, R_WALL = 3, R_OUT = 4 };

template <int kFeat>
__device__ __forceinline__ int axis_role(const StepParams& P, int a, int p, int n) {
    if (p < 0 || p > n - 1) return R_OUT;
    if (p == 0 || p == n - 1) {
        if constexpr ((kFeat & (F_WALL | F_INOUT)) == 0) return R_IMAGE;
        const int k = P.bc[a];
        return k == MBCG_BC_PERIODIC ? R_IMAGE : (k == MBCG_BC_INOUT ? R_GHOST : R_WALL);
    }
    return R_FLUID;
}
__device__ __forceinline__ int data_coord(const StepParams& P, int a, int p, int n) {
    return (P.bc[a] == MBCG_BC_PERIODIC) ? periodic_image(p, n) : min(max(p, 0), n - 1);
}
// neighbour rule of the colour gradient (forces.cuh:28-31, mathUtilities.cuh:25-33)
__device__ __forceinline__ int psi_coord(const StepParams& P, int a, int p, int n) {
    const int k = P.bc[a];
    if (k == MBCG_BC_PERIODIC) return periodic_image(p, n);
    if (k == MBCG_BC_INOUT) return p >= n - 1 ? n - 2 : max(p, 0);
    return min(max(p, 1), n - 2);
}

// ------------------------------------------------------------------ state access
// Fast reciprocal (<= 1 ulp, one MUFU instruction).  The flushing form: for the densities and
// gradients it is used on (far from the subnormal range) it gives the same value as
// __fdividef(1, v), which spends four more instructions on scaling subnormal operands.
__device__ __forceinline__ float fast_rcp(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

template <typename S>
struct Node {
    float rr, rb, ux, uy, uz, pxx, pxy, pyy, pyz, pzz, pxz;
};

template <typename S>
__device__ __forceinline__ float psi_of(const StepParams& P, S s0, S s1) {
    if constexpr (std::is_same<S, float>::value) {
        const float r = Codec<S>::to_f(s0), b = Codec<S>::to_f(s1);
        return (r - b) * fast_rcp(r + b);
    } else {
        (void)P;
        (void)s0;
        return phi_of_slot(Codec<S>::to_f(s1));
    }
}

// psi from the two stored slots already widened to float
template <typename S>
__device__ __forceinline__ float psi_of_slots(float v0, float v1) {
    if constexpr (std::is_same<S, float>::value) return (v0 - v1) * fast_rcp(v0 + v1);
    else return phi_of_slot(v1);
}

// decode the 11 stored slots into the reference's moments
template <typename S>
__device__ __forceinline__ void decode(const StepParams& P, const float (&v)[NF], Node<S>& n) {
    if constexpr (sizeof(S) == 4) {
        n.rr = v[0]; n.rb = v[1]; n.ux = v[2]; n.uy = v[3]; n.uz = v[4];
        n.pxx = v[5]; n.pxy = v[6]; n.pyy = v[7]; n.pyz = v[8]; n.pzz = v[9]; n.pxz = v[10];
    } else {
        const float phi = phi_of_slot(v[1]);
        const float rho = P.rho_mean + phi * P.rho_half_diff + P.rho_scale * v[0];
        colour_split(v[1], rho, n.rr, n.rb);
        n.ux = P.u_ref * v[2]; n.uy = P.u_ref * v[3]; n.uz = P.u_ref * v[4];
        n.pxx = P.pi_scale * v[5]; n.pxy = P.pi_scale * v[6]; n.pyy = P.pi_scale * v[7];
        n.pyz = P.pi_scale * v[8]; n.pzz = P.pi_scale * v[9]; n.pxz = P.pi_scale * v[10];
    }
}

// The 16-bit forms round every stored slot stochastically (`key`: the node's random stream).
// Rounded to nearest, a slowly changing state is rounded the same way step after step and the
// errors add up (field error growing in proportion to the step count); rounded stochastically
// they are unbiased and independent from step to step.
template <typename S>
__device__ __forceinline__ void encode(const StepParams& P, float rr, float rb, const float (&u)[3],
                                       const float (&pi)[6], S (&out)[NF], unsigned key) {
    if constexpr (sizeof(S) == 4) {
        (void)key;
        out[0] = rr; out[1] = rb; out[2] = u[0]; out[3] = u[1]; out[4] = u[2];
        for (int i = 0; i < 6; ++i) out[5 + i] = pi[i];
    } else {
        const float rho = rr + rb;
        S unused;
        // a minority density a rounding error below zero is zero: its sign would turn the slot's, and
        // with it the node's colour
        Codec<S>::from_f_sr(colour_slot(fmaxf(rr, 0.0f), fmaxf(rb, 0.0f), rho), 0.0f, lowbias32(key), out[1], unused);
        const float phi = phi_of_slot(Codec<S>::to_f(out[1])); // the phi a reader decodes
        Codec<S>::from_f_sr((rho - (P.rho_mean + phi * P.rho_half_diff)) * P.inv_rho_scale, u[0] * P.inv_u_ref,
                            lowbias32(key + 1), out[0], out[2]);
        Codec<S>::from_f_sr(u[1] * P.inv_u_ref, u[2] * P.inv_u_ref, lowbias32(key + 2), out[3], out[4]);
        Codec<S>::from_f_sr(pi[0] * P.inv_pi_scale, pi[1] * P.inv_pi_scale, lowbias32(key + 3), out[5], out[6]);
        Codec<S>::from_f_sr(pi[2] * P.inv_pi_scale, pi[3] * P.inv_pi_scale, lowbias32(key + 4), out[7], out[8]);
        Codec<S>::from_f_sr(pi[4] * P.inv_pi_scale, pi[5] * P.inv_pi_scale, lowbias32(key + 5), out[9], out[10]);
    }
}

// random stream of node (x, y, z) given the step's key base: six consecutive keys per node
__device__ __forceinline__ unsigned node_round_key(const StepParams& P, unsigned base, int x, int y, int z) {
    // unsigned arithmetic: the index wraps (harmlessly) on lattices beyond 2^32 nodes
    const unsigned node = (static_cast<unsigned>(z) * static_cast<unsigned>(P.ny) + static_cast<unsigned>(y)) *
                              static_cast<unsigned>(P.nx) +
                          static_cast<unsigned>(x);
    return base + 6U * node;
}

// Store a node at byte offset `off` from `tile` (bytes) in every field.  The offset within a tile's
// planes fits 32 bits (the launch caps zchunk for it), so each store is a uniform base and one
// 32-bit register instead of a 64-bit sum per field.
template <typename S>
__device__ __forceinline__ void store_node(const StepParams& P, long long tile, unsigned off, const S (&v)[NF]) {
#pragma unroll
    for (int f = 0; f < NF; ++f)
        *reinterpret_cast<S*>(static_cast<unsigned char*>(P.b[f]) + tile + off) = v[f];
}

template <typename S>
__device__ __forceinline__ void load_global(const StepParams& P, long long o, float (&v)[NF]) {
#pragma unroll
    for (int f = 0; f < NF; ++f) v[f] = Codec<S>::to_f(static_cast<const S*>(P.a[f])[o]);
}

// ------------------------------------------------------------------ packed pairs
// Every thread advances two nodes of its column, one in each half of f32x2 registers
// (add / mul / fma .rn.f32x2, sm_100 and later: two FP32 operations per issued instruction, each
// rounded exactly like the scalar one).
using F2 = float2;
__device__ __forceinline__ F2 pair(float v) { return make_float2(v, v); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ F2 operator*(float a, F2 b) { return __fmul2_rn(pair(a), b); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
    F2 r;
    asm("{.reg .b64 pa, pb, pd;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\t"
        "sub.rn.f32x2 pd, pa, pb;\n\tmov.b64 {%0, %1}, pd;}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ F2 fma2(float a, F2 b, F2 c) { return __ffma2_rn(pair(a), b, c); }
__device__ __forceinline__ F2 neg2(F2 a) { return make_float2(-a.x, -a.y); } // a free operand modifier
__device__ __forceinline__ F2 swap2(F2 a) { return make_float2(a.y, a.x); }
__device__ __forceinline__ F2 shfl_up2(F2 v) {
    return make_float2(__shfl_up_sync(kFull, v.x, 1), __shfl_up_sync(kFull, v.y, 1));
}
__device__ __forceinline__ F2 shfl_down2(F2 v) {
    return make_float2(__shfl_down_sync(kFull, v.x, 1), __shfl_down_sync(kFull, v.y, 1));
}

// ------------------------------------------------------------------ source coefficients
// Phase-dependent relaxation (forces.cuh:101-108): tau_eff = (1 + psi)/2 tau_r + (1 - psi)/2 tau_b
__device__ __forceinline__ float tau_eff_of(const StepParams& P, float rr, float rb) {
    const float psix = (rr - rb) / (rr + rb);
    return 0.5f * (1.0f + psix) * P.tau_r + 0.5f * (1.0f - psix) * P.tau_b;
}

// Moments of a source pair.
struct Node2 {
    F2 rr, rb, ux, uy, uz, pxx, pxy, pyy, pyz, pzz, pxz;
};

// Decode the stored slots of this thread's two nodes; the second node's y axis is mirrored (see
// step_tile), so its y-odd moments change sign.  The 16-bit forms leave Pi in units of pi_scale: the
// relaxation factor it is multiplied by carries that.
template <typename S>
__device__ __forceinline__ void decode2(const StepParams& P, const float (&va)[NF], const float (&vb)[NF], Node2& n) {
    auto even = [&](int f) { return make_float2(va[f], vb[f]); };
    auto odd = [&](int f) { return make_float2(va[f], -vb[f]); };
    if constexpr (sizeof(S) == 4) {
        n.rr = even(0);
        n.rb = even(1);
        n.ux = even(2);
        n.uy = odd(3);
        n.uz = even(4);
    } else {
        const F2 phi = make_float2(phi_of_slot(va[1]), phi_of_slot(vb[1]));
        const F2 rho = fma2(P.rho_scale, even(0), fma2(P.rho_half_diff, phi, pair(P.rho_mean)));
        const F2 minor = (0.5f * rho) * make_float2(fabsf(va[1]), fabsf(vb[1]));
        const F2 major = rho - minor;
        const bool ra = !signbit(va[1]), rb = !signbit(vb[1]); // red is the majority
        n.rr = make_float2(ra ? major.x : minor.x, rb ? major.y : minor.y);
        n.rb = make_float2(ra ? minor.x : major.x, rb ? minor.y : major.y);
        n.ux = P.u_ref * even(2);
        n.uy = P.u_ref * odd(3);
        n.uz = P.u_ref * even(4);
    }
    n.pxx = even(5);
    n.pxy = odd(6);
    n.pyy = even(7);
    n.pyz = odd(8);
    n.pzz = even(9);
    n.pxz = even(10);
}
// encode() of a pair of nodes: the same values, the arithmetic packed.  ir: the reciprocal density; keys of
// both nodes.  With decode2() it takes the D3Q27 jet 256x256x1024 in FP16 from 2.33 to 2.30 ms, the 128^3
// RTI in FP16 from 745 to 724 us.
template <typename S>
__device__ __forceinline__ void encode2(const StepParams& P, F2 rr, F2 rb, F2 ir, const F2 (&u)[3], const F2 (&pi)[6],
                                        S (&oa)[NF], S (&ob)[NF], unsigned ka, unsigned kb) {
    if constexpr (sizeof(S) == 4) {
        const F2 v[NF] = {rr, rb, u[0], u[1], u[2], pi[0], pi[1], pi[2], pi[3], pi[4], pi[5]};
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            oa[f] = v[f].x;
            ob[f] = v[f].y;
        }
    } else {
        auto put = [&](F2 p, F2 q, unsigned i, int fp, int fq) {
            Codec<S>::from_f_sr(p.x, q.x, lowbias32(ka + i), oa[fp], oa[fq]);
            Codec<S>::from_f_sr(p.y, q.y, lowbias32(kb + i), ob[fp], ob[fq]);
        };
        const F2 rho = rr + rb, lead = rr - rb; // lead >= 0: red is the majority
        // a minority density a rounding error below zero is zero: its sign would turn the slot's, and
        // with it the node's colour
        const F2 minor = make_float2(fmaxf(fminf(rr.x, rb.x), 0.0f), fmaxf(fminf(rr.y, rb.y), 0.0f));
        const F2 c = (2.0f * minor) * ir;
        S unused;
        Codec<S>::from_f_sr(copysignf(c.x, lead.x), 0.0f, lowbias32(ka), oa[1], unused);
        Codec<S>::from_f_sr(copysignf(c.y, lead.y), 0.0f, lowbias32(kb), ob[1], unused);
        // the phi a reader decodes
        const F2 phi = make_float2(phi_of_slot(Codec<S>::to_f(oa[1])), phi_of_slot(Codec<S>::to_f(ob[1])));
        const float iu = P.inv_u_ref, is = P.inv_pi_scale;
        put(P.inv_rho_scale * (rho - fma2(P.rho_half_diff, phi, pair(P.rho_mean))), iu * u[0], 1, 0, 2);
        put(iu * u[1], iu * u[2], 2, 3, 4);
        put(is * pi[0], is * pi[1], 3, 5, 6);
        put(is * pi[2], is * pi[3], 4, 7, 8);
        put(is * pi[4], is * pi[5], 5, 9, 10);
    }
}

// The post-collision population of direction c, divided by its weight and less the reference
// density, is a polynomial in c:
//   rhod + p000 + p100 cx + p010 cy + p001 cz + 3/2 (exx cx^2 + eyy cy^2 + ezz cz^2)
//   + 3 (exy cx cy + exz cx cz + eyz cy cz)
//   + 9/2 (kxxy cx^2 cy + kxxz cx^2 cz + kxyy cx cy^2 + kxzz cx cz^2 + kyyz cy^2 cz + kyzz cy cz^2)
//   + 9 kxyz cx cy cz
// with the numeric factors left out of the coefficients: they fold into the multiply-adds of the
// transform.  Equilibrium (pdf.cuh:16-36) at (rho, u) + oms * regularised non-equilibrium
// (pdf.cuh:38-79) from (Pi, v) + 1/2 Guo force (pdf.cuh:94-136); v = u except at ghost sources
// (kGhost), whose non-equilibrium part comes from the fluid node behind them.
struct Coef {
    F2 p000, p100, p010, p001, exx, eyy, ezz, exy, exz, eyz;
    F2 kxxy, kxxz, kxyy, kxzz, kyyz, kyzz, kxyz;
};

template <int kFeat>
__device__ __forceinline__ void build_coef(const StepParams& P, Coef& c, const Node2& n, F2 rho, F2 vx, F2 vy, F2 vz,
                                           F2 o3, F2 fgx, F2 fgy, F2 fgz) {
    constexpr bool kGhost = (kFeat & F_INOUT) != 0, kF = (kFeat & F_FORCE) != 0;
    const F2 r3 = 3.0f * rho;
    const F2 nx = r3 * n.ux, ny = r3 * n.uy, nz = r3 * n.uz;
    const F2 fxx = o3 * n.pxx, fyy = o3 * n.pyy, fzz = o3 * n.pzz;
    const F2 fxy = o3 * n.pxy, fxz = o3 * n.pxz, fyz = o3 * n.pyz;
    c.exx = fma2(nx, n.ux, fxx);
    c.eyy = fma2(ny, n.uy, fyy);
    c.ezz = fma2(nz, n.uz, fzz);
    c.exy = fma2(nx, n.uy, fxy);
    c.exz = fma2(nx, n.uz, fxz);
    c.eyz = fma2(ny, n.uz, fyz);
    F2 dxy = fxy + fxy, dxz = fxz + fxz, dyz = fyz + fyz;
    if constexpr (!kGhost) {
        F2 gxy = dxy, gyx = dxy, gxz = dxz, gzx = dxz, gyz = dyz, gzy = dyz, hxz = fxz;
        F2 exx = c.exx, eyy = c.eyy, ezz = c.ezz, exy = c.exy;
        if constexpr (kF) {
            if (P.forced) {
                // s_ab = 3/2 F_b u_a; the force adds s_ab + s_ba to e_ab
                const F2 h = 1.5f * rho;
                const F2 Fx = h * fgx, Fy = h * fgy, Fz = h * fgz;
                const F2 sxy = Fy * n.ux, syx = Fx * n.uy, sxz = Fz * n.ux, szx = Fx * n.uz, syz = Fz * n.uy, szy = Fy * n.uz;
                exx = c.exx = fma2(2.0f, Fx * n.ux, c.exx);
                eyy = c.eyy = fma2(2.0f, Fy * n.uy, c.eyy);
                ezz = c.ezz = fma2(2.0f, Fz * n.uz, c.ezz);
                exy = c.exy = c.exy + (sxy + syx);
                c.exz = c.exz + (sxz + szx);
                c.eyz = c.eyz + (syz + szy);
                gxy = gxy + sxy;
                gyx = gyx + syx;
                gxz = gxz + sxz;
                gzx = gzx + szx;
                gyz = gyz + syz;
                gzy = gzy + szy;
                hxz = hxz + sxz;
            }
        }
        c.kxxy = fma2(gxy, n.ux, exx * n.uy);
        c.kxxz = fma2(gxz, n.ux, exx * n.uz);
        c.kxyy = fma2(gyx, n.uy, eyy * n.ux);
        c.kyyz = fma2(gyz, n.uy, eyy * n.uz);
        c.kxzz = fma2(gzx, n.uz, ezz * n.ux);
        c.kyzz = fma2(gzy, n.uz, ezz * n.uy);
        c.kxyz = fma2(fyz, n.ux, fma2(hxz, n.uy, exy * n.uz));
    } else {
        F2 qxx = nx * n.ux, qyy = ny * n.uy, qzz = nz * n.uz, qxy = nx * n.uy;
        c.kxxy = fma2(dxy, vx, fma2(fxx, vy, qxx * n.uy));
        c.kxxz = fma2(dxz, vx, fma2(fxx, vz, qxx * n.uz));
        c.kxyy = fma2(dxy, vy, fma2(fyy, vx, qyy * n.ux));
        c.kyyz = fma2(dyz, vy, fma2(fyy, vz, qyy * n.uz));
        c.kxzz = fma2(dxz, vz, fma2(fzz, vx, qzz * n.ux));
        c.kyzz = fma2(dyz, vz, fma2(fzz, vy, qzz * n.uy));
        c.kxyz = fma2(fyz, vx, fma2(fxz, vy, fma2(fxy, vz, qxy * n.uz)));
        if constexpr (kF) {
            if (P.forced) {
                const F2 h = 1.5f * rho;
                const F2 Fx = h * fgx, Fy = h * fgy, Fz = h * fgz;
                const F2 sxx = Fx * n.ux, syy = Fy * n.uy, szz = Fz * n.uz;
                const F2 sxy = Fy * n.ux, syx = Fx * n.uy, sxz = Fz * n.ux, szx = Fx * n.uz, syz = Fz * n.uy, szy = Fy * n.uz;
                c.exx = fma2(2.0f, sxx, c.exx);
                c.eyy = fma2(2.0f, syy, c.eyy);
                c.ezz = fma2(2.0f, szz, c.ezz);
                c.exy = c.exy + (sxy + syx);
                c.exz = c.exz + (sxz + szx);
                c.eyz = c.eyz + (syz + szy);
                c.kxxy = c.kxxy + fma2(sxy, n.ux, 2.0f * (sxx * n.uy));
                c.kxxz = c.kxxz + fma2(sxz, n.ux, 2.0f * (sxx * n.uz));
                c.kxyy = c.kxyy + fma2(syx, n.uy, 2.0f * (syy * n.ux));
                c.kyyz = c.kyyz + fma2(syz, n.uy, 2.0f * (syy * n.uz));
                c.kxzz = c.kxzz + fma2(szx, n.uz, 2.0f * (szz * n.ux));
                c.kyzz = c.kyzz + fma2(szy, n.uz, 2.0f * (szz * n.uy));
                c.kxyz = c.kxyz + fma2(sxz, n.uy, (sxy + syx) * n.uz);
            }
        }
    }
    c.p100 = fma2(-1.5f, c.kxyy + c.kxzz, nx);
    c.p010 = fma2(-1.5f, c.kxxy + c.kyzz, ny);
    c.p001 = fma2(-1.5f, c.kxxz + c.kyyz, nz);
    if constexpr (kF) {
        if (P.forced) {
            const F2 h = 1.5f * rho;
            c.p100 = fma2(h, fgx, c.p100);
            c.p010 = fma2(h, fgy, c.p010);
            c.p001 = fma2(h, fgz, c.p001);
        }
    }
    // the isotropic part from the same rounded e as the anisotropic one, so that the second-order
    // terms sum to zero over the directions
    c.p000 = -0.5f * (c.exx + c.eyy + c.ezz);
}

// Sums of one destination pair over the directions received so far (weights scaled to integers): tot (less
// the reference density), red (likewise less part E), momentum and second moments in the plane.  Those with
// cz need none of their own while a plane is plane k: they are what came with cz = +1 (walls aside).
struct Acc2 {
    F2 tot, red, E, jx, jy, xx, xy, yy;
    __device__ __forceinline__ void zero() { tot = red = E = jx = jy = xx = xy = yy = make_float2(0.0f, 0.0f); }
};

// ------------------------------------------------------------------ the kernel

// On periodic x / y axes the first and last fluid layers are also written to their image in the
// opposite ghost layer, so the next step reads every source (including wrapped ones) from the staged
// box (bounds.cuh:34-77 wraps on read instead).  tile / off: the node's address, as in store_node;
// ix / iy: the column's periodic image in x / y (-1: none).
template <typename S>
__device__ __forceinline__ void store_images(const StepParams& P, long long tile, unsigned off, int x, int y,
                                             const S (&out)[NF], int ix, int iy) {
    const long long dx = static_cast<long long>(ix - x) * static_cast<int>(sizeof(S));
    const long long dy = static_cast<long long>(iy - y) * P.pitch * static_cast<int>(sizeof(S));
    if (ix >= 0) store_node<S>(P, tile + dx, off, out);
    if (iy >= 0) store_node<S>(P, tile + dy, off, out);
    if (ix >= 0 && iy >= 0) store_node<S>(P, tile + dx + dy, off, out);
}
// Store one node at (x, y, z) and its images.
template <typename S>
__device__ __forceinline__ void finalize_store(const StepParams& P, long long tile, unsigned off, int x, int y, int z,
                                               float rr, float rb, float ux, float uy, float uz, const float (&pi)[6],
                                               int ix, int iy, unsigned key_base) {
    const float u[3] = {ux, uy, uz};
    S out[NF];
    encode<S>(P, rr, rb, u, pi, out, sizeof(S) == 4 ? 0U : node_round_key(P, key_base, x, y, z));
    store_node<S>(P, tile, off, out);
    if ((ix & iy) != -1) store_images<S>(P, tile, off, x, y, out, ix, iy); // either is >= 0
}

// 128-byte aligned base of the dynamic shared memory (TMA destinations need it; every Geo
// size carries the slack).  Plain pointer arithmetic on the shared array, so that the compiler
// knows every access through it for a shared-memory one (LDS / STS with 32-bit addresses; through
// an integer cast they become generic accesses with 64-bit address arithmetic).
__device__ __forceinline__ unsigned char* aligned_smem_base() {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    return smem_raw + ((128U - (smem_u32(smem_raw) & 127U)) & 127U);
}

// Initialise the mbarriers (one elected thread) before the first tile of a CTA.  The one after the
// stages' is never arrived at: the bounded-wait test hook waits on it.  kPlaneBar counts the H warps of a
// CTA, kYBar + w the warps that warp w waits for in the y exchange: those of the rows beside its own (the
// innermost is its own neighbour), or, warp 0, all others.
template <int H>
__device__ __forceinline__ void init_barriers(unsigned char* smem) {
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        for (int s = 0; s <= kMaxStages; ++s) mbar_init(&bars[s], 1);
        if constexpr (H > 0) {
            mbar_init(&bars[kPlaneBar], H);
            for (int w = 0; w < H; ++w) mbar_init(&bars[kYBar + w], w == 0 ? H - 1 : (w < H - 1 ? 2 : 1));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

// One tile of one time step.  (bx, by, bz) index the tile in the lattice's tile grid; `step`
// is the index of the state being written (keys the inlet noise); `phase` carries the parities
// of the mbarriers (a bit for each stage's, for kPlaneBar and for kYBar) from one tile of a CTA to the next
// (0 before the first tile), also to a tile of another body.
// Returns false if a staged plane never arrived (the status word is set and the CTA must stop).
// kStride: a tile of a batch kernel, whose CTAs run many.  The next state's fields lie P.b_stride bytes apart
// (states the library owns): with the parameters from a table, that keeps one pointer instead of eleven.
template <int Q, typename S, int W, bool kTMA, int kFeat, bool kStride = false>
__device__ __forceinline__ bool step_tile(const StepParams& P, const CUtensorMap* maps, int bx, int by, int bz,
                                          long long step, unsigned char* smem, uint32_t& phase) {
    using G = Geo<S, W>;
    float* psi_ring = reinterpret_cast<float*>(smem + G::off_psi);
    float2* xbuf = reinterpret_cast<float2*>(smem + G::off_xbuf);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + G::off_bar);

    const int lane = threadIdx.x;
    const int w = threadIdx.y;
    constexpr int H = G::H;       // warps of the CTA
    constexpr int kThreads = 32 * H;
    constexpr bool kSepW = (Q == 27);
    constexpr int kNSTAGE = G::NST;
    const int tid = w * 32 + lane;
    const int nx = P.nx, ny = P.ny, nz = P.nz;

    const int xb = kTX * bx;     // source column of lane 0
    const int yb = (W - 2) * by; // source row 0
    const int xs = xb + lane;
    // this thread's rows: w from below and w from above.  The second is computed in a frame with y
    // mirrored, where both rows have warp w-1 behind them (outwards) and warp w+1 before them, so
    // the two halves take the same operations everywhere.
    const int wa = w, wb = W - 1 - w;
    const int ysa = yb + wa, ysb = yb + wb;
    int zd0, zd1; // destination planes
    z_range(nz, P.bc[2], P.zchunk, bz, zd0, zd1);
    const int kfirst = zd0 - 2;

    const int xr0 = floor8(xb - 1); // first staged column of rhor/rhob
    const int xm0 = floor8(xb);     // first staged column of the other fields
    const int offRB = xb - xr0;
    const int offM = xb - xm0;
    // these nodes in the rhor/rhob boxes and in the other boxes
    const int bRa = (wa + 1) * kRBX + lane + offRB, bRb = (wb + 1) * kRBX + lane + offRB;
    const int bMa = wa * kMX + lane + offM, bMb = wb * kMX + lane + offM;

    const bool dest_x = lane >= 1 && lane <= kTX && xs <= nx - 2 && w >= 1; // warp 0: the halo rows
    const bool dest_a = dest_x && ysa <= ny - 2, dest_b = dest_x && ysb <= ny - 2;
    const int rx = axis_role<kFeat>(P, 0, xs, nx);
    const int rya = axis_role<kFeat>(P, 1, ysa, ny), ryb = axis_role<kFeat>(P, 1, ysb, ny);
    const bool in_xy_a = rx != R_OUT && rya != R_OUT, in_xy_b = rx != R_OUT && ryb != R_OUT;
    const int ia = P.inout_axis;
    // a node's role, given the roles of its row and plane
    auto role_of = [&](int ry, int rz) -> int {
        if (rx == R_OUT || ry == R_OUT || rz == R_OUT) return R_OUT;
        if ((kFeat & F_WALL) && (rx == R_WALL || ry == R_WALL || rz == R_WALL)) return R_WALL;
        if ((kFeat & F_INOUT) && (rx == R_GHOST || ry == R_GHOST || rz == R_GHOST)) return R_GHOST;
        return R_FLUID;
    };
    const int role_xy[2] = {role_of(rya, R_FLUID), role_of(ryb, R_FLUID)}; // on fluid planes
    // stochastic rounding of the 16-bit stores: key base of this step
    const unsigned key_base = sizeof(S) == 4 ? 0U : round_key_base(P.seed, step);
    // periodic images of this column's stores (x = 1 / nx-2, y = 1 / ny-2 on a periodic axis)
    auto image_of = [&](int a, int p, int n) {
        return P.bc[a] == MBCG_BC_PERIODIC ? (p == 1 ? n - 1 : (p == n - 2 ? 0 : -1)) : -1;
    };
    const bool images = (image_of(0, xs, nx) & image_of(1, ysa, ny) & image_of(1, ysb, ny)) != -1; // any

    // psi ring: each thread fills its two nodes' elements.  pa / pb: the box element whose psi stands
    // for the node (itself; on non-periodic x / y axes the colour-gradient rule maps ghost layers).
    constexpr bool kMapXY = (kFeat & (F_WALL | F_INOUT)) != 0;
    auto own_coord = [&](int a, int p, int n) {
        const int kind = P.bc[a];
        if (kind == MBCG_BC_INOUT) return p >= n - 1 ? n - 2 : p;
        return kind == MBCG_BC_WALL ? min(max(p, 1), n - 2) : p;
    };
    const int pxo = kMapXY ? own_coord(0, xs, nx) : xs;
    const int pya = kMapXY ? own_coord(1, ysa, ny) : ysa, pyb = kMapXY ? own_coord(1, ysb, ny) : ysb;
    const int bPa = (pya - (yb - 1)) * kRBX + pxo - xr0, bPb = (pyb - (yb - 1)) * kRBX + pxo - xr0;

    // Plane k lives in stage slot (k - kfirst) mod kNSTAGE, and its psi in the ring slot of the same
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
        } else if constexpr (sizeof(S) == 4) {
            // layouts TMA cannot describe (row pitch not a multiple of 16 bytes): every thread copies its
            // two nodes by 4-byte cp.async (no one else reads them, but for the elements beside a
            // boundary); zeros outside the lattice, as TMA fills
            const long long zo = static_cast<long long>(kz) * P.plane;
            auto node = [&](int ys, int iR, int iM) {
                const bool in = xs < nx && ys < ny;
                const long long o = zo + (in ? static_cast<long long>(ys) * P.pitch + xs : 0);
#pragma unroll
                for (int f = 0; f < NF; ++f)
                    cp_async4(f < 2 ? rb_box(st, f) + iR : m_box(st, f) + iM, static_cast<const S*>(P.a[f]) + o, in);
            };
            node(ysa, bRa, bMa);
            node(ysb, bRb, bMb);
        } else {
            // 16-bit elements (a copy moves four bytes at least): plain loads and stores
            const long long zo = static_cast<long long>(kz) * P.plane;
            auto node = [&](int ys, int iR, int iM) {
                const bool in = xs < nx && ys < ny;
                const long long o = zo + static_cast<long long>(ys) * P.pitch + xs;
#pragma unroll
                for (int f = 0; f < NF; ++f)
                    (f < 2 ? rb_box(st, f)[iR] : m_box(st, f)[iM]) =
                        in ? static_cast<const S*>(P.a[f])[o] : Codec<S>::from_f(0.0f);
            };
            node(ysa, bRa, bMa);
            node(ysb, bRb, bMb);
        }
    };
    constexpr long long kWaitLimit = 4000000000LL; // ~2 s at 2 GHz
    // Expected parity of the next phase of each slot's mbarrier; every completed wait flips it.
    // It starts from the parities the previous tile of this CTA left.
    uint32_t par = phase;
    int k_waited = kfirst - 1; // last plane whose load was waited for
    auto wait_slot = [&](int k, int sl) -> bool {
        if constexpr (kTMA) {
            const bool ok = mbar_wait_bounded(&bars[sl], (par >> sl) & 1u, kWaitLimit);
            if (ok) {
                par ^= 1u << sl;
                k_waited = k;
            }
            return ok;
        } else {
            k_waited = k;
            return true;
        }
    };
    // warp 0 looks at a plane before the CTA's own wait for it
    auto peek_slot = [&](int sl) -> bool {
        if constexpr (kTMA) return mbar_wait_bounded(&bars[sl], (par >> sl) & 1u, kWaitLimit);
        else return true;
    };
    // ---- the warps' synchronisation within a plane: psi of plane k+1 in the ring and the y exchange of
    // plane k-1 read (kPlaneBar, every warp for every warp), then the y exchange of plane k written and the
    // plane's fields and psi read.  A warp needs the latter of warps w-1 and w+1 only, warp 0, which refills
    // the ring, of all: kNearBar has each warp wait for just these, on a barrier of its own.  No warp arrives
    // there twice before the waiting one has passed: kPlaneBar comes between.
    // The slowest warp of a plane then does not hold the others: D3Q27 jet 256x256x1024 1.94 -> 1.90 ms, in
    // FP16 2.46 -> 2.33 ms; periodic 192^3 507 -> 493 us; 128^3 RTI 665 -> 652 us, in FP16 794 -> 745 us.  One
    // barrier of the CTA is the better where the warps are few (W = 8: periodic 64^3 493 against 515 us for
    // 20 steps) and in bodies with an inlet (128^3 jet along y, 456 against 469 us for 4 steps).
    constexpr bool kNearBar = kTMA && W > 8 && (kFeat & F_INOUT) == 0;
    // this lane's kYBar to arrive at
    int y_target = -1;
    if (lane == 0) y_target = w == 0 ? 1 : 0;
    if (lane == 1 && w >= 1 && w < H - 1) y_target = w + 1;
    if (lane == 2 && w >= 2) y_target = w - 1;
    // In a batch kernel the two kinds of barrier keep a parity bit each: a tile of a body without kNearBar
    // passes kPlaneBar every plane and kYBar never, and a neighbour-wise tile may follow it.  A plain CTA
    // runs one tile, which passes both alike: one bit, two instructions a plane fewer (periodic 192^3 493
    // against 496 us for 2 steps).
    constexpr int kYBit = kStride ? kYBar : kPlaneBar;
    auto plane_wait = [&]() { return mbar_wait_bounded(&bars[kPlaneBar], (par >> kPlaneBar) & 1u, kWaitLimit); };
    auto y_wait = [&]() { return mbar_wait_bounded(&bars[kYBar + w], (par >> kYBit) & 1u, kWaitLimit); };
    // On a failed wait: flag it, drain the copies still in flight (bounded) and leave.  If the drain
    // gives up too, copies may still land in this block's shared memory after it exits, which the
    // status cannot tell apart (a flag for it once cost the batch kernel 3-5 %): the host treats
    // any non-zero status as a poisoned context.
    auto bail = [&](int k_issued) {
        if (tid == 0 && P.status) atomicOr(P.status, 1);
        if constexpr (kTMA) {
            for (int k = k_waited + 1; w == 0 && k <= k_issued; ++k) {
                const int sl = (k - kfirst) % kNSTAGE;
                mbar_wait_bounded(&bars[sl], (par >> sl) & 1u, kWaitLimit / 4);
            }
        }
    };

    // ---- psi ring: psi = (rhor - rhob)/rho (mathUtilities.cuh:12-19) of plane k over
    // columns xb-1..xb+32 and rows yb-1..yb+W, colour-gradient neighbour rule applied.  mz: the plane
    // the rule maps k to; plane_in_box: it is the staged plane.
    // The elements that are no node of the lattice in this tile (the frame: rows yb-1 and yb+W, columns
    // xb-1 and xb+32, and column nx and row ny where the lattice ends inside the tile) are warp 0's: it
    // has no destination rows, so it fills them for plane k+2 while the others finish plane k.  Two lists
    // in one table: from the front the elements whose value the staged box holds (ring position, box
    // index), from the back those it does not, the periodic images two layers out (ring position), each
    // with the node's (x, y) offset in global memory.  The far ones are copied to shared memory by
    // cp.async while the plane is computed.
    int2* ftab = reinterpret_cast<int2*>(smem + G::off_ftab);
    int* fcount = reinterpret_cast<int*>(ftab + G::frame);
    uint2* fbuf = reinterpret_cast<uint2*>(smem + G::off_fbuf);
    const int col_n = nx - (xb - 1), row_n = ny - (yb - 1); // ring column / row of nx / ny
    const bool has_col = col_n <= kPSX - 2, has_row = row_n <= W;
    const int nframe = 2 * kPSX + 2 * W + (has_col ? W + 2 : 0) + (has_row ? kPSX : 0);
    auto build_frame = [&]() {
        constexpr int kSkip = kTMA ? 32 : 0; // (warp 0 starts the copies)
        for (int e = tid - kSkip; e < nframe; e += kThreads - kSkip) {
            int r, c, i = e;
            if (i < 2 * kPSX) {
                r = i < kPSX ? 0 : W + 1;
                c = i < kPSX ? i : i - kPSX;
            } else if ((i -= 2 * kPSX) < 2 * W) {
                r = 1 + (i >> 1);
                c = (i & 1) ? kPSX - 1 : 0;
            } else if ((i -= 2 * W) < W + 2 && has_col) {
                r = i;
                c = col_n;
            } else {
                r = row_n;
                c = has_col ? i - (W + 2) : i;
            }
            const int gx = xb - 1 + c, gy = yb - 1 + r;
            // beyond the ghost frame and its one-node halo: read only by the colour gradient of
            // sources outside the lattice, whose populations reach no destination of the tile
            if (gx < -1 || gx > nx || gy < -1 || gy > ny) continue;
            const int mx = psi_coord(P, 0, gx, nx), my = psi_coord(P, 1, gy, ny);
            const bool px = P.bc[0] == MBCG_BC_PERIODIC, py = P.bc[1] == MBCG_BC_PERIODIC;
            const int dx = (px && gx >= 0 && gx <= nx - 1) ? gx : mx;
            const int dy = (py && gy >= 0 && gy <= ny - 1) ? gy : my;
            const int bc_ = dx - xr0, br_ = dy - (yb - 1);
            // (the plain copies stage the source nodes only)
            const bool box = kTMA && bc_ >= 0 && bc_ < kRBX && br_ >= 0 && br_ < G::RBY;
            const int off = static_cast<int>(static_cast<long long>(my) * P.pitch + mx); // a plane is below 2^31 elements
            const int at = atomicAdd(&fcount[box ? 0 : 1], 1);
            ftab[box ? at : G::frame - 1 - at] = make_int2(((box ? br_ * kRBX + bc_ : 0) << 16) | (r * kPSX + c), off);
        }
    };
    // The 4-byte word of global memory that holds element o of field f of plane mz, and the element in it.
    auto far_word = [&](int f, int mz, int o) -> uintptr_t {
        return reinterpret_cast<uintptr_t>(static_cast<const S*>(P.a[f]) + static_cast<long long>(mz) * P.plane + o);
    };
    auto far_value = [&](unsigned word, uintptr_t at) -> S {
        if constexpr (sizeof(S) == 4) {
            return __uint_as_float(word);
        } else {
            const unsigned short h = static_cast<unsigned short>((at & 2) ? word >> 16 : word & 0xffffU);
            return *reinterpret_cast<const S*>(&h);
        }
    };
    auto fetch_far = [&](int mz) { // warp 0
        for (int e = lane; e < fcount[1]; e += 32) {
            const int o = ftab[G::frame - 1 - e].y;
            cp_async4(&fbuf[e].x, reinterpret_cast<const void*>(far_word(0, mz, o) & ~uintptr_t(3)));
            cp_async4(&fbuf[e].y, reinterpret_cast<const void*>(far_word(1, mz, o) & ~uintptr_t(3)));
        }
    };
    constexpr int kFramePer = (G::frame + 31) / 32;
    auto fill_frame = [&](int mz, bool plane_in_box, int sl) { // warp 0, after fetch_far(mz)
        float* ring = psi_ring + sl * G::psi_plane;
        unsigned char* st = stage_at(sl);
        const int near = fcount[0], far = fcount[1];
        if (plane_in_box) {
#pragma unroll
            for (int i = 0; i < kFramePer; ++i) {
                const int e = lane + 32 * i;
                if (e < near) {
                    const int t = ftab[e].x;
                    ring[t & 0xffff] = psi_of<S>(P, rb_box(st, 0)[t >> 16], rb_box(st, 1)[t >> 16]);
                }
            }
        } else { // a few planes at the ends of a non-periodic z axis
            for (int e = lane; e < near; e += 32) {
                const int2 t = ftab[e];
                const long long o = static_cast<long long>(mz) * P.plane + t.y;
                ring[t.x & 0xffff] = psi_of<S>(P, static_cast<const S*>(P.a[0])[o], static_cast<const S*>(P.a[1])[o]);
            }
        }
        cp_async_wait_all(); // this lane's words
        for (int e = lane; e < far; e += 32) {
            const int2 t = ftab[G::frame - 1 - e];
            const uint2 v = fbuf[e];
            ring[t.x & 0xffff] = psi_of<S>(P, far_value(v.x, far_word(0, mz, t.y)), far_value(v.y, far_word(1, mz, t.y)));
        }
    };
    // psi of this thread's nodes into the ring; c0, c1: the nodes' own stored slots (fields 0 and 1)
    const int rPa = (wa + 1) * kPSX + lane + 1, rPb = (wb + 1) * kPSX + lane + 1; // ring elements
    const bool lat_a = xs < nx && ysa < ny, lat_b = xs < nx && ysb < ny; // nodes of the lattice
    auto fill_own = [&](auto mapped, int mz, bool plane_in_box, int sl, F2 c0, F2 c1) {
        float* ring = psi_ring + sl * G::psi_plane;
        if constexpr (decltype(mapped)::value) {
            S a0, a1, b0, b1;
            if (plane_in_box) {
                unsigned char* st = stage_at(sl);
                a0 = rb_box(st, 0)[bPa];
                a1 = rb_box(st, 1)[bPa];
                b0 = rb_box(st, 0)[bPb];
                b1 = rb_box(st, 1)[bPb];
            } else { // (nodes outside the lattice: any node serves, their psi is not stored)
                const long long x = min(pxo, nx - 1), z = static_cast<long long>(mz) * P.plane;
                const long long oa = z + min(pya, ny - 1) * P.pitch + x, ob = z + min(pyb, ny - 1) * P.pitch + x;
                a0 = static_cast<const S*>(P.a[0])[oa];
                a1 = static_cast<const S*>(P.a[1])[oa];
                b0 = static_cast<const S*>(P.a[0])[ob];
                b1 = static_cast<const S*>(P.a[1])[ob];
            }
            if (lat_a) ring[rPa] = psi_of<S>(P, a0, a1);
            if (lat_b) ring[rPb] = psi_of<S>(P, b0, b1);
        } else {
            if (lat_a) ring[rPa] = psi_of_slots<S>(c0.x, c1.x);
            if (lat_b) ring[rPb] = psi_of_slots<S>(c0.y, c1.y);
        }
    };
    // fields 0 and 1 of this thread's nodes on a staged plane
    auto load_colours = [&](int sl, F2& c0, F2& c1) {
        unsigned char* st = stage_at(sl);
        c0 = make_float2(Codec<S>::to_f(rb_box(st, 0)[bRa]), Codec<S>::to_f(rb_box(st, 0)[bRb]));
        c1 = make_float2(Codec<S>::to_f(rb_box(st, 1)[bRa]), Codec<S>::to_f(rb_box(st, 1)[bRb]));
    };

    // ---- set-up ------------------------------------------------------------------
    // every thread is done with the previous tile's shared memory before it is refilled
    __syncthreads();
    if (tid < 2) fcount[tid] = 0;
    __syncthreads();
    // no state is read before the kernel that wrote it is complete
    if (!kTMA || w != 0) build_frame();
    wait_prior_grid();
    for (int k = kfirst; k < kfirst + kNSTAGE; ++k) issue(k, k - kfirst);
    if constexpr (!kTMA) {
        cp_async_wait_all();
        __syncthreads();
    }
    {
        // The first wait.  Testing only (wait_test_cycles > 0): it waits on the barrier nothing
        // completes, with that limit, so it runs out and the tile takes the bail path with all its
        // planes in flight.  (Folded into the one wait: a second wait-and-bail path at the tile
        // start once cost the batch kernel ~20 %.)
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
            bail(kfirst + kNSTAGE - 1);
            return false;
        }
    }
    {
        F2 c0, c1;
        const int m0 = psi_coord(P, 2, kfirst, nz), m1 = psi_coord(P, 2, kfirst + 1, nz);
        load_colours(0, c0, c1);
        fill_own(std::bool_constant<kMapXY>{}, m0, m0 == zload(kfirst), 0, c0, c1);
        load_colours(1, c0, c1);
        fill_own(std::bool_constant<kMapXY>{}, m1, m1 == zload(kfirst + 1), 1, c0, c1);
        if (w == 0) {
            for (int i = 0; i < 3; ++i) {
                const int m = psi_coord(P, 2, kfirst + i, nz);
                fetch_far(m);
                if (i < 2 || peek_slot(i)) fill_frame(m, m == zload(kfirst + i), i);
            }
        }
    }
    // Plane kfirst is a source of nothing: once every warp has its psi, which beside an x or y boundary comes
    // from a neighbour's node, its slot is free (plain copies: refilled by the first plane's step (2)).
    __syncthreads();
    if constexpr (kTMA)
        if (kfirst + kNSTAGE <= zd1 + 1) issue(kfirst + kNSTAGE, 0);

    // store addresses: bytes from the tile's first destination plane, advanced plane by plane
    const long long tile_base = static_cast<long long>(zd0) * P.plane * static_cast<int>(sizeof(S));
    const unsigned plane_bytes = static_cast<unsigned>(P.plane) * static_cast<unsigned>(sizeof(S));
    unsigned off_a = (static_cast<unsigned>(ysa) * static_cast<unsigned>(P.pitch) + static_cast<unsigned>(xs)) *
                           static_cast<unsigned>(sizeof(S));
    unsigned off_b = (static_cast<unsigned>(ysb) * static_cast<unsigned>(P.pitch) + static_cast<unsigned>(xs)) *
                           static_cast<unsigned>(sizeof(S));

    Acc2 accP, accC; // destination planes k-1 and k (accC: what plane k-1 sent with cz = +1)
    F2 jzP, yzP, zzP, xzP; // plane k-1's sums with cz, less what plane k sends it
    accP.zero();
    accC.zero();
    jzP = yzP = zzP = xzP = make_float2(0.0f, 0.0f);

    // inlet / outlet functors fused into the store of the first and last fluid layer: the ghost node
    // behind node (xs, ys, d), whose new moments are given
    auto boundary = [&](int ys, int bR, int bM, unsigned char* st, int d, float rr, float rb, float ux, float uy,
                        float uz, const float (&pi)[6]) {
        if (ia < 0 || !P.do_bc) return;
        const int pa = ia == 0 ? xs : (ia == 1 ? ys : d);
        if (pa != 1 && pa != (ia == 0 ? nx : (ia == 1 ? ny : nz)) - 2) return;
        const bool inlet = pa == 1;
        const int gx = ia == 0 ? (inlet ? 0 : nx - 1) : xs;
        const int gy = ia == 1 ? (inlet ? 0 : ny - 1) : ys;
        const int gz = ia == 2 ? (inlet ? 0 : nz - 1) : d;
        const long long og = static_cast<long long>(gz) * P.plane + static_cast<long long>(gy) * P.pitch + gx;
        float orr, orb, oux, ouy, ouz;
        if (inlet) {
            // jet/boundary_conditions.cuh:16-39 (+ seeded per-node noise)
            const int t0 = ia == 0 ? ys : xs;
            const int t1 = ia == 2 ? ys : d;
            const float du = static_cast<float>(t0) - P.jet_c0;
            const float dv = static_cast<float>(t1) - P.jet_c1;
            const float m = (du * du + dv * dv) <= (P.jet_radius * P.jet_radius) ? 1.0f : 0.0f;
            orr = P.jet_blue ? (1.0f - m) * P.rho_r0 : m * P.rho_r0;
            orb = P.jet_blue ? m * P.rho_b0 : (1.0f - m) * P.rho_b0;
            float gu[3] = {0.0f, 0.0f, 0.0f};
            if (m != 0.0f) {
                if (P.noise_amp != 0.0f) {
                    const unsigned long long node = static_cast<unsigned long long>(gx) +
                                                    static_cast<unsigned long long>(gy) * nx +
                                                    static_cast<unsigned long long>(gz) * nx * ny;
                    gu[0] = m * P.noise_amp * noise_xi(P.seed, step, node, 0);
                    gu[1] = m * P.noise_amp * noise_xi(P.seed, step, node, 1);
                    gu[2] = m * P.noise_amp * noise_xi(P.seed, step, node, 2);
                }
            }
            oux = gu[0] + (ia == 0 ? m * P.jet_velocity : 0.0f);
            ouy = gu[1] + (ia == 1 ? m * P.jet_velocity : 0.0f);
            ouz = gu[2] + (ia == 2 ? m * P.jet_velocity : 0.0f);
        } else if (P.outlet == MBCG_OUTLET_ZERO_GRADIENT) {
            orr = rr; orb = rb; oux = ux; ouy = uy; ouz = uz;
        } else {
            // convective outlet (jet/boundary_conditions.cuh:45-109), old ghost from A
            float ov[NF];
            if (ia == 2) {
                ov[0] = Codec<S>::to_f(rb_box(st, 0)[bR]);
                ov[1] = Codec<S>::to_f(rb_box(st, 1)[bR]);
#pragma unroll
                for (int f = 2; f < NF; ++f) ov[f] = Codec<S>::to_f(m_box(st, f)[bM]);
            } else {
                load_global<S>(P, og, ov);
            }
            Node<S> on{};
            decode<S>(P, ov, on);
            const float ua = ia == 0 ? ux : (ia == 1 ? uy : uz);
            const float uc = fminf(fmaxf(ua, 0.0f), 1.0f);
            if (on.rr + on.rb <= 1.0e-20f) {
                orr = rr; orb = rb; oux = ux; ouy = uy; ouz = uz;
            } else {
                orr = on.rr - uc * (on.rr - rr);
                orb = on.rb - uc * (on.rb - rb);
                oux = on.ux - uc * (on.ux - ux);
                ouy = on.uy - uc * (on.uy - uy);
                ouz = on.uz - uc * (on.uz - uz);
            }
        }
        const int gix = P.bc[0] == MBCG_BC_PERIODIC ? (gx == 1 ? nx - 1 : (gx == nx - 2 ? 0 : -1)) : -1;
        const int giy = P.bc[1] == MBCG_BC_PERIODIC ? (gy == 1 ? ny - 1 : (gy == ny - 2 ? 0 : -1)) : -1;
        finalize_store<S>(P, og * static_cast<int>(sizeof(S)), 0U, gx, gy, gz, orr, orb, oux, ouy, ouz, pi, gix, giy, key_base);
    };

    bool ok = true; // kNearBar: this warp's (one that gave up arrives no more, and those that need it give up in turn)
    int sl = 1; // slot of plane k (k starts at kfirst + 1)
    int k = zd0 - 1;
    for (; k <= zd1; ++k, sl = nxt(sl)) {
        const int sl_next = nxt(sl), sl_prev = prv(sl);
        // (1) psi of plane k+1.  A warp waits for the others' part only where it needs it: before a colour
        // gradient, and before it overwrites the exchange buffer.
        // Plane coordinates: every mapping (staging, colour-gradient rule, node role) is the
        // identity while planes k .. k+3 are fluid planes, which is almost every plane.
        const bool zid = k >= 1 && k + 3 <= nz - 2;
        int mz1 = k + 1, mz2 = k + 2, rz = R_FLUID;
        bool inbox1 = true, inbox2 = true;
        if (!zid) {
            mz1 = psi_coord(P, 2, k + 1, nz);
            inbox1 = mz1 == zload(k + 1);
            mz2 = psi_coord(P, 2, k + 2, nz);
            inbox2 = mz2 == zload(k + 2);
            rz = axis_role<kFeat>(P, 2, k, nz);
        }
        // a plane that never arrived leaves garbage in the ring; the tile ends at the next barrier
        ok = wait_slot(k + 1, sl_next);
        if constexpr (kNearBar)
            if (!(ok = __all_sync(kFull, ok))) break;
        F2 c0, c1; // stored slots 0 and 1 of this thread's nodes
        load_colours(sl_next, c0, c1);
        if (ok) fill_own(std::bool_constant<kMapXY>{}, mz1, inbox1, sl_next, c0, c1);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[kPlaneBar]);
        if (w == 0 && k + 2 <= zd1 + 1) fetch_far(mz2); // far psi elements of plane k+2, used in (4)
        // (2) plain copies: plane k+kNSTAGE-1 into the slot plane k-1 used, complete before the next
        // barrier (TMA: at the end of (4))
        if constexpr (!kTMA)
            if (k + kNSTAGE - 1 <= zd1 + 1) issue(k + kNSTAGE - 1, sl_prev);

        // (3) this thread's source nodes at plane k
        const int role_a = zid ? role_xy[0] : role_of(rya, rz), role_b = zid ? role_xy[1] : role_of(ryb, rz);
        // Sources outside the lattice (lanes / rows past the last ghost layer) only ever stream
        // into nodes that are not destinations of this tile, so without walls every source is
        // processed branch-free; wall ghost layers hold data and must not emit.
        const bool act_a = ((kFeat & F_WALL) == 0) || (role_a == R_FLUID || role_a == R_GHOST);
        const bool act_b = ((kFeat & F_WALL) == 0) || (role_b == R_FLUID || role_b == R_GHOST);

        unsigned char* st = stage_at(sl);
        Node2 nd;
        F2 vx, vy, vz; // velocity of the non-equilibrium part
        {
            float va[NF], vb[NF];
#pragma unroll
            for (int f = 2; f < NF; ++f) {
                va[f] = Codec<S>::to_f(m_box(st, f)[bMa]);
                vb[f] = Codec<S>::to_f(m_box(st, f)[bMb]);
            }
            load_colours(sl, c0, c1); // (again: kept from the plane before, they spill others)
            va[0] = c0.x;
            vb[0] = c0.y;
            va[1] = c1.x;
            vb[1] = c1.y;
            decode2<S>(P, va, vb, nd);
            vx = nd.ux;
            vy = nd.uy;
            vz = nd.uz;
            if constexpr ((kFeat & F_INOUT) != 0) {
                // a ghost source (lbm.cuh:85-89) takes Pi and its velocity from the first fluid node
                // behind it: plane 1 or nz-2 (still staged: the slot of plane nz-2 is not refilled in
                // the chunk that ends at nz-1), or the neighbouring column / row of the staged plane
                auto ghost = [&](int role, int ryh, int ysh, int bMh, float (&v)[NF]) {
                    if (role != R_GHOST) return;
                    const unsigned char* sf = st;
                    int b2 = bMh;
                    if (rz == R_GHOST) {
                        sf = stage_at(k == 0 ? sl_next : sl_prev);
                    } else {
                        const int dx = (rx == R_GHOST) ? (xs == 0 ? 1 : -1) : 0;
                        const int dy = (ryh == R_GHOST) ? (ysh == 0 ? 1 : -1) : 0;
                        b2 = bMh + dy * kMX + dx;
                    }
#pragma unroll
                    for (int f = 2; f < NF; ++f)
                        v[f] = Codec<S>::to_f(reinterpret_cast<const S*>(sf + 2 * G::rb_field + (f - 2) * G::m_field)[b2]);
                };
                if (role_a == R_GHOST || role_b == R_GHOST) {
                    ghost(role_a, rya, ysa, bMa, va);
                    ghost(role_b, ryb, ysb, bMb, vb);
                    Node2 fn;
                    decode2<S>(P, va, vb, fn);
                    vx = fn.ux;
                    vy = fn.uy;
                    vz = fn.uz;
                    nd.pxx = fn.pxx; nd.pxy = fn.pxy; nd.pyy = fn.pyy;
                    nd.pyz = fn.pyz; nd.pzz = fn.pzz; nd.pxz = fn.pxz;
                }
            }
        }
        if constexpr ((kFeat & F_WALL) != 0) {
            // a wall source emits nothing: the reference density of the second colour at rest
            auto rest = [&](bool act, float& rr, float& rb, float& a0, float& a1, float& a2, float& a3, float& a4,
                            float& a5, float& a6, float& a7, float& a8) {
                if (act) return;
                rr = 0.0f;
                rb = P.rho_ref;
                a0 = a1 = a2 = a3 = a4 = a5 = a6 = a7 = a8 = 0.0f;
            };
            rest(act_a, nd.rr.x, nd.rb.x, nd.ux.x, nd.uy.x, nd.uz.x, nd.pxx.x, nd.pxy.x, nd.pyy.x, nd.pyz.x, nd.pzz.x, nd.pxz.x);
            rest(act_b, nd.rr.y, nd.rb.y, nd.ux.y, nd.uy.y, nd.uz.y, nd.pxx.y, nd.pxy.y, nd.pyy.y, nd.pyz.y, nd.pzz.y, nd.pxz.y);
        }

        const F2 ref = pair(P.rho_ref);
        const F2 rho = nd.rr + nd.rb;
        const F2 inv = make_float2(fast_rcp(rho.x), fast_rcp(rho.y));
        // Colour fraction as a correctly rounded quotient (one residual correction): a product with
        // a rounded reciprocal is biased (aR rho - rr averages +2.5e-10 per mixed node), which would
        // move colour mass the same way every step.
        const F2 q0 = nd.rr * inv;
        const F2 aR = fma2(fma2(neg2(q0), rho, nd.rr), inv, q0);
        // Red populations are W (rr + aR sm) + Delta, sm the population's part without the density.
        // In a near-steady state every rounding repeats from step to step and moves red mass the same
        // way (1.3e-5 in 10^4 steps on the 64^3 D3Q19 bubble when rr was rounded once more on its
        // way), so rr travels in two parts: rho_ref times the colour fraction on a 2^-16 grid, whose
        // weighted sums are exact in FP32, and the small rest rl.  Likewise the density: rhod, what it
        // has over rho_ref, is the sum of both colours' rests.  In a pure phase the grid part is 0 or 1
        // and rl is 0 or rhod: the red sums are then 0 or the total's own bits.
        auto grid = [](F2 a) { return (a + pair(192.0f)) - pair(192.0f); };
        const F2 ec = grid(aR);
        const F2 rl = fma2(-P.rho_ref, ec, nd.rr);
        const F2 rhod = rl + fma2(P.rho_ref, ec, nd.rb - ref);
        const F2 ind = 4.0f * nd.rr * nd.rb * inv * inv; // lbm.cuh:181,187
        bool if_a = ind.x > 1.0e-4f, if_b = ind.y > 1.0e-4f;
        if constexpr ((kFeat & F_INOUT) != 0) {
            if_a = if_a && role_a == R_FLUID;
            if_b = if_b && role_b == R_FLUID;
        }
        // zero-filled staging outside the lattice: keep those (never written) sources off the
        // interface path in the 16-bit forms
        if constexpr (sizeof(S) != 4) {
            if_a = if_a && in_xy_a;
            if_b = if_b && in_xy_b;
        }
        const F2 o3 = [&]() {
            const float unit = sizeof(S) == 4 ? 1.0f : P.pi_scale; // of nd's Pi
            if constexpr ((kFeat & F_FORCE) != 0) {
                if (P.tau_var)
                    return unit * make_float2(3.0f * (1.0f - 1.0f / tau_eff_of(P, nd.rr.x, nd.rb.x)),
                                              3.0f * (1.0f - 1.0f / tau_eff_of(P, nd.rr.y, nd.rb.y)));
            }
            return pair(3.0f * P.oms * unit);
        }();
        F2 fgx = pair(0.0f), fgy = fgx, fgz = fgx; // acceleration at the source, mirrored frame
        if constexpr ((kFeat & F_FORCE) != 0) {
            fgx = make_float2(act_a ? P.g[0] : 0.0f, act_b ? P.g[0] : 0.0f);
            fgy = make_float2(act_a ? P.g[1] : 0.0f, act_b ? -P.g[1] : 0.0f);
            fgz = make_float2(act_a ? P.g[2] : 0.0f, act_b ? P.g[2] : 0.0f);
        }
        Coef cf;
        build_coef<kFeat & ~F_INOUT>(P, cf, nd, rho, nd.ux, nd.uy, nd.uz, o3, fgx, fgy, fgz);
        if constexpr ((kFeat & F_INOUT) != 0) {
            // ghost sources only: the same node as a fluid source keeps the same bits in any tile
            if (role_a == R_GHOST || role_b == R_GHOST) {
                Coef cg;
                build_coef<kFeat>(P, cg, nd, rho, vx, vy, vz, o3, fgx, fgy, fgz);
                auto sel = [&](F2& c, F2 g) {
                    if (role_a == R_GHOST) c.x = g.x;
                    if (role_b == R_GHOST) c.y = g.y;
                };
                sel(cf.p000, cg.p000); sel(cf.p100, cg.p100); sel(cf.p010, cg.p010); sel(cf.p001, cg.p001);
                sel(cf.exx, cg.exx); sel(cf.eyy, cg.eyy); sel(cf.ezz, cg.ezz);
                sel(cf.exy, cg.exy); sel(cf.exz, cg.exz); sel(cf.eyz, cg.eyz);
                sel(cf.kxxy, cg.kxxy); sel(cf.kxxz, cg.kxxz); sel(cf.kxyy, cg.kxyy); sel(cf.kxzz, cg.kxzz);
                sel(cf.kyyz, cg.kyyz); sel(cf.kyzz, cg.kyzz); sel(cf.kxyz, cg.kxyz);
            }
        }
        // rest-population correction in value units before the rest weight (64 of 216, or 12 of 36)
        F2 rc0 = pair(0.0f);
        if constexpr ((kFeat & F_FORCE) != 0) {
            if (P.ratio) {
                F2 K = fma2(P.kappa_r, nd.rr, P.kappa_b * nd.rb);
                if (!act_a) K.x = 0.0f;
                if (!act_b) K.y = 0.0f;
                cf.p000 = cf.p000 + K;
                rc0 = (kSepW ? -3.375f : -3.0f) * K;
            }
        }

        // Interface sources: Omega2 into the coefficients, and the recolouring vector dF = d F, of
        // which Delta_c = W d(|c|) (F . c), d(|c|) = d / |c| (collisionOperators.cuh:60-80).  Other
        // sources have F = 0, which changes none of their sums, so a warp may take either side.
        const bool any_iface = __any_sync(kFull, if_a || if_b);
        F2 dFx = pair(0.0f), dFy = dFx, dFz = dFx;
        if (any_iface) {
            ok = plane_wait() && ok;
            const float* rm = psi_ring + sl_prev * G::psi_plane;
            const float* r0p = psi_ring + sl * G::psi_plane;
            const float* rp = psi_ring + sl_next * G::psi_plane;
            // colour gradient (forces.cuh:20-60) from the psi ring, rows in the mirrored frame of
            // the second node: R[dy][dz] weighted row sums, D[dy][dz] row differences along x
            F2 R[3][3], D[3][3];
#pragma unroll
            for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
                for (int dy = -1; dy <= 1; ++dy) {
                    const float* ring = dz < 0 ? rm : (dz == 0 ? r0p : rp);
                    const float* pa = ring + (wa + 1 + dy) * kPSX + lane + 1;
                    const float* pb = ring + (wb + 1 - dy) * kPSX + lane + 1;
                    const int n = dy * dy + dz * dz;
                    F2& r = R[dy + 1][dz + 1];
                    F2& d = D[dy + 1][dz + 1];
                    if (Q == 27 || n < 2) {
                        const F2 l = make_float2(pa[-1], pb[-1]), h = make_float2(pa[1], pb[1]);
                        d = h - l;
                        if (n != 0) r = fma2(Q == 27 ? 4.0f : 2.0f, make_float2(pa[0], pb[0]), h + l);
                    } else {
                        r = make_float2(pa[0], pb[0]);
                    }
                }
            F2 Fx, Fy, Fz;
            const F2 de = (D[0][1] + D[2][1]) + (D[1][0] + D[1][2]);
            const F2 ry = R[2][1] - R[0][1], rz_ = R[1][2] - R[1][0];
            const F2 py = R[2][2] - R[0][0], pz = R[2][0] - R[0][2];
            if constexpr (Q == 27) {
                const F2 dc = (D[0][0] + D[2][2]) + (D[0][2] + D[2][0]);
                constexpr float s = 3.0f / 216.0f;
                Fx = s * fma2(16.0f, D[1][1], fma2(4.0f, de, dc));
                Fy = s * fma2(4.0f, ry, py + pz);
                Fz = s * fma2(4.0f, rz_, py - pz);
            } else {
                constexpr float s = 3.0f / 36.0f;
                Fx = s * fma2(2.0f, D[1][1], de);
                Fy = s * (ry + (py + pz));
                Fz = s * (rz_ + (py - pz));
            }
            if (!if_a) Fx.x = Fy.x = Fz.x = 0.0f;
            if (!if_b) Fx.y = Fy.y = Fz.y = 0.0f;
            const F2 F2s = fma2(Fz, Fz, fma2(Fy, Fy, Fx * Fx));
            F2 qf = pair(0.0f), hA = pair(0.0f), dco = pair(0.0f);
            const F2 mix = P.beta * (nd.rr * nd.rb) * inv * inv;
            auto amp = [&](float f2, float rr, float rb, float rho_, float mx, float& q, float& h, float& dc) {
                const float absF = sqrtf(f2);
                float Aeff = P.A; // A_calculation (forces.cuh:114-117) at the node's relaxation time
                if constexpr ((kFeat & F_FORCE) != 0)
                    if (P.tau_var) Aeff = P.s4 / tau_eff_of(P, rr, rb);
                // Omega2 (collisionOperators.cuh:16-25); below the cut-off only its isotropic part
                h = P.omega2_conservative ? 0.0f : 0.5f * Aeff * absF;
                if (absF > 1.0e-4f) {
                    const float ia_ = fast_rcp(absF);
                    q = 0.5f * Aeff * ia_;
                    h = q * f2; // so Omega2 sums to zero over the directions in floating point too
                    // recolouring: beta rr rb / (rho^2 |F|) * feq0, where the rest equilibrium of moving
                    // directions is w rho (w (rho + K) with a density ratio)
                    const float feq0 = ((kFeat & F_FORCE) && P.ratio) ? rho_ + rr * P.kappa_r + rb * P.kappa_b : rho_;
                    dc = mx * ia_ * feq0;
                }
            };
            if (if_a) amp(F2s.x, nd.rr.x, nd.rb.x, rho.x, mix.x, qf.x, hA.x, dco.x);
            if (if_b) amp(F2s.y, nd.rr.y, nd.rb.y, rho.y, mix.y, qf.y, hA.y, dco.y);
            const F2 qx = (2.0f / 3.0f) * qf * Fx, qy = (2.0f / 3.0f) * qf * Fy, qz = (2.0f / 3.0f) * qf * Fz;
            const F2 oxx = qx * Fx, oyy = qy * Fy, ozz = qz * Fz;
            cf.exx = cf.exx + oxx;
            cf.eyy = cf.eyy + oyy;
            cf.ezz = cf.ezz + ozz;
            cf.exy = fma2(qx, Fy, cf.exy);
            cf.exz = fma2(qx, Fz, cf.exz);
            cf.eyz = fma2(qy, Fz, cf.eyz);
            cf.p000 = cf.p000 - hA;
            // rest part -hA (B0 - w0) = +2/3 hA, in value units of the rest weight
            rc0 = fma2(kSepW ? 2.25f : 2.0f, hA, rc0);
            dFx = dco * Fx;
            dFy = dco * Fy;
            dFz = dco * Fz;
        }

        // wall bounce-back of this thread's own populations (destination = source, plane k)
        [[maybe_unused]] F2 wall[4]; // its part of jz, yz, zz, xz, less that of tot, jy, tot, jx
        if constexpr ((kFeat & F_WALL) != 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) wall[i] = pair(0.0f);
            auto reflect = [&](int half, int role, bool dest, int ysh) {
                const bool wx0 = P.bc[0] == MBCG_BC_WALL && xs == 1, wx1 = P.bc[0] == MBCG_BC_WALL && xs == nx - 2;
                const bool wy0 = P.bc[1] == MBCG_BC_WALL && ysh == 1, wy1 = P.bc[1] == MBCG_BC_WALL && ysh == ny - 2;
                const bool wz0 = P.bc[2] == MBCG_BC_WALL && k == 1, wz1 = P.bc[2] == MBCG_BC_WALL && k == nz - 2;
                if (!(role == R_FLUID && dest && (wx0 | wx1 | wy0 | wy1 | wz0 | wz1))) return;
                auto h = [&](F2 v) { return half ? v.y : v.x; };
                const float mir = half ? -1.0f : 1.0f; // y of the mirrored frame
                float sums[12];
#pragma unroll
                for (int i = 0; i < 12; ++i) sums[i] = 0.0f;
                for (int i = 0; i < 27; ++i) {
                    const int cxi = i % 3 - 1, cyi = (i / 3) % 3 - 1, czi = i / 9 - 1;
                    const int n = cxi * cxi + cyi * cyi + czi * czi;
                    if (n == 0 || (Q == 19 && n == 3)) continue;
                    const bool into = (wx0 && cxi < 0) || (wx1 && cxi > 0) || (wy0 && cyi < 0) || (wy1 && cyi > 0) ||
                                      (wz0 && czi < 0) || (wz1 && czi > 0);
                    if (!into) continue;
                    const float cx = static_cast<float>(cxi), cy = mir * static_cast<float>(cyi), cz = static_cast<float>(czi);
                    const float wt = kSepW ? (n == 1 ? 16.0f : (n == 2 ? 4.0f : 1.0f)) : (n == 1 ? 2.0f : 1.0f);
                    float sm = h(cf.p000) + cx * h(cf.p100) + cy * h(cf.p010) + cz * h(cf.p001);
                    sm += 1.5f * (cx * cx * h(cf.exx) + cy * cy * h(cf.eyy) + cz * cz * h(cf.ezz));
                    sm += 3.0f * (cx * cy * h(cf.exy) + cx * cz * h(cf.exz) + cy * cz * h(cf.eyz));
                    sm += 4.5f * (cx * cx * (cy * h(cf.kxxy) + cz * h(cf.kxxz)) + cy * cy * (cx * h(cf.kxyy) + cz * h(cf.kyyz)) +
                                  cz * cz * (cx * h(cf.kxzz) + cy * h(cf.kyzz)));
                    sm += 9.0f * (cx * cy * cz * h(cf.kxyz));
                    const float g = wt * (h(rhod) + sm);
                    const float dn = n == 1 ? 1.0f : (n == 2 ? 0.7071067811865475f : 0.5773502691896258f);
                    const float dl = wt * dn * (cx * h(dFx) + cy * h(dFy) + cz * h(dFz));
                    // it returns with the opposite velocity
                    sums[0] += g;
                    sums[1] += fmaf(wt, fmaf(h(aR), sm, h(rl)), dl);
                    sums[2] += wt * h(ec);
                    sums[3] -= cx * g;
                    sums[4] -= cy * g;
                    sums[5] -= cz * g;
                    sums[6] += cx * cx * g;
                    sums[7] += cx * cy * g;
                    sums[8] += cy * cy * g;
                    sums[9] += cy * cz * g;
                    sums[10] += cz * cz * g;
                    sums[11] += cx * cz * g;
                }
                F2* a[12] = {&accC.tot, &accC.red, &accC.E, &accC.jx, &accC.jy, &wall[0],
                             &accC.xx, &accC.xy, &accC.yy, &wall[1], &wall[2], &wall[3]};
                sums[5] -= sums[0];
                sums[9] -= sums[4];
                sums[10] -= sums[0];
                sums[11] -= sums[3];
#pragma unroll
                for (int i = 0; i < 12; ++i) {
                    if (half) a[i]->y += sums[i];
                    else a[i]->x += sums[i];
                }
            };
            reflect(0, role_a, dest_a, ysa);
            reflect(1, role_b, dest_b, ysb);
        }

        // ---- x streaming.  For each power (b, c) of (cy, cz) the source evaluates its polynomial at
        // cx = -1, 0, +1; the outer two cross to the neighbouring lanes and the destination column
        // forms the moments of order 0, 1, 2 in x (and the red sum) of that coefficient.
        const F2 aRl = shfl_up2(aR), aRr = shfl_down2(aR);
        const F2 s00 = fma2(1.5f, cf.exx, cf.p000);
        // P: sum over cx = +-1, D: difference; X and rP: order 0 (weights 4 and 1) of the total and of
        // red for D3Q27; for D3Q19 X = cx = 0 alone and rP, rC red like P and X.
        struct XM {
            F2 P, D, X, rP, rC;
        };
        const F2 aR4 = 4.0f * aR;
        auto moments_x = [&](F2 l, F2 r, F2 centre) -> XM {
            XM m;
            m.P = l + r;
            m.D = l - r;
            m.X = kSepW ? fma2(4.0f, centre, m.P) : centre;
            return m;
        };
        auto stream_x = [&](F2 plus, F2 centre, F2 minus) -> XM {
            const F2 l = shfl_up2(plus), r = shfl_down2(minus);
            XM m = moments_x(l, r, centre);
            m.rP = fma2(aRr, r, aRl * l);
            if constexpr (kSepW) m.rP = fma2(aR4, centre, m.rP);
            else m.rC = aR * centre;
            return m;
        };
        XM m00;
        {
            const F2 sp = s00 + cf.p100, sm = s00 - cf.p100;
            const F2 l = shfl_up2(rhod + sp), r = shfl_down2(rhod + sm);
            m00 = moments_x(l, r, rhod + cf.p000);
            const F2 lr = shfl_up2(fma2(aR, sp, rl)), rr = shfl_down2(fma2(aR, sm, rl));
            const F2 cr = fma2(aR, cf.p000, rl);
            m00.rP = lr + rr;
            if constexpr (kSepW) m00.rP = fma2(4.0f, cr, m00.rP);
            else m00.rC = cr;
        }
        const F2 b10 = fma2(4.5f, cf.kxxy, cf.p010), b01 = fma2(4.5f, cf.kxxz, cf.p001);
        XM m10 = stream_x(fma2(3.0f, cf.exy, b10), cf.p010, fma2(-3.0f, cf.exy, b10));
        XM m01 = stream_x(fma2(3.0f, cf.exz, b01), cf.p001, fma2(-3.0f, cf.exz, b01));
        // the remaining ones without their factors 3/2, 3/2, 3, 9/2, 9/2
        XM m20 = stream_x(fma2(3.0f, cf.kxyy, cf.eyy), cf.eyy, fma2(-3.0f, cf.kxyy, cf.eyy));
        XM m02 = stream_x(fma2(3.0f, cf.kxzz, cf.ezz), cf.ezz, fma2(-3.0f, cf.kxzz, cf.ezz));
        XM m11 = stream_x(fma2(3.0f, cf.kxyz, cf.eyz), cf.eyz, fma2(-3.0f, cf.kxyz, cf.eyz));
        XM m21 = stream_x(cf.kyyz, cf.kyyz, cf.kyyz);
        XM m12 = stream_x(cf.kyzz, cf.kyzz, cf.kyzz);
        const F2 eS = grid(aRl) + grid(aRr);
        F2 red22 = pair(0.0f); // red sum of cy^2 cz^2, without the factor 3/2
        if (any_iface) {
            // Delta is odd in c: as a polynomial in (cy, cz) its coefficients at cx = +-1 and 0 are
            // multiples of dF with d(1) = d, d(2) = d / sqrt 2, d(3) = d / sqrt 3
            constexpr float i2 = 0.7071067811865475f;
            [[maybe_unused]] constexpr float i3 = 0.5773502691896258f;
            const F2 gx = shfl_up2(dFx) - shfl_down2(dFx);
            const F2 gy = shfl_up2(dFy) + shfl_down2(dFy);
            const F2 gz = shfl_up2(dFz) + shfl_down2(dFz);
            m00.rP = m00.rP + gx;
            m10.rP = fma2(i2, gy, m10.rP);
            m01.rP = fma2(i2, gz, m01.rP);
            m20.rP = fma2((i2 - 1.0f) / 1.5f, gx, m20.rP);
            m02.rP = fma2((i2 - 1.0f) / 1.5f, gx, m02.rP);
            if constexpr (kSepW) {
                m10.rP = fma2(4.0f, dFy, m10.rP);
                m01.rP = fma2(4.0f, dFz, m01.rP);
                m12.rP = fma2(4.0f * (i2 - 1.0f) / 4.5f, dFy, m12.rP);
                m21.rP = fma2(4.0f * (i2 - 1.0f) / 4.5f, dFz, m21.rP);
                m12.rP = fma2((i3 - i2) / 4.5f, gy, m12.rP);
                m21.rP = fma2((i3 - i2) / 4.5f, gz, m21.rP);
                red22 = ((i3 - 2.0f * i2 + 1.0f) / 1.5f) * gx;
            } else {
                m10.rC = m10.rC + dFy;
                m01.rC = m01.rC + dFz;
                m12.rC = fma2((i2 - 1.0f) / 4.5f, dFy, m12.rC);
                m21.rC = fma2((i2 - 1.0f) / 4.5f, dFz, m21.rC);
            }
        }

        ok = plane_wait() && ok;

        // ---- y streaming.  What leaves a row for the next row inwards (cy' = +1 of the mirrored
        // frame) and outwards (cy' = -1) goes through shared memory; the row's own part waits in
        // registers.  Weights: D3Q27 216 w = product over the axes of (4 if c_a = 0 else 1), the 4s
        // applied when an axis is summed; D3Q19 36 w = 12, 2, 1 by |c|^2.
        // The innermost pair is its own outer neighbour with the halves exchanged: it also writes its
        // inward values, swapped, to the outward slot after the last warp's.
        constexpr int kX = (H + 1) * 32; // one quantity's slots
        float2* xw = xbuf + w * 32 + lane;
        const bool innermost = w == H - 1;
        constexpr int kDir = kSepW ? 12 : 8; // quantities each way
        auto put = [&](int q, F2 in, F2 out) {
            xw[q * kX] = in;
            xw[(kDir + q) * kX] = out;
            if (innermost) xw[(kDir + q) * kX + 32] = swap2(in);
        };
        auto put_both = [&](int q, F2 v) {
            xw[q * kX] = v;
            if (innermost) xw[q * kX + 32] = swap2(v);
        };
        // own part of the destination sums: [channel][power of cz] (D3Q27), or by class (D3Q19)
        F2 own[4][3], ownE0;
        if constexpr (kSepW) {
            auto rows = [&](int ch, F2 a00, F2 a10, F2 a01, F2 a20, F2 a02, F2 a11, F2 a21, F2 a12) {
                const F2 e0 = fma2(1.5f, a20, a00), e1 = fma2(4.5f, a21, a01);
                put(3 * ch, e0 + a10, e0 - a10);
                put(3 * ch + 1, fma2(3.0f, a11, e1), fma2(-3.0f, a11, e1));
                put(3 * ch + 2, fma2(3.0f, a12, a02), fma2(-3.0f, a12, a02));
                own[ch][0] = a00;
                own[ch][1] = a01;
                own[ch][2] = a02;
            };
            rows(0, m00.X, m10.X, m01.X, m20.X, m02.X, m11.X, m21.X, m12.X);
            rows(1, m00.D, m10.D, m01.D, m20.D, m02.D, m11.D, m21.D, m12.D);
            rows(2, m00.P, m10.P, m01.P, m20.P, m02.P, m11.P, m21.P, m12.P);
            rows(3, m00.rP, m10.rP, m01.rP, m20.rP, m02.rP + red22, m11.rP, m21.rP, m12.rP);
            own[3][2] = m02.rP;
            ownE0 = fma2(4.0f, ec, eS);
            put_both(24, ownE0);
        } else {
            // channels 0 (order 0), 1 (D), 2 (P), 3 (red); cz = 0 rows have |c|^2 - cx^2 = 1 beside,
            // cz = +-1 rows beside this one only the centre (C)
            auto axis = [&](int ch, F2 a00, F2 a10, F2 a20) { // cz = 0
                const F2 e0 = fma2(1.5f, a20, a00);
                put(ch, e0 + a10, e0 - a10);
            };
            auto corner = [&](int q, F2 c00, F2 c10, F2 c01, F2 c20, F2 c02, F2 c11, F2 c21, F2 c12) { // cz = +1, -1
                const F2 e0 = fma2(1.5f, c02, fma2(1.5f, c20, c00));
                const F2 oy = fma2(4.5f, c12, c10), oz = fma2(4.5f, c21, c01);
                const F2 a = e0 + oy, b = fma2(3.0f, c11, oz), a2 = e0 - oy, b2 = fma2(-3.0f, c11, oz);
                put(q, a + b, a2 + b2);
                put(q + 1, a - b, a2 - b2);
            };
            auto a1 = [&](const XM& m) { return fma2(2.0f, m.X, m.P); };
            auto r1 = [&](const XM& m) { return fma2(2.0f, m.rC, m.rP); };
            auto a0 = [&](const XM& m) { return fma2(12.0f, m.X, 2.0f * m.P); };
            auto r0 = [&](const XM& m) { return fma2(12.0f, m.rC, 2.0f * m.rP); };
            axis(0, a1(m00), a1(m10), a1(m20));
            axis(1, m00.D, m10.D, m20.D);
            axis(2, m00.P, m10.P, m20.P);
            axis(3, r1(m00), r1(m10), r1(m20));
            corner(4, m00.X, m10.X, m01.X, m20.X, m02.X, m11.X, m21.X, m12.X);
            corner(6, m00.rC, m10.rC, m01.rC, m20.rC, m02.rC, m11.rC, m21.rC, m12.rC);
            // own row: cz = 0 (weights 12, 2), then cz = +1 and -1 (weights 2, 1)
            auto zrow = [&](int ch, F2 b00, F2 b01, F2 b02) {
                const F2 e0 = fma2(1.5f, b02, b00);
                own[ch][1] = e0 + b01;
                own[ch][2] = e0 - b01;
            };
            own[0][0] = a0(m00);
            own[1][0] = 2.0f * m00.D;
            own[2][0] = 2.0f * m00.P;
            own[3][0] = r0(m00);
            zrow(0, a1(m00), a1(m01), a1(m02));
            zrow(1, m00.D, m01.D, m02.D);
            zrow(2, m00.P, m01.P, m02.P);
            zrow(3, r1(m00), r1(m01), r1(m02));
            ownE0 = fma2(2.0f, ec, eS); // |c|^2 - cx^2 = 1; the row itself is 2 eS + 12 e
            put_both(16, ownE0);
            put_both(17, ec);
        }
        if constexpr (!kTMA) cp_async_wait_all();
        if constexpr (kNearBar) {
            if (!(ok = __all_sync(kFull, ok))) break;
            __syncwarp();
            if (y_target >= 0) mbar_arrive(&bars[kYBar + y_target]);
            if (!(ok = __all_sync(kFull, y_wait()))) break;
        } else {
            if (!(ok = !__syncthreads_or(!ok))) break;
        }
        par ^= kNearBar ? (1u << kPlaneBar) | (1u << kYBit) : 1u << kPlaneBar;

        // (4) y sums, z streaming; warp 0 holds the two halo rows and receives nothing: it refills the
        // slot of plane k (whose fields everyone has read) and prepares the psi frame of plane k+2
        const int d = k - 1;
        if (w == 0) {
            if constexpr (kTMA) {
                // Nothing more to stage: the next step's CTAs may take the SMs that fall idle (from the start
                // of the kernel they took them in another order: D3Q19 RTI 61^2x243, 8 steps, 494 against 512 us).
                if (k + kNSTAGE <= zd1 + 1) issue(k + kNSTAGE, sl);
                else launch_dependents();
            }
            const int sl2 = nxt(sl_next);
            if (k + 2 <= zd1 + 1 && peek_slot(sl2)) fill_frame(mz2, inbox2, sl2);
        } else {
            // [moment][cz = -1, 0, +1], moments tot, jx, jy, xx, xy, yy, red
            F2 Z0[7], Zp[7], Zm[7], Ep, E0;
            auto in_ = [&](int q) { return xw[q * kX - 32]; };
            auto ou_ = [&](int q) { return xw[(kDir + q) * kX + 32]; };
            auto both = [&](int q) { return xw[q * kX - 32] + xw[q * kX + 32]; };
            if constexpr (kSepW) {
                // powers of cz -> cz = -1, 0, +1; the last coefficient carries the factor 3/2
                auto zexp = [&](int i, const F2 (&c)[3]) {
                    const F2 e = fma2(1.5f, c[2], c[0]);
                    Zp[i] = e + c[1];
                    Zm[i] = e - c[1];
                    Z0[i] = c[0];
                };
                F2 y0[3], y1[3], y2[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const F2 i = in_(c), o = ou_(c);
                    y2[c] = i + o;
                    y1[c] = i - o;
                    y0[c] = fma2(4.0f, own[0][c], y2[c]);
                }
                zexp(0, y0);
                zexp(2, y1);
                zexp(5, y2);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const F2 i = in_(3 + c), o = ou_(3 + c);
                    y1[c] = i - o;
                    y0[c] = fma2(4.0f, own[1][c], i + o);
                }
                zexp(1, y0);
                zexp(4, y1);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    y0[c] = fma2(4.0f, own[2][c], in_(6 + c) + ou_(6 + c));
                    y1[c] = fma2(4.0f, own[3][c], in_(9 + c) + ou_(9 + c));
                }
                zexp(3, y0);
                zexp(6, y1);
                Ep = fma2(4.0f, ownE0, both(24));
                E0 = Ep;
            } else {
                // cz = 0: quantities 0 order 0, 1 D, 2 P, 3 red
                {
                    const F2 i = in_(0), o = ou_(0), s0 = i + o;
                    Z0[0] = s0 + own[0][0];
                    Z0[2] = i - o;
                    Z0[5] = s0;
                }
                {
                    const F2 i = in_(1), o = ou_(1);
                    Z0[1] = (i + o) + own[1][0];
                    Z0[4] = i - o;
                }
                Z0[3] = (in_(2) + ou_(2)) + own[2][0];
                Z0[6] = (in_(3) + ou_(3)) + own[3][0];
                // cz = +1 (quantities 4, 6) and -1 (5, 7): the neighbours send their centres
                {
                    const F2 i = in_(4), o = ou_(4), sp = i + o;
                    Zp[0] = sp + own[0][1];
                    Zp[2] = i - o;
                    Zp[5] = sp;
                }
                {
                    const F2 i = in_(5), o = ou_(5), sm = i + o;
                    Zm[0] = sm + own[0][2];
                    Zm[2] = i - o;
                    Zm[5] = sm;
                }
                Zp[1] = own[1][1];
                Zm[1] = own[1][2];
                Zp[4] = Zm[4] = pair(0.0f);
                Zp[3] = own[2][1];
                Zm[3] = own[2][2];
                Zp[6] = (in_(6) + ou_(6)) + own[3][1];
                Zm[6] = (in_(7) + ou_(7)) + own[3][2];
                E0 = both(16) + fma2(12.0f, ec, 2.0f * eS);
                Ep = both(17) + ownE0;
            }
            // destination plane k-1 receives cz = -1, plane k cz = 0, plane k+1 cz = +1
            // (5) destination plane k-1 is complete: moments (lbm.cuh:239-261), store, boundary
            if (d >= zd0 && d < zd1) {
                accP.tot = accP.tot + Zm[0];
                accP.jx = accP.jx + Zm[1];
                accP.jy = accP.jy + Zm[2];
                accP.xx = accP.xx + Zm[3];
                accP.xy = accP.xy + Zm[4];
                accP.yy = accP.yy + Zm[5];
                accP.red = accP.red + Zm[6];
                accP.E = accP.E + Ep;
                const F2 jz = jzP - Zm[0], zz = zzP + Zm[0], xz = xzP - Zm[1], yz = yzP - Zm[2];
                constexpr float kS = kSepW ? 216.0f : 36.0f;
                constexpr float sc = 1.0f / kS;
                // correctly rounded mass quotients (no systematic bias), plain scaling for the rest
                auto quot = [&](F2 a) {
                    const F2 q = sc * a;
                    return fma2(sc, fma2(-kS, q, a), q);
                };
                const F2 dev = quot(accP.tot);
                const F2 rho_n = ref + dev;
                // each colour: the grid part's quotient and its remainder, then the small part, one
                // rounding at the density's own magnitude
                const F2 devR = quot(accP.red);
                auto colour = [&](F2 e, F2 low) {
                    const F2 q = quot(e);
                    return fma2(ref, q, fma2(pair(P.rho_ref * sc), fma2(-kS, q, e), low));
                };
                const F2 rr_n = colour(accP.E, devR);
                const F2 rb_n = colour(pair(kS) - accP.E, dev - devR);
                const F2 ir = make_float2(fast_rcp(rho_n.x), fast_rcp(rho_n.y));
                const F2 isc = sc * ir;
                const F2 iscy = make_float2(isc.x, -isc.y); // back from the mirrored frame
                const F2 scy = make_float2(sc, -sc);
                F2 u_x = accP.jx * isc, u_y = accP.jy * iscy, u_z = jz * isc;
                constexpr bool kF = (kFeat & F_FORCE) != 0;
                if (kF && P.forced) {
                    // u = (j + F/2) / rho with F = rho g
                    u_x = u_x + pair(0.5f * P.g[0]);
                    u_y = u_y + pair(0.5f * P.g[1]);
                    u_z = u_z + pair(0.5f * P.g[2]);
                }
                const F2 ctr = (-1.0f / 3.0f) * dev;
                const F2 rho_m = fma2(-1.0f, dev, pair(-P.rho_ref)); // -rho
                const F2 mx = rho_m * u_x, my = rho_m * u_y, mz = rho_m * u_z;
                F2 pi[6];
                pi[0] = fma2(mx, u_x, fma2(sc, accP.xx, ctr));
                pi[1] = fma2(mx, u_y, scy * accP.xy);
                pi[2] = fma2(my, u_y, fma2(sc, accP.yy, ctr));
                pi[3] = fma2(my, u_z, scy * yz);
                pi[4] = fma2(mz, u_z, fma2(sc, zz, ctr));
                pi[5] = fma2(mx, u_z, sc * xz);
                if (kF && P.forced) {
                    const float hx = -0.5f * P.g[0], hy = -0.5f * P.g[1], hz = -0.5f * P.g[2];
                    pi[0] = fma2(2.0f * hx, mx, pi[0]);
                    pi[1] = fma2(hy, mx, fma2(hx, my, pi[1]));
                    pi[2] = fma2(2.0f * hy, my, pi[2]);
                    pi[3] = fma2(hz, my, fma2(hy, mz, pi[3]));
                    pi[4] = fma2(2.0f * hz, mz, pi[4]);
                    pi[5] = fma2(hz, mx, fma2(hx, mz, pi[5]));
                }
                if (kF && P.ratio) {
                    const F2 Kc = (-1.0f / 3.0f) * fma2(P.kappa_r, rr_n, P.kappa_b * rb_n);
                    pi[0] = pi[0] + Kc;
                    pi[2] = pi[2] + Kc;
                    pi[4] = pi[4] + Kc;
                }
                const float pa[6] = {pi[0].x, pi[1].x, pi[2].x, pi[3].x, pi[4].x, pi[5].x};
                const float pb[6] = {pi[0].y, pi[1].y, pi[2].y, pi[3].y, pi[4].y, pi[5].y};
                S oa[NF], ob[NF];
                {
                    const F2 u[3] = {u_x, u_y, u_z};
                    const unsigned ka = sizeof(S) == 4 ? 0U : node_round_key(P, key_base, xs, ysa, d);
                    const unsigned kb = sizeof(S) == 4 ? 0U : node_round_key(P, key_base, xs, ysb, d);
                    encode2<S>(P, rr_n, rb_n, ir, u, pi, oa, ob, ka, kb);
                }
                if constexpr (kStride) {
                    unsigned char* base_a = static_cast<unsigned char*>(P.b[0]) + tile_base + off_a;
                    unsigned char* base_b = static_cast<unsigned char*>(P.b[0]) + tile_base + off_b;
#pragma unroll
                    for (int f = 0; f < NF; ++f, base_a += P.b_stride, base_b += P.b_stride) {
                        if (dest_a) *reinterpret_cast<S*>(base_a) = oa[f];
                        if (dest_b) *reinterpret_cast<S*>(base_b) = ob[f];
                    }
                } else {
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        unsigned char* base = static_cast<unsigned char*>(P.b[f]) + tile_base;
                        if (dest_a) *reinterpret_cast<S*>(base + off_a) = oa[f];
                        if (dest_b) *reinterpret_cast<S*>(base + off_b) = ob[f];
                    }
                }
                if (images) { // the faces of a periodic x / y axis only
                    const int ix = image_of(0, xs, nx);
                    if (dest_a) store_images<S>(P, tile_base, off_a, xs, ysa, oa, ix, image_of(1, ysa, ny));
                    if (dest_b) store_images<S>(P, tile_base, off_b, xs, ysb, ob, ix, image_of(1, ysb, ny));
                }
                if constexpr ((kFeat & F_INOUT) != 0) {
                    if (dest_a) boundary(ysa, bRa, bMa, st, d, rr_n.x, rb_n.x, u_x.x, u_y.x, u_z.x, pa);
                    if (dest_b) boundary(ysb, bRb, bMb, st, d, rr_n.y, rb_n.y, u_x.y, u_y.y, u_z.y, pb);
                }
                off_a += plane_bytes;
                off_b += plane_bytes;
            }
            jzP = zzP = accC.tot;
            yzP = accC.jy;
            xzP = accC.jx;
            if constexpr ((kFeat & F_WALL) != 0) {
                jzP = jzP + wall[0];
                yzP = yzP + wall[1];
                zzP = zzP + wall[2];
                xzP = xzP + wall[3];
            }
            auto addz = [](F2 a, F2 b) { return kSepW ? fma2(4.0f, b, a) : a + b; };
            accP.tot = fma2(kSepW ? 64.0f : 12.0f, rc0, addz(accC.tot, Z0[0]));
            accP.red = fma2(kSepW ? 64.0f : 12.0f, aR * rc0, addz(accC.red, Z0[6]));
            accP.E = addz(accC.E, E0);
            accP.jx = addz(accC.jx, Z0[1]);
            accP.jy = addz(accC.jy, Z0[2]);
            accP.xx = addz(accC.xx, Z0[3]);
            accP.xy = addz(accC.xy, Z0[4]);
            accP.yy = addz(accC.yy, Z0[5]);
            accC.tot = Zp[0];
            accC.jx = Zp[1];
            accC.jy = Zp[2];
            accC.xx = Zp[3];
            accC.xy = Zp[4];
            accC.yy = Zp[5];
            accC.red = Zp[6];
            accC.E = Ep;
        }
    }
    if constexpr (kNearBar) ok = !__syncthreads_or(!ok);
    if (!ok) {
        bail(min(zd1 + 1, k - 1 + kNSTAGE)); // (what warp 0 had issued)
        return false;
    }
    // every load of this tile was waited for: carry the parities over to the next tile
    phase = par;
    return true;
}

// Whether a tile stays clear of the non-periodic axis: every node it reads is then a fluid node of that
// axis (or a periodic image), and it needs none of the inlet/outlet or wall parts.  Both kinds of tile
// do the same arithmetic on a fluid source, so which one a node falls into does not show in its bits.
template <int W>
__device__ __forceinline__ bool tile_is_interior(const StepParams& P, int bx, int by, int bz) {
    int zd0, zd1;
    z_range(P.nz, P.bc[2], P.zchunk, bz, zd0, zd1);
    const int xb = kTX * bx, yb = (W - 2) * by;
    const bool x = P.bc[0] == MBCG_BC_PERIODIC || (xb - 1 >= 1 && xb + 32 <= P.nx - 2);
    const bool y = P.bc[1] == MBCG_BC_PERIODIC || (yb - 1 >= 1 && yb + W <= P.ny - 2);
    const bool z = P.bc[2] == MBCG_BC_PERIODIC || (zd0 - 2 >= 1 && zd1 + 1 <= P.nz - 2);
    return x && y && z;
}

// ------------------------------------------------------------------ plain step kernel
// One tile per CTA over the grid ((nx-2)/30, (ny-2)/(W-2), z_tiles), rounded up.
template <int Q, typename S, int W, bool kTMA, int kFeat>
__global__ void __launch_bounds__(16 * W, W <= 8 ? 2 : 1) step_kernel(const __grid_constant__ StepParams P,
                                                                      const __grid_constant__ TensorMaps T) {
    unsigned char* smem = aligned_smem_base();
    init_barriers<W / 2>(smem);
    uint32_t phase = 0;
    if constexpr ((kFeat & (F_WALL | F_INOUT)) != 0) {
        if (tile_is_interior<W>(P, blockIdx.x, blockIdx.y, blockIdx.z)) {
            step_tile<Q, S, W, kTMA, kFeat & ~(F_WALL | F_INOUT)>(P, T.m, blockIdx.x, blockIdx.y, blockIdx.z, P.step, smem,
                                                                  phase);
            return;
        }
    }
    step_tile<Q, S, W, kTMA, kFeat>(P, T.m, blockIdx.x, blockIdx.y, blockIdx.z, P.step, smem, phase);
}

// Opt a kernel into its dynamic shared memory once per device; `done` is the kernel's own
// per-device bit set.
template <typename K>
cudaError_t configure_once(K kern, int smem, std::atomic<unsigned long long>& done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_acq_rel);
    return e;
}

// Launch as a programmatic dependent of the kernel before it in the stream: that one's last CTAs, the launch
// itself and this kernel's set-up overlap.  Every CTA waits for the prior grid before it touches a state, so
// a grid is complete only when all before it are.  Measured a step: 32^3 18.8 -> 16.1 us, 64^3 D3Q19 24.7 ->
// 22.9 us, 128^3 jet 114 -> 111 us, 192^3 247 -> 245 us.  (The batch kernels gain nothing: their launches
// run side by side, and a CTA that waits holds an SM another kind could use, 3.5 -> 3.7 ms for 8 requests.)
template <typename... Par, typename... Arg>
cudaError_t launch_pdl(void (*kern)(Par...), dim3 grid, dim3 block, int smem, cudaStream_t s, const Arg&... arg) {
    cudaLaunchAttribute pdl{};
    pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &pdl;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, arg...);
}

template <int Q, typename S, int W, bool kTMA, int kFeat>
cudaError_t launch_one(const StepParams& P, const TensorMaps& T, cudaStream_t s) {
    using G = Geo<S, W>;
    auto kern = step_kernel<Q, S, W, kTMA, kFeat>;
    static std::atomic<unsigned long long> configured{0};
    if (cudaError_t e = configure_once(kern, G::smem, configured)) return e;
    StepParams L = P;
    L.zchunk = std::min(L.zchunk, max_zchunk(L.plane, static_cast<int>(sizeof(S))));
    dim3 block(32, W / 2, 1);
    dim3 grid((L.nx - 2 + kTX - 1) / kTX, (L.ny - 2 + W - 3) / (W - 2), z_tiles(L.nz, L.bc[2], L.zchunk));
    return launch_pdl(kern, grid, block, G::smem, s, L, T);
}

// Feature set: the smallest instantiation covering the lattice (TMA path); the plain-load
// path, for layouts TMA cannot describe, carries every feature.
template <int Q, typename S, int W>
cudaError_t launch_w(bool tma, const StepParams& P, const TensorMaps& T, cudaStream_t s) {
    if (!tma) return launch_one<Q, S, W, false, F_ALL>(P, T, s);
    if (std::getenv("MBCG_ALL_FEATURES")) return launch_one<Q, S, W, true, F_ALL>(P, T, s); // (parity tests)
    const int f = features_of(P);
    if constexpr (sizeof(S) == 4) // (for what the 16-bit forms step by populations, see uses_pop)
        if (f == 0) return launch_one<Q, S, W, true, 0>(P, T, s);
    if (f == F_INOUT) return launch_one<Q, S, W, true, F_INOUT>(P, T, s);
    if constexpr (!std::is_same<S, __nv_bfloat16>::value)
        if ((f & F_INOUT) == 0) return launch_one<Q, S, W, true, F_WALL | F_FORCE>(P, T, s); // walls, force
    return launch_one<Q, S, W, true, F_ALL>(P, T, s);
}

template <int Q, typename S>
cudaError_t launch_qs(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s) {
    if (w == kStepWSmall) return launch_w<Q, S, step_rows(kStepWSmall)>(tma, P, T, s);
    return launch_w<Q, S, step_rows(kStepW)>(tma, P, T, s);
}

} // namespace

} // namespace mbcg
