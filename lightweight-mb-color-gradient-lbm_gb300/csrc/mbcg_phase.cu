// mbcg_phase.cu -- in-situ phase statistics of a case's current state (declared in
// include/mbcg.h, mbcg_phase_statistics): phase volumes, diffuse-interface area, interface node
// count, jet penetration and centroid as deterministic FP64 reductions, and optionally the
// connected regions of the tracked phase (droplets) by a lock-free union-find over the fluid
// nodes.  No counterpart in the reference, which declares a jet-breakup statistics sampler
// (constants.cuh:11,53) but never implements it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "mbcg_internal.h"

using namespace mbcg;

namespace {

int fail(int code, const std::string& msg) {
    set_last_error(msg);
    return code;
}

constexpr int kSlots = 8; // tracked volume, other volume, area, interface nodes, centroid x/y/z, penetration (max)
constexpr int kBlock = 256;
constexpr int kLoopCap = 1 << 22; // union-find iterations before a loop gives up

struct PhaseArgs {
    StepParams P;
    int sign;    // +1: red tracked, -1: blue tracked
    int ia;      // inlet/outlet axis, -1 if none
    int nf[3];   // fluid nodes per axis
    int* labels; // per fluid node, or null
    int* status;
};

// the two stored slots that hold a node's colour
template <typename S>
struct Raw {
    S s0, s1;
};
template <typename S>
__device__ __forceinline__ Raw<S> raw_at(const StepParams& P, long long o) {
    return {static_cast<const S*>(P.a[0])[o], static_cast<const S*>(P.a[1])[o]};
}
template <typename S>
__device__ __forceinline__ float phi_of(const StepParams& P, const Raw<S>& r) {
    float rr, rb;
    if constexpr (sizeof(S) == 4) {
        rr = r.s0;
        rb = r.s1;
    } else {
        const float c = Codec<S>::to_f(r.s1);
        const float rho = P.rho_mean + phi_of_slot(c) * P.rho_half_diff + P.rho_scale * Codec<S>::to_f(r.s0);
        colour_split(c, rho, rr, rb);
    }
    return (rr - rb) / (rr + rb);
}

// neighbour coordinate along an axis: periodic axes wrap over the fluid nodes 1..n-2, the others
// stay inside them (one-sided difference at the first and last fluid layer)
__device__ __forceinline__ int nb_coord(const StepParams& P, int a, int c, int n) {
    if (P.bc[a] == MBCG_BC_PERIODIC) return periodic_image(c, n);
    return min(max(c, 1), n - 2);
}

// Tiles of 32 x 8 columns marched along z.  Each node's phi is formed once (its division and the
// stencil's loads were made seven times a node before) and shared: along z in registers, in the plane
// through shared memory, with the tile's edge columns added by its first threads.  Volumes, interface
// nodes, centroid and penetration are whole numbers, counted as such; the area's terms are formed in FP32
// pairs and summed in FP64 (GB300 has two FP64 lanes per SM and clock: with FP64 roots at the nodes where
// phi varies, 223 us).  192x192x512 FP32: 3,100 us before.  The area is within 6e-16 of the exact sum of the terms
// of the FP32 phi (drops 24^3 to 150^3, RTI, jet, 16-bit forms; 3e-15 with FP64 terms), and as far as before, 2e-10
// to 7e-8, from that of phi in 64 bits.
constexpr int kTileX = 32, kTileY = 8;

template <typename S>
__global__ void __launch_bounds__(kBlock) phase_sums_kernel(const PhaseArgs A, int depth, long long tiles, double* partials) {
    const StepParams& P = A.P;
    __shared__ float ph[2][kTileY + 2][kTileX + 2];
    __shared__ double sh[kSlots][kBlock / 32];
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const int gx = (A.nf[0] + kTileX - 1) / kTileX, gy = (A.nf[1] + kTileY - 1) / kTileY;
    long long vol[2] = {0, 0}, mixed = 0, cen[3] = {0, 0, 0};
    int pen = -1;
    double area = 0.0;
    PairSum grad{0.0f, 0.0f}; // terms of the area not yet in it
    int held = 0;
    // the tile's edge column this thread adds (the first 2 x 32 + 2 x 8 threads)
    int ex = -1, ey = -1;
    if (tid < 32) { ex = tid; ey = -1; }
    else if (tid < 64) { ex = tid - 32; ey = kTileY; }
    else if (tid < 64 + kTileY) { ex = -1; ey = tid - 64; }
    else if (tid < 64 + 2 * kTileY) { ex = kTileX; ey = tid - 64 - kTileY; }
    const bool edge = tid < 64 + 2 * kTileY;
    int buf = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int x0 = 1 + kTileX * static_cast<int>(t % gx), y0 = 1 + kTileY * static_cast<int>((t / gx) % gy);
        const int z0 = 1 + depth * static_cast<int>(t / (static_cast<long long>(gx) * gy));
        const int z1 = min(z0 + depth, P.nz - 1);
        const int x = x0 + tx, y = y0 + ty;
        const bool inside = x <= P.nx - 2 && y <= P.ny - 2;
        // columns past the last fluid layer hold its neighbour under the boundary rule
        const int mx = nb_coord(P, 0, min(x, P.nx - 1), P.nx), my = nb_coord(P, 1, min(y, P.ny - 1), P.ny);
        const int hx = nb_coord(P, 0, min(x0 + ex, P.nx - 1), P.nx), hy = nb_coord(P, 1, min(y0 + ey, P.ny - 1), P.ny);
        const long long own = static_cast<long long>(my) * P.pitch + mx, far = static_cast<long long>(hy) * P.pitch + hx;
        auto raw_z = [&](long long col, int z) {
            return raw_at<S>(P, static_cast<long long>(nb_coord(P, 2, z, P.nz)) * P.plane + col);
        };
        float below = phi_of(P, raw_z(own, z0 - 1)), here = phi_of(P, raw_z(own, z0)), above = phi_of(P, raw_z(own, z0 + 1));
        float rim = edge ? phi_of(P, raw_z(far, z0)) : 0.0f;
        const int c[2] = {x, y}, n[2] = {P.nx, P.ny};
        for (int z = z0; z < z1; ++z, buf ^= 1) {
            ph[buf][ty + 1][tx + 1] = here;
            if (edge) ph[buf][ey + 1][ex + 1] = rim;
            // the next planes' loads are in flight while this one is summed
            Raw<S> next{}, next_rim{};
            if (z + 1 < z1) {
                next = raw_z(own, z + 2);
                if (edge) next_rim = raw_z(far, z + 1);
            }
            __syncthreads(); // (the other buffer is rewritten only after the next one)
            if (inside) {
                const float phi = here;
                const bool tracked = A.sign * phi > 0.0f;
                vol[tracked ? 0 : 1] += 1;
                if (1.0f - phi * phi > 1.0e-4f) mixed += 1; // 4 rho_r rho_b / rho^2 = 1 - phi^2 (lbm.cuh:181)
                const float lo[3] = {ph[buf][ty + 1][tx], ph[buf][ty][tx + 1], below};
                const float hi[3] = {ph[buf][ty + 1][tx + 2], ph[buf][ty + 2][tx + 1], above};
                if (lo[0] != hi[0] || lo[1] != hi[1] || lo[2] != hi[2]) {
                    // |grad phi|^2 = G + g in FP32 pairs (differences and squares with their rounding errors)
                    PairSum q;
                    q.hi = q.lo = 0.0f;
                    for (int a = 0; a < 3; ++a) {
                        // central difference; one-sided next to a boundary that is not periodic
                        const int p = a == 2 ? z : c[a], e = a == 2 ? P.nz : n[a];
                        const int span = P.bc[a] == MBCG_BC_PERIODIC ? 2 : min(p + 1, e - 2) - max(p - 1, 1);
                        if (span <= 0) continue;
                        const float f = span == 2 ? 0.5f : 1.0f, h = f * hi[a], l = f * lo[a];
                        const float d = h - l, zb = d - h;
                        const float de = (h - (d - zb)) - (l + zb); // h - l = d + de
                        const float s2 = d * d;
                        q.add(s2, fmaf(d, d, -s2) + 2.0f * d * de);
                    }
                    if (q.hi > 1.0e-28f) {
                        // sqrt(G + g) = s + (G + g - s^2) / (2 s), s = sqrt(G): 2^-46
                        const float s = sqrtf(q.hi);
                        grad.add(0.5f * s, 0.25f * (fmaf(-s, s, q.hi) + q.lo) / s);
                        if (++held == 16) {
                            grad.flush(area);
                            held = 0;
                        }
                    } else {
                        area += 0.5 * sqrt(static_cast<double>(q.hi) + q.lo);
                    }
                }
                if (tracked) {
                    cen[0] += x;
                    cen[1] += y;
                    cen[2] += z;
                    if (A.ia >= 0) pen = max(pen, A.ia == 0 ? x : (A.ia == 1 ? y : z));
                }
                if (A.labels) {
                    const long long e = (x - 1) + static_cast<long long>(A.nf[0]) * ((y - 1) + static_cast<long long>(A.nf[1]) * (z - 1));
                    A.labels[e] = tracked ? static_cast<int>(e) : -1;
                }
            }
            below = here;
            here = above;
            if (z + 1 < z1) {
                above = phi_of(P, next);
                if (edge) rim = phi_of(P, next_rim);
            }
        }
    }
    grad.flush(area);
    const double acc[kSlots] = {static_cast<double>(vol[0]), static_cast<double>(vol[1]), area,
                                static_cast<double>(mixed),  static_cast<double>(cen[0]), static_cast<double>(cen[1]),
                                static_cast<double>(cen[2]), static_cast<double>(pen)};
    for (int s = 0; s < kSlots; ++s) {
        double v = acc[s];
        for (int o = 16; o > 0; o >>= 1) {
            const double w = __shfl_down_sync(0xffffffffu, v, o);
            v = s == 7 ? fmax(v, w) : v + w;
        }
        if (tx == 0) sh[s][ty] = v;
    }
    __syncthreads();
    if (tid < kSlots) {
        double v = sh[tid][0];
        for (int w = 1; w < kBlock / 32; ++w) v = tid == 7 ? fmax(v, sh[tid][w]) : v + sh[tid][w];
        partials[blockIdx.x * kSlots + tid] = v;
    }
}

// fixed-order sum of the block partials (deterministic), one warp per slot
__global__ void __launch_bounds__(32 * kSlots) phase_final_kernel(const double* partials, int nparts, double* result) {
    const int s = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double v = s == 7 ? -1.0 : 0.0;
#pragma unroll 16
    for (int b = lane; b < nparts; b += 32) {
        const double p = partials[b * kSlots + s];
        v = s == 7 ? fmax(v, p) : v + p;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double w = __shfl_down_sync(0xffffffffu, v, o);
        v = s == 7 ? fmax(v, w) : v + w;
    }
    if (lane == 0) result[s] = v;
}

// ---------------------------------------------------------------- connected regions
// Lock-free union-find (labels only ever decrease towards a root); every loop is capped and
// reports through the status word instead of spinning on.
__device__ __forceinline__ int find_root(int* L, int i, int* status) {
    for (int it = 0; it < kLoopCap; ++it) {
        const int p = L[i];
        if (p == i) return i;
        const int gp = L[p];
        if (gp != p) L[i] = gp; // path halving (benign race: any value on the path is valid)
        i = gp;
    }
    atomicOr(status, 4);
    return i;
}

__device__ __forceinline__ void unite(int* L, int a, int b, int* status) {
    for (int it = 0; it < kLoopCap; ++it) {
        a = find_root(L, a, status);
        b = find_root(L, b, status);
        if (a == b) return;
        if (a > b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicCAS(&L[b], b, a); // link the larger root under the smaller
        if (old == b) return;
        b = old;
    }
    atomicOr(status, 4);
}

__global__ void merge_kernel(const PhaseArgs A) {
    const long long total = static_cast<long long>(A.nf[0]) * A.nf[1] * A.nf[2];
    for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < total;
         e += static_cast<long long>(gridDim.x) * blockDim.x) {
        if (A.labels[e] < 0) continue;
        int c[3] = {static_cast<int>(e % A.nf[0]), static_cast<int>((e / A.nf[0]) % A.nf[1]),
                    static_cast<int>(e / (static_cast<long long>(A.nf[0]) * A.nf[1]))};
        for (int a = 0; a < 3; ++a) {
            int d[3] = {c[0], c[1], c[2]};
            d[a] += 1;
            if (d[a] == A.nf[a]) {
                if (A.P.bc[a] != MBCG_BC_PERIODIC) continue;
                d[a] = 0;
            }
            const long long f = d[0] + static_cast<long long>(A.nf[0]) * (d[1] + static_cast<long long>(A.nf[1]) * d[2]);
            if (f != e && A.labels[f] >= 0) unite(A.labels, static_cast<int>(e), static_cast<int>(f), A.status);
        }
    }
}

// Region sizes.  Most lanes of a warp share a root: one atomic per distinct root and warp (one per node
// on the few roots took 174 us for 1.2 M tracked nodes of 192x192x512).  Every lane of a warp goes through
// the loop as often as the others and takes part in the match, with a root of -1 where it has no node.
__global__ void region_kernel(const PhaseArgs A, int* volume, unsigned char* touches) {
    const long long total = static_cast<long long>(A.nf[0]) * A.nf[1] * A.nf[2];
    const int lane = threadIdx.x & 31;
    for (long long e0 = blockIdx.x * static_cast<long long>(blockDim.x) + (threadIdx.x - lane); e0 < total;
         e0 += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long e = e0 + lane;
        int r = -1;
        if (e < total && A.labels[e] >= 0) r = find_root(A.labels, static_cast<int>(e), A.status);
        if (!__any_sync(0xffffffffu, r >= 0)) continue;
        const unsigned peers = __match_any_sync(0xffffffffu, r);
        if (r < 0) continue;
        if (lane == __ffs(peers) - 1) atomicAdd(&volume[r], __popc(peers));
        if (A.ia >= 0) {
            const int c[3] = {static_cast<int>(e % A.nf[0]), static_cast<int>((e / A.nf[0]) % A.nf[1]),
                              static_cast<int>(e / (static_cast<long long>(A.nf[0]) * A.nf[1]))};
            if (c[A.ia] == 0) touches[r] = 1;
        }
    }
}

// per root: count, largest, detached count and volume (integer atomics: order-independent)
__global__ void region_stats_kernel(const PhaseArgs A, const int* volume, const unsigned char* touches,
                                    unsigned long long* out) {
    const long long total = static_cast<long long>(A.nf[0]) * A.nf[1] * A.nf[2];
    for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < total;
         e += static_cast<long long>(gridDim.x) * blockDim.x) {
        if (A.labels[e] != static_cast<int>(e)) continue; // roots only
        const unsigned long long v = static_cast<unsigned long long>(volume[e]);
        atomicAdd(&out[0], 1ULL);
        atomicMax(&out[1], v);
        if (!touches[e]) {
            atomicAdd(&out[2], 1ULL);
            atomicAdd(&out[3], v);
        }
    }
}

template <typename S>
cudaError_t sums(const PhaseArgs& A, int depth, long long tiles, double* partials, int nparts, double* result,
                 cudaStream_t s) {
    phase_sums_kernel<S><<<nparts, kBlock, 0, s>>>(A, depth, tiles, partials);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    phase_final_kernel<<<1, 32 * kSlots, 0, s>>>(partials, nparts, result);
    return cudaGetLastError();
}

int phase_statistics(const mbcg_params& p, const StepParams& P, int32_t flags, mbcg_phase_stats* out, mbcg_stream_t s) {
    PhaseArgs A;
    std::memset(&A, 0, sizeof(A));
    A.P = P;
    A.ia = A.P.inout_axis;
    A.sign = (A.ia >= 0 && p.ic == MBCG_IC_JET && p.jet_phase < 0.0) ? -1 : 1;
    A.nf[0] = p.nx - 2;
    A.nf[1] = p.ny - 2;
    A.nf[2] = p.nz - 2;
    const long long nodes = static_cast<long long>(A.nf[0]) * A.nf[1] * A.nf[2];
    const bool comps = (flags & MBCG_STATS_COMPONENTS) != 0;
    if (comps && nodes >= (1LL << 31)) return fail(MBCG_E_UNSUPPORTED, "region labels need fewer than 2^31 fluid nodes");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(s);
    // z depth of the tiles: about eight tiles per block slot (152 SMs x 8 blocks), 8 to 64 planes (a tile
    // loads two planes more than it sums)
    const long long columns = static_cast<long long>((A.nf[0] + kTileX - 1) / kTileX) * ((A.nf[1] + kTileY - 1) / kTileY);
    const int depth = static_cast<int>(std::min<long long>(64, std::max<long long>(8, columns * A.nf[2] / (8 * 1216))));
    const long long tiles = columns * ((A.nf[2] + depth - 1) / depth);
    const int nparts = static_cast<int>(std::min<long long>(tiles, 1216));
    // one scratch allocation: partials; results, region counters and status (copied back together); labels
    const size_t small = sizeof(double) * (kSlots * (nparts + 1)) + 4 * sizeof(unsigned long long) + 64;
    const size_t big = comps ? static_cast<size_t>(nodes) * (2 * sizeof(int) + 1) : 0;
    unsigned char* scratch = nullptr;
    cudaError_t e = cudaMalloc(&scratch, small + big + 256);
    if (e != cudaSuccess) return fail(MBCG_E_NOMEM, "phase statistics scratch allocation failed");
    double* partials = reinterpret_cast<double*>(scratch);
    double* result = partials + kSlots * nparts;
    unsigned long long* counters = reinterpret_cast<unsigned long long*>(result + kSlots);
    int* status = reinterpret_cast<int*>(counters + 4);
    int* labels = nullptr;
    int* volume = nullptr;
    unsigned char* touches = nullptr;
    if (comps) {
        unsigned char* b = scratch + ((small + 255) / 256) * 256;
        labels = reinterpret_cast<int*>(b);
        volume = labels + nodes;
        touches = reinterpret_cast<unsigned char*>(volume + nodes);
    }
    A.labels = labels;
    A.status = status;
    e = cudaMemsetAsync(scratch, 0, small + big + 256, st);
    if (e == cudaSuccess) {
        switch (p.precision) {
        case MBCG_FP16: e = sums<__half>(A, depth, tiles, partials, nparts, result, st); break;
        case MBCG_BF16: e = sums<__nv_bfloat16>(A, depth, tiles, partials, nparts, result, st); break;
        default: e = sums<float>(A, depth, tiles, partials, nparts, result, st); break;
        }
    }
    const int grid = static_cast<int>(std::min<long long>((nodes + kBlock - 1) / kBlock, 4 * 1184));
    if (comps && e == cudaSuccess) {
        merge_kernel<<<grid, kBlock, 0, st>>>(A);
        e = cudaGetLastError();
        if (e == cudaSuccess) {
            region_kernel<<<grid, kBlock, 0, st>>>(A, volume, touches);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) {
            region_stats_kernel<<<grid, kBlock, 0, st>>>(A, volume, touches, counters);
            e = cudaGetLastError();
        }
    }
    struct {
        double r[kSlots];
        unsigned long long cnt[4];
        int stat;
    } back{};
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&back, result, sizeof(back.r) + sizeof(back.cnt) + sizeof(int), cudaMemcpyDeviceToHost, st);
    const auto& r = back.r;
    const auto& cnt = back.cnt;
    const int stat = back.stat;
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(scratch);
    if (e != cudaSuccess) return fail(MBCG_E_CUDA, std::string("phase statistics: ") + cudaGetErrorString(e));
    std::memset(out, 0, sizeof(*out));
    out->volume_tracked = r[0];
    out->volume_other = r[1];
    out->interface_area = r[2];
    out->interface_nodes = static_cast<int64_t>(r[3]);
    for (int a = 0; a < 3; ++a) out->centroid[a] = r[0] > 0 ? r[4 + a] / r[0] : 0.0;
    out->penetration = A.ia >= 0 ? r[7] : -1.0; // fluid coordinate = distance from the inlet ghost layer
    out->components = comps ? static_cast<int64_t>(cnt[0]) : -1;
    out->largest_component = comps ? static_cast<int64_t>(cnt[1]) : -1;
    out->detached = comps ? static_cast<int64_t>(cnt[2]) : -1;
    out->detached_volume = comps ? static_cast<int64_t>(cnt[3]) : -1;
    out->status = stat;
    return MBCG_OK;
}

} // namespace

extern "C" {

int mbcg_phase_statistics(mbcg_case* c, int32_t flags, mbcg_phase_stats* out, mbcg_stream_t s) {
    if (!c || !out) return fail(MBCG_E_INVALID, "null argument");
    mbcg_params p;
    if (int rc = mbcg_case_params(c, &p)) return rc;
    StepParams P;
    if (int rc = case_state_params(c, &P)) return rc;
    return phase_statistics(p, P, flags, out, s);
}

int mbcg_phase_statistics_moments(const mbcg_params* p, const mbcg_moments* a, int32_t flags, mbcg_phase_stats* out,
                                  mbcg_stream_t s) {
    if (!p || !a || !out) return fail(MBCG_E_INVALID, "null argument");
    if (int rc = validate_params(p)) return rc;
    if (a->precision != p->precision || a->pitch < p->nx) return fail(MBCG_E_INVALID, "moments do not match params");
    for (int i = 0; i < NF; ++i)
        if (!a->f[i]) return fail(MBCG_E_INVALID, "null field pointer");
    StepParams P;
    fill_step_physics(*p, P);
    P.pitch = a->pitch;
    P.plane = a->pitch * p->ny;
    for (int i = 0; i < NF; ++i) P.a[i] = a->f[i];
    return phase_statistics(*p, P, flags, out, s);
}

} // extern "C"
