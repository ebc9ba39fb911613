// Laden-particle kernels (sim/lp.py): grid-to-particle sampling with the
// quadratic B-spline MAC interpolant, the explicit particle update, the
// particle-to-grid drag scatter and the face-grid viscous Laplacian.
#include <cuda_runtime.h>

#include <algorithm>

#include "edge_common.cuh"

using namespace edge;

namespace {

inline int grid_for(long long n, int b = 256) { return (int)((n + b - 1) / b); }
inline int st(void) {
    cudaError_t e = cudaPeekAtLastError();
    return e == cudaSuccess ? EDGE_OK : (int)e;
}
inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// The samplers at points: nine blocks of 128 per SM (10^6 points at random in
// 128x256x128 131 us, at eight and ten 134 and 135; 200 000 of them 35, 38, 37)
constexpr int kPointBlock = 128;

// lp.py:6-29 update_particles_acc
template <bool P2>
__global__ void __launch_bounds__(kPointBlock, 9) k_lp_acc(Mac mac_, const float* __restrict__ vel,
                                                           const float* __restrict__ pos, float* acc, int num, int nmax,
                                                           float dt, float St, float gravity) {
    const Mac mac = with_pow2<P2>(mac_);
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nmax) return;
    float a[3] = {0.f, 0.f, 0.f};
    if (e < num) {
        float kk = 1.0f / St;
        float p[3] = {pos[3 * e], pos[3 * e + 1], pos[3 * e + 2]};
        float v[3];
        mac_sample_points(mac, p, lanes_below(e, num), v);
        a[1] += gravity;
        for (int c = 0; c < 3; c++) a[c] -= kk * (vel[3 * e + c] - v[c]);
        for (int c = 0; c < 3; c++) a[c] /= (1.0f + kk * dt);
    }
    for (int c = 0; c < 3; c++) acc[3 * e + c] = a[c];
}

// lp.py:32-70 update_particles_velocity
__global__ void k_lp_velocity(const float* __restrict__ acc, float* vel, const float* __restrict__ pos, float dt,
                              float dx, int num, float Lx, float Ly, float Lz) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= num) return;
    float v[3], p[3] = {pos[3 * e], pos[3 * e + 1], pos[3 * e + 2]};
    for (int c = 0; c < 3; c++) v[c] = vel[3 * e + c] + acc[3 * e + c] * dt;
    if (p[1] < dx && v[1] < 0) v[1] = 0.0f;
    if (p[1] > Ly - 3 * dx && v[1] > 0) v[1] = 0.0f;
    if (p[0] < 3 * dx && v[0] < 0) v[0] = 0.0f;
    if (p[0] > Lx - 3 * dx && v[0] > 0) v[0] = 0.0f;
    if (p[2] < 3 * dx && v[2] < 0) v[2] = 0.0f;
    if (p[2] > Lz - 3 * dx && v[2] > 0) v[2] = 0.0f;
    for (int c = 0; c < 3; c++) vel[3 * e + c] = v[c];
}

// lp.py:73-97 calculate_velocity_diff
template <bool P2>
__global__ void __launch_bounds__(kPointBlock, 9) k_lp_vel_diff(Mac mac_, const float* __restrict__ vel, float* vdiff,
                                                                const float* __restrict__ pos, int num, float kk) {
    const Mac mac = with_pow2<P2>(mac_);
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= num) return;
    float p[3] = {pos[3 * e], pos[3 * e + 1], pos[3 * e + 2]};
    float v[3];
    mac_sample_points(mac, p, lanes_below(e, num), v);
    for (int c = 0; c < 3; c++) vdiff[3 * e + c] = kk * (vel[3 * e + c] - v[c]);
}

// lp.py:100-156 laden_particles_back_with_computing_particle: quadratic
// B-spline scatter of the drag onto the three face grids (atomic adds, like
// the reference's `+=` in a parallel loop)
template <bool P2>
EDGE_D void scatter_particle(int e, int nx, int ny, int nz, float dx, float inv_dx, float* dx_, float* dy_, float* dz_,
                             const float* __restrict__ vdiff, const float* __restrict__ pos,
                             const float* __restrict__ rad, float lrad, float Lx, float Ly, float Lz) {
    float p[3] = {pos[3 * e], pos[3 * e + 1], pos[3 * e + 2]};
    if (p[0] < 3 * dx || p[1] < 3 * dx || p[2] < 3 * dx || p[0] > Lx - 3 * dx || p[1] > Ly - 3 * dx ||
        p[2] > Lz - 3 * dx)
        return;
    float g[3] = {over_dx(p[0], dx, inv_dx, P2), over_dx(p[1], dx, inv_dx, P2), over_dx(p[2], dx, inv_dx, P2)};
    float r = rad[e];
    float scale = r * r * r / (lrad * lrad * lrad);
    float* D[3] = {dx_, dy_, dz_};
    for (int a = 0; a < 3; a++) {
        float off[3];
        int base[3];
        for (int c = 0; c < 3; c++) {
            off[c] = (c == a) ? 0.0f : 0.5f;
            base[c] = (int)(g[c] - off[c]);
        }
        int n0 = nx + (a == 0), n1 = ny + (a == 1), n2 = nz + (a == 2);
        float val = vdiff[3 * e + a];
        // the four taps' weights of each axis, once (the loops below used to
        // re-evaluate N2 for every tap of the inner loops)
        float W[3][4];
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int o = 0; o < 4; o++) W[c][o] = N2(g[c] - (float)(base[c] + o - 1) - off[c]);
#pragma unroll
        for (int oi = -1; oi < 3; oi++) {
            int f0 = base[0] + oi;
            if (f0 < 0 || f0 >= n0) continue;
            float wx = W[0][oi + 1];
            if (wx == 0.0f) continue;
#pragma unroll
            for (int oj = -1; oj < 3; oj++) {
                int f1 = base[1] + oj;
                if (f1 < 0 || f1 >= n1) continue;
                float wy = W[1][oj + 1];
                if (wy == 0.0f) continue;
#pragma unroll
                for (int ok = -1; ok < 3; ok++) {
                    int f2 = base[2] + ok;
                    if (f2 < 0 || f2 >= n2) continue;
                    float w = wx * wy * W[2][ok + 1];
                    if (w == 0.0f) continue;
                    atomicAdd(D[a] + idx3(f0, f1, f2, n1, n2), val * w * scale);
                }
            }
        }
    }
}
template <bool P2>
__global__ void k_lp_p2g(int nx, int ny, int nz, float dx, float inv_dx, float* dx_, float* dy_, float* dz_,
                         const float* __restrict__ vdiff, const float* __restrict__ pos,
                         const float* __restrict__ rad, int num, float lrad, float Lx, float Ly, float Lz) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < num)
        scatter_particle<P2>(e, nx, ny, nz, dx, inv_dx, dx_, dy_, dz_, vdiff, pos, rad, lrad, Lx, Ly, Lz);
}

// ---------------------------------------------------------------------------
// The same scatter through particles grouped by cell.  k_lp_p2g adds every
// particle to 81 faces with one atomic each and runs at the rate of the L2's
// atomic units; where several particles share a cell their sums over its faces
// can be formed first.  A counting sort groups the particles (no order of the
// cells is needed: a cell's segment starts wherever the running total stands),
// then a warp walks over consecutive particles with the cell's faces in its
// lanes' registers and adds them to the grids when the cell changes.
//
// The faces a particle of cell floor(p / dx) can reach are, in each component's
// grid, four along the component's own axis and three along the other two
// (nodes c - 1 .. c + 2 and c - 1 .. c + 1); N2 is 0 where it does not.  Lane
// 9 a + 3 u + v < 27 holds the four faces of component a at node u of the next
// axis and v of the one after.  Million-particle drop of 20 per cell, 128x256x128
// cells: 746 us for the atomics of k_lp_p2g, 140 us so; 1.3 per cell: 642 and
// 302 us (27 lanes add to neighbouring faces at once).
// ---------------------------------------------------------------------------
struct P2G {
    int nx, ny, nz, num;
    float dx, inv_dx, lrad, L[3];
    const float *vdiff, *pos, *rad;
    int* cell;   // particles per cell, then the start of the cell's segment
    int* key;    // cell of a particle, -1 where it does not scatter
    int* rank;   // its place among the cell's particles
    int* order;  // the particles, grouped by cell
    int* total;  // [0] particles grouped, [1] whether they scatter directly instead
};

template <bool P2>
EDGE_D bool p2g_coord(const P2G& a, int e, float g[3]) {
    bool in = true;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float p = a.pos[3 * (long long)e + c];
        in = in && p >= 3 * a.dx && p <= a.L[c] - 3 * a.dx;  // a NaN position reaches no face
        g[c] = over_dx(p, a.dx, a.inv_dx, P2);
    }
    return in;
}

// Zeroes the drag and the counts, and looks whether grouping pays.  The direct
// scatter is bound by the sectors that a warp's atomics fall on and by particles
// that share a face.  In an order where they follow one another cell by cell (a
// lattice, a line) both are few and it is the faster one; so it is where none
// reaches a face.  16 warps of consecutive particles are looked at: their cells,
// and the sectors of their first staggered taps, which alternate between rows
// where the particles lie at random in sorted cells.  us, direct, grouped and
// so: 10^6 on a lattice in 192x96x96 138, 281, 142, in 128x256x128 178, 302, 188;
// 200 000 in 64^3 35, 69, 40; sorted by cell in 192x96x96 348, 233, 232; at
// random 541, 247, 245; 10^6 out of reach 12, 23, 18.
template <bool P2>
__global__ void __launch_bounds__(512) k_p2g_begin(P2G a, float* Dx, float* Dy, float* Dz) {
    if (blockIdx.x == 0) {
        const unsigned lane = threadIdx.x & 31, before = (1u << lane) - 1u;
        // multiples of the golden ratio: no lattice's period
        const unsigned at = (threadIdx.x >> 5) * 0x9e3779b9u;
        const int e = (int)((unsigned long long)at * (unsigned)max(a.num - 31, 1) >> 32) + (int)lane;
        float g[3];
        const bool in = e < a.num && p2g_coord<P2>(a, e, g);
        const unsigned mask = __ballot_sync(0xffffffffu, in);
        bool direct = false;
        if (in) {
            const int cell = idx3((int)g[0], (int)g[1], (int)g[2], a.ny, a.nz),
                      face = idx3((int)(g[0] - 0.5f), (int)(g[1] - 0.5f), (int)(g[2] - 0.5f), a.ny, a.nz);
            const int all = __popc(mask), cells = __popc(__ballot_sync(mask, !(__match_any_sync(mask, cell) & before))),
                      sectors = __popc(__ballot_sync(mask, !(__match_any_sync(mask, face >> 3) & before)));
            direct = 8 * cells >= 5 * all && 8 * sectors <= 3 * all + 8;
        }
        const int reach = __syncthreads_count(in), yes = __syncthreads_count(direct);
        if (threadIdx.x == 0) {
            a.total[0] = 0;
            a.total[1] = 2 * yes >= reach;
        }
    }
    const int n = a.nx * a.ny * a.nz;
    const long long fx = n + (long long)a.ny * a.nz, fy = n + (long long)a.nx * a.nz, fz = n + (long long)a.nx * a.ny,
                    step = (long long)gridDim.x * blockDim.x;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < fx || t < fy || t < fz; t += step) {
        if (t < fx) Dx[t] = 0.0f;
        if (t < fy) Dy[t] = 0.0f;
        if (t < fz) Dz[t] = 0.0f;
        if (t < n) a.cell[t] = 0;
    }
}

template <bool P2>
__global__ void __launch_bounds__(256) k_p2g_count(P2G a, float* Dx, float* Dy, float* Dz) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.num) return;
    if (a.total[1]) {
        scatter_particle<P2>(e, a.nx, a.ny, a.nz, a.dx, a.inv_dx, Dx, Dy, Dz, a.vdiff, a.pos, a.rad, a.lrad, a.L[0],
                             a.L[1], a.L[2]);
        return;
    }
    float g[3];
    int key = -1;
    if (p2g_coord<P2>(a, e, g)) {
        const int i = (int)g[0], j = (int)g[1], k = (int)g[2];
        // a particle past the grid (a domain larger than it) reaches the faces
        // its clamped cell does or none; k_p2g_sum tests every face's range
        key = idx3(clampi(i, 0, a.nx - 1), clampi(j, 0, a.ny - 1), clampi(k, 0, a.nz - 1), a.ny, a.nz);
        a.rank[e] = atomicAdd(a.cell + key, 1);
    }
    a.key[e] = key;
}

// counts to segment starts; one atomic on the running total per block
__global__ void __launch_bounds__(256) k_p2g_start(int n, int* cell, int* total) {
    if (total[1]) return;
    __shared__ int warp_sum[8], base;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int e0 = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    int c[4], s = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        c[q] = e0 + q < n ? cell[e0 + q] : 0;
        s += c[q];
    }
    int incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int q = 0; q < 8; q++) {
            const int v = warp_sum[q];
            warp_sum[q] = t;
            t += v;
        }
        base = t ? atomicAdd(total, t) : 0;
    }
    __syncthreads();
    int at = base + warp_sum[w] + incl - s;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (e0 + q < n && c[q]) cell[e0 + q] = at;
        at += c[q];
    }
}

__global__ void __launch_bounds__(256) k_p2g_place(P2G a) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.num || a.total[1]) return;
    const int k = a.key[e];
    if (k >= 0) a.order[a.cell[k] + a.rank[e]] = e;
}

constexpr int kSumWarps = 4;
template <bool P2>
__global__ void __launch_bounds__(32 * kSumWarps) k_p2g_sum(P2G a, float* Dx, float* Dy, float* Dz, int batches) {
    // per particle of a batch: three axes' four own-axis weights, three axes'
    // three other-axis weights, three values
    __shared__ float4 own[kSumWarps][32][3];
    __shared__ float side[kSumWarps][32][13];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int total = a.total[0];
    const int first = (blockIdx.x * kSumWarps + w) * batches * 32;
    if (first >= total) return;
    const int last = min(total, first + batches * 32);
    // this lane's faces
    const int c = lane / 9, u = lane % 9 / 3, v = lane % 3;
    const bool holds = lane < 27;
    const int b1 = c == 0 ? 1 : 0, b2 = c == 2 ? 1 : 2;  // the other axes, in order
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    int cur = -1;
    auto flush = [&]() {
        if (cur < 0 || !holds) return;
        const int k = cur % a.nz, j = cur / a.nz % a.ny, i = cur / (a.ny * a.nz);
        const int n1 = a.ny + (c == 1), n2 = a.nz + (c == 2);
        float* D = c == 0 ? Dx : (c == 1 ? Dy : Dz);
#pragma unroll
        for (int o = 0; o < 4; o++) {
            const int f0 = i - 1 + (c == 0 ? o : u), f1 = j - 1 + (c == 1 ? o : (c == 0 ? u : v)),
                      f2 = k - 1 + (c == 2 ? o : v);
            if (acc[o] != 0.0f && f0 >= 0 && f1 >= 0 && f2 >= 0 && f0 < a.nx + (c == 0) && f1 < n1 && f2 < n2)
                atomicAdd(D + idx3(f0, f1, f2, n1, n2), acc[o]);
            acc[o] = 0.0f;
        }
    };
    for (int at = first; at < last; at += 32) {
        const int m = min(32, last - at);
        int key = -1;
        __syncwarp();
        if (lane < m) {
            const int e = a.order[at + lane];
            key = a.key[e];
            float g[3];
            p2g_coord<P2>(a, e, g);
            const float r = a.rad[e];
            const float scale = r * r * r / (a.lrad * a.lrad * a.lrad);
            const int base[3] = {key / (a.ny * a.nz), key / a.nz % a.ny, key % a.nz};
#pragma unroll
            for (int d = 0; d < 3; d++) {
                float W[4];
#pragma unroll
                for (int o = 0; o < 4; o++) W[o] = N2(g[d] - (float)(base[d] + o - 1));
                own[w][lane][d] = make_float4(W[0], W[1], W[2], W[3]);
#pragma unroll
                for (int o = 0; o < 3; o++) side[w][lane][3 * d + o] = N2(g[d] - (float)(base[d] + o - 1) - 0.5f);
                side[w][lane][9 + d] = a.vdiff[3 * (long long)e + d] * scale;
            }
        }
        // a value that is not finite must not reach a face through a zero weight
        const bool finite = __all_sync(0xffffffffu, lane >= m || (isfinite(side[w][lane][9]) && isfinite(side[w][lane][10]) &&
                                                                  isfinite(side[w][lane][11])));
        __syncwarp();
        for (int q = 0; q < m; q++) {
            const int kq = __shfl_sync(0xffffffffu, key, q);
            if (kq != cur) {
                flush();
                cur = kq;
            }
            if (holds) {
                const float4 W = own[w][q][c];
                const float wuv = side[w][q][3 * b1 + u] * side[w][q][3 * b2 + v], f = side[w][q][9 + c] * wuv;
                if (finite) {
                    acc[0] += f * W.x;
                    acc[1] += f * W.y;
                    acc[2] += f * W.z;
                    acc[3] += f * W.w;
                } else if (wuv != 0.0f) {
                    if (W.x != 0.0f) acc[0] += f * W.x;
                    if (W.y != 0.0f) acc[1] += f * W.y;
                    if (W.z != 0.0f) acc[2] += f * W.z;
                    if (W.w != 0.0f) acc[3] += f * W.w;
                }
            }
        }
    }
    flush();
}

// lp.py:158-181 update_particles_position
__global__ void k_lp_position(const float* __restrict__ vel, float* pos, float dt, int num, float Lx, float Ly,
                              float Lz) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= num) return;
    float L[3] = {Lx, Ly, Lz};
    for (int c = 0; c < 3; c++) {
        float p = pos[3 * e + c] + vel[3 * e + c] * dt;
        if (p < 0) p = 0.0f;
        if (p > L[c]) p = L[c];
        pos[3 * e + c] = p;
    }
}

// lp.py:183-219 calculate_viscous_force on the three face grids
template <bool P2>
__global__ void __launch_bounds__(256) k_lp_viscous(Star g, float dx, float inv_dx, float nu, Face3 u, float* vx,
                                                    float* vy, float* vz) {
    face_star(g, u, [&](int axis, int e, float at, float l, float r, float b, float t, float a, float c) {
        float* o = axis == 0 ? vx : (axis == 1 ? vy : vz);
        const float v = nu * (r + l + t + b + c + a + -6.0f * at);
        o[e] = over_dx(over_dx(v, dx, inv_dx, P2), dx, inv_dx, P2);
    });
}

// calc_max_particle_speed (run_edge.py:256-261): max |v| over the live
// particles, at least 1e-3 (bits of non-negative floats order as integers)
__global__ void k_lp_init_max(float* out) { *out = 1.0e-3f; }
__global__ void k_lp_max_speed(const float* __restrict__ vel, int num, float* out) {
    float best = 0.0f;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < num; e += gridDim.x * blockDim.x) {
        float a = vel[3 * e], b = vel[3 * e + 1], c = vel[3 * e + 2];
        best = fmaxf(best, sqrtf(a * a + b * b + c * c));
    }
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(out), __float_as_int(best));
}

}  // namespace

extern "C" {

int edge_lp_max_speed(const float* vel, int num, float* out, void* stream) {
    if (num < 0 || !out || (num && !vel)) return EDGE_EINVAL;
    k_lp_init_max<<<1, 1, 0, S(stream)>>>(out);
    if (num > 0) k_lp_max_speed<<<std::min(grid_for(num), 148 * 8), 256, 0, S(stream)>>>(vel, num, out);
    return st();
}

int edge_lp_acc(int nx, int ny, int nz, float dx, const float* ux, const float* uy, const float* uz, const float* vel,
                const float* pos, float* acc, int num, int nmax, float dt, float St, float gravity, void* stream) {
    if (nx < 4 || ny < 4 || nz < 4 || !ux || !uy || !uz || num < 0 || nmax < num || (nmax && (!vel || !pos || !acc)))
        return EDGE_EINVAL;
    if (nmax == 0) return EDGE_OK;
    const Mac mac = make_mac(ux, uy, uz, nx, ny, nz, dx);
    const int g = grid_for(nmax, kPointBlock);
    if (mac.pow2) k_lp_acc<true><<<g, kPointBlock, 0, S(stream)>>>(mac, vel, pos, acc, num, nmax, dt, St, gravity);
    else k_lp_acc<false><<<g, kPointBlock, 0, S(stream)>>>(mac, vel, pos, acc, num, nmax, dt, St, gravity);
    return st();
}

int edge_lp_velocity(const float* acc, float* vel, const float* pos, float dt, float dx, int num, float Lx, float Ly,
                     float Lz, void* stream) {
    if (num < 0 || (num && (!acc || !vel || !pos))) return EDGE_EINVAL;
    if (num == 0) return EDGE_OK;
    k_lp_velocity<<<grid_for(num), 256, 0, S(stream)>>>(acc, vel, pos, dt, dx, num, Lx, Ly, Lz);
    return st();
}

int edge_lp_vel_diff(int nx, int ny, int nz, float dx, const float* ux, const float* uy, const float* uz,
                     const float* vel, float* vdiff, const float* pos, int num, float St, float density_ratio,
                     float epiral_radius_ratio, void* stream) {
    if (nx < 4 || ny < 4 || nz < 4 || !ux || !uy || !uz || num < 0 || (num && (!vel || !vdiff || !pos)))
        return EDGE_EINVAL;
    if (num == 0) return EDGE_OK;
    float eratio = 1.0f / (epiral_radius_ratio * epiral_radius_ratio * epiral_radius_ratio);
    float kk = 1.0f / St * density_ratio * eratio;
    const Mac mac = make_mac(ux, uy, uz, nx, ny, nz, dx);
    const int g = grid_for(num, kPointBlock);
    if (mac.pow2) k_lp_vel_diff<true><<<g, kPointBlock, 0, S(stream)>>>(mac, vel, vdiff, pos, num, kk);
    else k_lp_vel_diff<false><<<g, kPointBlock, 0, S(stream)>>>(mac, vel, vdiff, pos, num, kk);
    return st();
}

int edge_lp_p2g(int nx, int ny, int nz, float dx, float* dragx, float* dragy, float* dragz, const float* vdiff,
                const float* pos, const float* rad, int num, float laden_radius, float Lx, float Ly, float Lz,
                void* stream) {
    if (nx < 1 || ny < 1 || nz < 1 || !dragx || !dragy || !dragz || num < 0 || (num && (!vdiff || !pos || !rad)))
        return EDGE_EINVAL;
    cudaStream_t s = S(stream);
    cudaError_t e;
    if ((e = cudaMemsetAsync(dragx, 0, (size_t)(nx + 1) * ny * nz * 4, s)) != cudaSuccess) return (int)e;
    if ((e = cudaMemsetAsync(dragy, 0, (size_t)nx * (ny + 1) * nz * 4, s)) != cudaSuccess) return (int)e;
    if ((e = cudaMemsetAsync(dragz, 0, (size_t)nx * ny * (nz + 1) * 4, s)) != cudaSuccess) return (int)e;
    if (num == 0) return EDGE_OK;
    // p / dx as the reference writes it: the exact multiply by 1/dx when dx is a power of two
    if (pow2f(dx))
        k_lp_p2g<true><<<grid_for(num), 256, 0, s>>>(nx, ny, nz, dx, 1.0f / dx, dragx, dragy, dragz, vdiff, pos, rad,
                                                     num, laden_radius, Lx, Ly, Lz);
    else
        k_lp_p2g<false><<<grid_for(num), 256, 0, s>>>(nx, ny, nz, dx, 1.0f / dx, dragx, dragy, dragz, vdiff, pos, rad,
                                                      num, laden_radius, Lx, Ly, Lz);
    return st();
}

// layout of the grouped scatter's workspace: ints, 256-byte aligned parts
static long long p2g_part(long long ints) { return (ints * 4 + 255) / 256 * 256; }

int edge_lp_p2g_workspace(int nx, int ny, int nz, int num, long long* bytes) {
    if (nx < 1 || ny < 1 || nz < 1 || num < 0 || !bytes) return EDGE_EINVAL;
    const long long n = (long long)nx * ny * nz;
    if (n >= (1LL << 31)) return EDGE_EINVAL;
    *bytes = p2g_part(n + 2) + 3 * p2g_part(num);
    return EDGE_OK;
}

int edge_lp_p2g_grouped(int nx, int ny, int nz, float dx, float* dragx, float* dragy, float* dragz, const float* vdiff,
                        const float* pos, const float* rad, int num, float laden_radius, float Lx, float Ly, float Lz,
                        void* work, long long work_bytes, void* stream) {
    long long need = 0;
    if (edge_lp_p2g_workspace(nx, ny, nz, num, &need) != EDGE_OK) return EDGE_EINVAL;
    if (!dragx || !dragy || !dragz || (num && (!vdiff || !pos || !rad)) || !work || work_bytes < need) return EDGE_EINVAL;
    if ((uintptr_t)work & 15) return EDGE_EALIGN;
    cudaStream_t s = S(stream);
    if (num == 0)
        return edge_lp_p2g(nx, ny, nz, dx, dragx, dragy, dragz, vdiff, pos, rad, 0, laden_radius, Lx, Ly, Lz, stream);
    const int n = nx * ny * nz;
    char* w = (char*)work;
    P2G a;
    a.nx = nx; a.ny = ny; a.nz = nz; a.num = num;
    a.dx = dx; a.inv_dx = 1.0f / dx; a.lrad = laden_radius;
    a.L[0] = Lx; a.L[1] = Ly; a.L[2] = Lz;
    a.vdiff = vdiff; a.pos = pos; a.rad = rad;
    a.cell = (int*)w;
    a.total = a.cell + n;
    w += p2g_part(n + 2LL);
    a.key = (int*)w;
    w += p2g_part(num);
    a.rank = (int*)w;
    w += p2g_part(num);
    a.order = (int*)w;
    // a warp walks over more than one batch when that still leaves 32 warps per SM
    const int batches = (int)std::max(1LL, std::min(8LL, num / (32LL * 32 * 148)));
    const int warps = grid_for(num, 32 * batches);
    const bool p2 = pow2f(dx);
    const int zero = std::min(grid_for(n, 1024), 148 * 4);
    if (p2) k_p2g_begin<true><<<zero, 512, 0, s>>>(a, dragx, dragy, dragz);
    else k_p2g_begin<false><<<zero, 512, 0, s>>>(a, dragx, dragy, dragz);
    if (p2) k_p2g_count<true><<<grid_for(num), 256, 0, s>>>(a, dragx, dragy, dragz);
    else k_p2g_count<false><<<grid_for(num), 256, 0, s>>>(a, dragx, dragy, dragz);
    k_p2g_start<<<grid_for(n, 1024), 256, 0, s>>>(n, a.cell, a.total);
    k_p2g_place<<<grid_for(num), 256, 0, s>>>(a);
    if (p2) k_p2g_sum<true><<<grid_for(warps, kSumWarps), 32 * kSumWarps, 0, s>>>(a, dragx, dragy, dragz, batches);
    else k_p2g_sum<false><<<grid_for(warps, kSumWarps), 32 * kSumWarps, 0, s>>>(a, dragx, dragy, dragz, batches);
    return st();
}

int edge_lp_position(const float* vel, float* pos, float dt, int num, float Lx, float Ly, float Lz, void* stream) {
    if (num < 0 || (num && (!vel || !pos))) return EDGE_EINVAL;
    if (num == 0) return EDGE_OK;
    k_lp_position<<<grid_for(num), 256, 0, S(stream)>>>(vel, pos, dt, num, Lx, Ly, Lz);
    return st();
}

int edge_lp_viscous(int nx, int ny, int nz, float dx, float Re, const float* ux, const float* uy, const float* uz,
                    float* visx, float* visy, float* visz, void* stream) {
    if (nx < 1 || ny < 1 || nz < 1 || !ux || !uy || !uz || !visx || !visy || !visz) return EDGE_EINVAL;
    const Star g = make_star(nx, ny, nz);
    const Face3 u = {{ux, uy, uz}};
    const float inv = 1.0f / dx, nu = 1.0f / Re;
    if (pow2f(dx)) k_lp_viscous<true><<<star_grid(g, 256), 256, 0, S(stream)>>>(g, dx, inv, nu, u, visx, visy, visz);
    else k_lp_viscous<false><<<star_grid(g, 256), 256, 0, S(stream)>>>(g, dx, inv, nu, u, visx, visy, visz);
    return st();
}

}  // extern "C"
