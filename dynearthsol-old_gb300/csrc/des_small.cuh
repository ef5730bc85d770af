// Step kernels for small meshes, where the chip has more lanes than the mesh
// has elements or nodes and a step's time is the latency of one thread's
// work: eight lanes share a node, four an element.  Same arithmetic, in the
// same order, as des_kernels.cuh, des_elem.cuh and des_kernels32.cuh.  (One
// warp alone gets an FP64 instruction per 68 clocks and about one other per 4.)
// The FP64 step on 144 elements went from 55 to 31 us, on 9,600 from 65 to
// 37; the FP32 step on 27,702 from 47 to 33.  E-B in quads gained 1.4 us of
// 11.5 at 144 elements and lost 4 of 12.1 at 27k, and is not here.
#pragma once

#include "des_elem.cuh"
#include "des_kernels32.cuh"

namespace des {

constexpr int kSmallBlock = 128;

// ---- nodes: eight lanes each ------------------------------------------------------
// The lanes load a node's support entries and the values they point to side
// by side into shared memory, then lane r adds up array r in the list's order:
// three dependent memory latencies and one chain of additions, where one
// thread has a latency per batch of entries and five chains.
constexpr int kNodeLanes = 8, kNodeChunk = 32;

template <class R, int ARRAYS>
struct NodeTile {
    R v[kSmallBlock / kNodeLanes][ARRAYS][kNodeChunk];
};

// lane r's value of f over the node's entries of array r (r < ARRAYS):
// load(entry, v) fills the values of one entry.  All lanes of the warp call it.
template <class R, int ARRAYS, class Load, class F>
__device__ __forceinline__ void octet_walk(NodeTile<R, ARRAYS> &tile, const unsigned *ent, int q0, int q1, Load load,
                                           F f)
{
    const int l = threadIdx.x & (kNodeLanes - 1);
    R(*t)[kNodeChunk] = tile.v[threadIdx.x / kNodeLanes];
    for (int q = q0; __any_sync(0xffffffffu, q < q1); q += kNodeChunk) {
        unsigned p[kNodeChunk / kNodeLanes];
#pragma unroll
        for (int k = 0; k < kNodeChunk / kNodeLanes; ++k) {
            const int j = q + l + kNodeLanes * k;
            p[k] = j < q1 ? __ldg(ent + j) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kNodeChunk / kNodeLanes; ++k)
            if (q + l + kNodeLanes * k < q1) {
                R v[ARRAYS];
                load(p[k], v);
#pragma unroll
                for (int a = 0; a < ARRAYS; ++a) t[a][l + kNodeLanes * k] = v[a];
            }
        __syncwarp();
        if (l < ARRAYS) {
            const int n = min(q1 - q, kNodeChunk);
            for (int j = 0; j < n; ++j) f(t[l][j]);
        }
        __syncwarp();
    }
}

template <class R>
__device__ __forceinline__ R octet_get(R v, int lane)
{
    return __shfl_sync(0xffffffffu, v, lane, kNodeLanes);
}

// N-A (k_fn_a): lanes 0-2 the masses, 3 the temperature, 4 dvoldt
__global__ void __launch_bounds__(kSmallBlock) k_fn_a_small(Dev d)
{
    __shared__ NodeTile<double, 5> tile;
    const int n = (int)(blockIdx.x * kSmallBlock + threadIdx.x) / kNodeLanes, l = threadIdx.x & (kNodeLanes - 1);
    const Consts &K = *d.K;
    const bool live = n < d.nnode, thermal = K.thermal;
    const double dt = d.clk->dt;
    const bool stale = !d.clk->mass_valid;
    if (n == 0 && l == 0) {
        d.clk->steps += 1;
        d.clk->time += dt;
        d.clk->step_dt = dt;
    }
    const size_t E = d.nelem;
    const int q0 = live ? d.sup_off[n] : 0, q1 = live ? d.sup_off[n + 1] : 0;
    double acc = 0;
    octet_walk(
        tile, d.sup_ent, q0, q1,
        [&](unsigned p, double v[5]) {
            const size_t e = p >> 2;
            v[0] = stale ? d.vol[e] : 0;
            v[1] = stale ? d.c_mass[e] : 0;
            v[2] = stale && thermal ? d.c_tmass[e] : 0;
            v[3] = thermal ? d.tmp[(p & 3u) * E + e] : 0;
            v[4] = d.c_trdv[e];
        },
        [&](double v) { acc += v; });
    if (!stale && live) {
        if (l == 0) acc = d.vol_n[n];
        if (l == 2) acc = d.tmass[n];
    }
    const double vn = octet_get(acc, 0), tm = octet_get(acc, 2);
    if (!live) return;
    if (stale && l < 3) (l == 0 ? d.vol_n : l == 1 ? d.mass : d.tmass)[n] = acc;
    if (l == 3 && thermal) {
        if (d.bcflag[n] & kBoundZ1)
            d.T[n] = K.surface_temperature;
        else
            d.T[n] -= sf::div(sf::mul(acc, dt), tm);
    }
    if (l == 4) d.ntmp[n] = sf::div(acc, vn);
}

// N-B (k_sg_gather)
__global__ void __launch_bounds__(kSmallBlock) k_sg_gather_small(Dev d)
{
    __shared__ NodeTile<double, 1> tile;
    const int n = (int)(blockIdx.x * kSmallBlock + threadIdx.x) / kNodeLanes, l = threadIdx.x & (kNodeLanes - 1);
    const bool live = n < d.nnode;
    const int q0 = live ? d.sup_off[n] : 0, q1 = live ? d.sup_off[n + 1] : 0;
    const double vn = live ? d.vol_n[n] : 1.0;
    double s = 0.;
    octet_walk(
        tile, d.sup_ent, q0, q1, [&](unsigned p, double v[1]) { v[0] = d.tmp_sg[p >> 2]; }, [&](double v) { s += v; });
    if (live && l == 0) d.ntmp[n] = sf::div(s, vn);
}

// component j of stress_bc_node
__device__ __forceinline__ double stress_bc_component(const Consts &K, const BdryFacets &b, int n, unsigned flag,
                                                      double z, double z0, int j, double f)
{
    if (K.stress_bc_sides && (flag & kBoundAny)) {
        for (int q = b.node_off[n]; q < b.node_off[n + 1]; ++q) {
            const int k = b.node_facet[q];
            if (!(K.stress_bc_sides & (1u << (b.side_f[k] >> 2)))) continue;
            f -= b.val[j * b.nbf + k];
        }
    }
    if (j == 2 && K.elastic_foundation && (flag & kBoundZ0)) f -= K.elastic_foundation_constant * (z - z0);
    return f;
}

// N-C (k_fn_c): lane j < 3 has component j
__global__ void __launch_bounds__(kSmallBlock) k_fn_c_small(Dev d)
{
    __shared__ NodeTile<double, 3> tile;
    const int n = (int)(blockIdx.x * kSmallBlock + threadIdx.x) / kNodeLanes, l = threadIdx.x & (kNodeLanes - 1);
    const Consts &K = *d.K;
    const bool live = n < d.nnode, mine = live && l < 3;
    const double dt = d.clk->dt;
    const size_t E = d.nelem;
    const int q0 = live ? d.sup_off[n] : 0, q1 = live ? d.sup_off[n + 1] : 0;
    const unsigned flag = live ? d.bcflag[n] : 0u;
    const int nl = live ? n : 0, j = l < 3 ? l : 2;
    double *const vp = j == 0 ? d.vx : j == 1 ? d.vy : d.vz, *const xp = j == 0 ? d.x : j == 1 ? d.y : d.z,
                  *const fp = j == 0 ? d.fx : j == 1 ? d.fy : d.fz;
    const double x0 = xp[nl], v0 = vp[nl], m = d.mass[nl];
    double f = 0;
    octet_walk(
        tile, d.sup_ent, q0, q1,
        [&](unsigned p, double v[3]) {
            const double *t = d.tmp + (size_t)(p & 3u) * E + (p >> 2);
            v[0] = t[0];
            v[1] = t[4 * E];
            v[2] = t[8 * E];
        },
        [&](double v) { f -= v; });
    double v = v0;
    if (mine) {
        f = stress_bc_component(K, d.bf, n, flag, d.z[n], d.z0[n], j, f);
        if (K.is_qs) f = damp(K, f, v);
        fp[n] = f;
        v += sf::div(sf::mul(dt, f), m);
    }
    double w[3] = {octet_get(v, 0), octet_get(v, 1), octet_get(v, 2)};
    if (!mine) return;
    vbc_node(K, flag, w);
    v = j == 0 ? w[0] : j == 1 ? w[1] : w[2];
    vp[n] = v;
    const double x = x0 + sf::mul(v, dt);
    xp[n] = x;
    // output.cxx:195-208 stops on NaN/Inf coordinates
    if (not_finite(x)) atomicOr(&d.clk->status, 0x2u);
}

// ---- the FP32 form's nodes ------------------------------------------------------------

__global__ void __launch_bounds__(kSmallBlock) kf_fn_a_small(DevF d)
{
    __shared__ NodeTile<float, 5> tile;
    const int n = (int)(blockIdx.x * kSmallBlock + threadIdx.x) / kNodeLanes, l = threadIdx.x & (kNodeLanes - 1);
    const bool live = n < d.nnode, thermal = d.F->thermal;
    const double dt = d.clk->dt;
    const bool stale = !d.clk->mass_valid;
    if (n == 0 && l == 0) {
        d.clk->steps += 1;
        d.clk->time += dt;
        d.clk->npend = 0;
        d.clk->nexact = 0;
    }
    const size_t E = d.nelem;
    const int q0 = live ? d.sup_off[n] : 0, q1 = live ? d.sup_off[n + 1] : 0;
    float acc = 0.f;
    octet_walk(
        tile, d.sup_ent, q0, q1,
        [&](unsigned p, float v[5]) {
            const size_t e = p >> 2;
            v[0] = stale ? d.c_vol[e] : 0.f;
            v[1] = stale ? d.c_mass[e] : 0.f;
            v[2] = stale && thermal ? d.c_tmass[e] : 0.f;
            v[3] = thermal ? d.tmp[(p & 3u) * E + e] : 0.f;
            v[4] = d.c_trdv[e];
        },
        [&](float v) { acc += v; });
    if (!stale && live) {
        if (l == 0) acc = d.vol_n[n];
        if (l == 2) acc = d.tmass[n];
    }
    const float vn = octet_get(acc, 0), tm = octet_get(acc, 2);
    if (!live) return;
    if (stale && l < 3) (l == 0 ? d.vol_n : l == 1 ? d.mass : d.tmass)[n] = acc;
    if (l == 3 && thermal) {
        if (d.bcflag[n] & kBoundZ1)
            d.T[n] = d.K->surface_temperature;
        else
            d.T[n] -= sf::div(sf::mul(sf::widen(acc), dt), sf::widen(tm));
    }
    if (l == 4) d.ntmp[n] = acc / vn;
}

__global__ void __launch_bounds__(kSmallBlock) kf_sg_gather_small(DevF d)
{
    __shared__ NodeTile<float, 1> tile;
    const int n = (int)(blockIdx.x * kSmallBlock + threadIdx.x) / kNodeLanes, l = threadIdx.x & (kNodeLanes - 1);
    const bool live = n < d.nnode;
    const int q0 = live ? d.sup_off[n] : 0, q1 = live ? d.sup_off[n + 1] : 0;
    const float vn = live ? d.vol_n[n] : 1.f;
    float s = 0.f;
    octet_walk(
        tile, d.sup_ent, q0, q1, [&](unsigned p, float v[1]) { v[0] = d.tmp_sg[p >> 2]; }, [&](float v) { s += v; });
    if (live && l == 0) d.ntmp[n] = s / vn;
}

// lanes 0-2 the FP64 reference part, 3-5 the FP32 part
__global__ void __launch_bounds__(kSmallBlock) kf_fn_c_small(DevF d)
{
    __shared__ NodeTile<double, 6> tile;
    const int n = (int)(blockIdx.x * kSmallBlock + threadIdx.x) / kNodeLanes, l = threadIdx.x & (kNodeLanes - 1);
    const Consts &K = *d.K;
    const bool live = n < d.nnode, mine = live && l < 3;
    const double dt = d.clk->dt;
    const size_t E = d.nelem;
    const int q0 = live ? d.sup_off[n] : 0, q1 = live ? d.sup_off[n + 1] : 0;
    const unsigned flag = live ? d.bcflag[n] : 0u;
    const int nl = live ? n : 0, j = l < 3 ? l : 2;
    float *const vp = j == 0 ? d.vx : j == 1 ? d.vy : d.vz, *const fp = j == 0 ? d.fx : j == 1 ? d.fy : d.fz;
    double *const xp = j == 0 ? d.x : j == 1 ? d.y : d.z;
    const double x0 = xp[nl];
    const float v0 = vp[nl], m = d.mass[nl];
    double h = 0;
    float g = 0.f;
    // (both parts in one walk: the FP32 values travel as the low word of a double)
    octet_walk(
        tile, d.sup_ent, q0, q1,
        [&](unsigned p, double v[6]) {
            const size_t o = (size_t)(p & 3u) * E + (p >> 2);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                v[c] = d.f0[o + 4 * c * E];
                v[3 + c] = __hiloint2double(0, __float_as_int(d.tmp[o + 4 * c * E]));
            }
        },
        [&](double v) {
            if (l < 3)
                h -= v;
            else
                g -= __int_as_float(__double2loint(v));
        });
    g = octet_get(g, 3 + j);
    float v = v0;
    if (mine) {
        h = stress_bc_component(K, d.bf, n, flag, d.z[n], d.z0[n], j, h);
        float f = sf::to_float(h + sf::widen(g));
        if (d.F->is_qs) f = damp(K, f, v);
        fp[n] = f;
        v += sf::to_float(dt) * f / m;
    }
    float w[3] = {octet_get(v, 0), octet_get(v, 1), octet_get(v, 2)};
    if (!mine) return;
    vbc_node(K, flag, w);
    v = j == 0 ? w[0] : j == 1 ? w[1] : w[2];
    vp[n] = v;
    const double x = x0 + sf::mul(sf::widen(v), dt);
    xp[n] = x;
    if (not_finite(x)) atomicOr(&d.clk->status, 0x2u);
}

// ---- elements: four lanes each ----------------------------------------------------------

// r[k] = a[k] b[k] on the integer pipes, checked together; out of sf::unpack's
// range on the FP64 unit, out of line
static __device__ __noinline__ void products_exact(int n, const double *a, const double *b, double *r)
{
    for (int k = 0; k < n; ++k) r[k] = a[k] * b[k];
}

template <int N>
__device__ __forceinline__ void products(const double (&a)[N], const double (&b)[N], double (&r)[N])
{
    uint32_t far = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) r[k] = sf::prod(sf::unpack(a[k], far), sf::unpack(b[k], far));
    if (!sf::in_range(far)) {
        double u[N], v[N], w[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            u[k] = a[k];
            v[k] = b[k];
        }
        products_exact(N, u, v, w);
#pragma unroll
        for (int k = 0; k < N; ++k) r[k] = w[k];
    }
}

template <class R>
__device__ __forceinline__ R quad_get(R v, int lane)
{
    return __shfl_sync(0xffffffffu, v, lane, 4);
}

// entry i of a table of two-bit (four-bit) numbers
__device__ __forceinline__ int two(unsigned table, int i) { return (table >> (2 * i)) & 3; }
__device__ __forceinline__ int four(unsigned table, int i) { return (table >> (4 * i)) & 15; }

// x with its sign flipped where minus
__device__ __forceinline__ double signed_by(double x, bool minus)
{
    return sf::from_bits(sf::bits(x) ^ (minus ? sf::kSign : 0ull));
}

// The FP32 form's E-A (kf_fe_a) with lane i at node i: its cofactor, gradient,
// reference force and row of the conduction; lanes 0 and 1 rotate the stress
// and the strain, 2 and 3 store the strain rate and its trace.  The FP32 sums
// over the nodes are formed by every lane, in kf_fe_a's order.
// A small mesh's pass is one thread's chain of about 2,000 instructions, 37 of
// them on the FP64 unit: a lane's is a third of it, 12 on the FP64 unit (9.6k
// elements 12.9 -> 10.9 us).  Four lanes take 1.3 times the FP64 instructions
// of one thread, so beyond a few warps a scheduler the pass is slower.
__global__ void __launch_bounds__(kSmallBlock) kf_ea_quad(DevF d, int e0, unsigned nblocks)
{
    __shared__ double s_x[3][kSmallBlock];
    __shared__ float s_f[6][kSmallBlock];
    const int i = threadIdx.x & 3, base = threadIdx.x & ~3;
    const int e_ = e0 + (int)(blockIdx.x * kSmallBlock + threadIdx.x) / 4;
    const Consts &K = *d.K;
    const ConstsF &F = *d.F;
    const bool live = e_ < d.nelem;
    const int e = live ? e_ : d.nelem - 1;
    const bool dt_step = (K.fixed_dt == 0) && (d.clk->steps % 10 == 0);
    if (e_ == 0 && i == 0) d.clk->mass_valid = 0;
    const size_t E = d.nelem;
    const int n = reinterpret_cast<const int *>(d.conn)[4 * (size_t)e + i];
    const MixF &xf = F.mix[d.mix[e]];
    const bool rotate = F.rheol & 1;
    const float dt = sf::to_float(d.clk->dt);
    float *field = i == 0 ? d.stress : d.strain, s[6];
    if (rotate && i < 2) f_load6(field, E, e, s);
    const double T = d.T[n], vol_was = d.vol[e], s0 = d.s0[e];
    const double x[3] = {d.x[n], d.y[n], d.z[n]};
    s_f[0][threadIdx.x] = d.vx[n];
    s_f[1][threadIdx.x] = d.vy[n];
    s_f[2][threadIdx.x] = d.vz[n];
    // f_cofactors: the edge to each lane's node; lanes 1-3 the cross products of
    // the two others' (b, q) (q, a) (a, b); lane k < 3 the three products' k-th
    // components' sum, which is minus lane 0's cofactor
    double cf[3], det;
    {
        const int iu = two(0x7a, i), iv = two(0x9f, i), kk = i < 3 ? i : 2;     // - 2 3 1 | - 3 1 2
        double u[3], v[3], a[3], c1[3];
        uint32_t far = 0;
        sf::Op ou[3], ov[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) s_x[k][threadIdx.x] = x[k] - quad_get(x[k], 0);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            u[k] = s_x[k][base + iu];
            v[k] = s_x[k][base + iv];
            a[k] = s_x[k][base + 1];
            ou[k] = sf::unpack(u[k], far);
            ov[k] = sf::unpack(v[k], far);
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int p = (k + 1) % 3, q = (k + 2) % 3;
            cf[k] = fma(u[p], v[q], -sf::prod(ou[q], ov[p]));
            s_x[k][threadIdx.x] = cf[k];
        }
        __syncwarp();
        const double sum = s_x[kk][base + 1] + s_x[kk][base + 2] + s_x[kk][base + 3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            c1[k] = s_x[k][base + 1];
            const double c0 = signed_by(quad_get(sum, k), true);
            if (i == 0) cf[k] = c0;
        }
        det = fma(a[0], c1[0], fma(a[1], c1[1], sf::prod(sf::unpack(a[2], far), sf::unpack(c1[2], far))));
        far = max(far, __shfl_xor_sync(0xffffffffu, far, 1, 4));
        far = max(far, __shfl_xor_sync(0xffffffffu, far, 2, 4));
        if (!sf::in_range(far)) {
            double r[12];
            det = f_cofactors_exact(d, d.conn[e], r);
#pragma unroll
            for (int k = 0; k < 3; ++k) cf[k] = r[3 * i + k];
        }
    }
    const double vol = sf::mul(det, 1.0 / 6.0);
    const float volf = sf::to_float(vol);
    if (live && i == 0) {
        d.vol_old[e] = vol_was;
        d.vol[e] = vol;
        d.c_vol[e] = volf;
        if (not_positive(vol)) atomicOr(&d.clk->status, 0x4u);
    }
    // f_reference_force, node i
    {
        const double s6 = sf::mul(s0, 1.0 / 6.0), buoy = F.gravity != 0.f ? sf::mul(xf.rho_g4, vol) : 0.0;
        uint32_t far = 0;
        const sf::Op o6 = sf::unpack(s6, far);
        double fx = sf::prod(o6, sf::unpack(cf[0], far)), fy = sf::prod(o6, sf::unpack(cf[1], far));
        if (!sf::in_range(far)) {
            fx = sf::from_bits(sf::mul_slow(sf::bits(s6), sf::bits(cf[0])));
            fy = sf::from_bits(sf::mul_slow(sf::bits(s6), sf::bits(cf[1])));
        }
        if (live) {
            d.f0[i * E + e] = fx;
            d.f0[(i + 4) * E + e] = fy;
            d.f0[(i + 8) * E + e] = fma(s6, cf[2], buoy);
        }
    }
    double minh = 0;
    if (dt_step) {
        const double m = fma(cf[0], cf[0], fma(cf[1], cf[1], cf[2] * cf[2]));
        minh = 6 * vol / sqrt(fmax(fmax(quad_get(m, 0), quad_get(m, 1)), fmax(quad_get(m, 2), quad_get(m, 3))));
    }
    const float iv = 1.f / sf::to_float(det);
    float g[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        g[k] = sf::to_float(cf[k]) * iv;
        s_f[3 + k][threadIdx.x] = g[k];
        if (live) d.shp[(size_t)(4 * k + i) * E + e] = g[k];
    }
    __syncwarp();
    float V[4][3], dx[4], dy[4], dz[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int k = 0; k < 3; ++k) V[j][k] = s_f[k][base + j];
        dx[j] = s_f[3][base + j];
        dy[j] = s_f[4][base + j];
        dz[j] = s_f[5][base + j];
    }
    {
        const float t = sf::to_float(T);
        const float rT = f_rho(F, xf, elem_mean4(quad_get(t, 0), quad_get(t, 1), quad_get(t, 2), quad_get(t, 3)));
        if (live && i == 2) d.c_mass[e] = (F.is_qs ? xf.rho_qs : rT) * volf * 0.25f;
        if (live && i == 3 && F.thermal) d.c_tmass[e] = rT * xf.cp * volf * 0.25f;
    }
    if (rotate && i < 2) {
        float w3, w4, w5;
        spin(V, dx, dy, dz, w3, w4, w5);
        jaumann(s, dt, w3, w4, w5);
        if (live) f_store6(field, E, e, s);
    }
    // f_next_contrib
    if (i >= 2) {
        float D[6];
        strain_rate(V, dx, dy, dz, D);
        if (live && i == 2) f_store6(d.srate_next, E, e, D);
        if (live && i == 3) d.c_trdv[e] = tr3(D) * volf;
    }
    if (F.thermal) {
        const double T0 = quad_get(T, 0);
        const float t = sf::to_float(T - T0);
        const float t1 = quad_get(t, 1), t2 = quad_get(t, 2), t3 = quad_get(t, 3);
        const float gx = dx[1] * t1 + dx[2] * t2 + dx[3] * t3;
        const float gy = dy[1] * t1 + dy[2] * t2 + dy[3] * t3;
        const float gz = dz[1] * t1 + dz[2] * t2 + dz[3] * t3;
        const float kv = xf.k * volf;
        if (live) d.tmp[i * E + e] = kv * (g[0] * gx + g[1] * gy + g[2] * gz);
    }
    if (dt_step) {
        Dev dd;
        dd.conn = d.conn;
        dd.T = d.T;
        dd.mix = d.mix;
        dd.K = d.K;
        dd.clk = d.clk;
        dt_reduce_and_finalize(dd, minh, live, nblocks);
    }
}

// E-A (k_ea_geometry, k_ea_rotate, k_ea_conduction in one): lane i has node i
// of the element: its gradient, its products with the velocity, its row of
// the conduction matrix; lanes 0-2 sum the rates' components and rotate one
// normal and one off-diagonal component each.
__global__ void __launch_bounds__(kSmallBlock) k_ea_quad(Dev d, int e0, unsigned nblocks)
{
    __shared__ double s_x[9][kSmallBlock], s_g[3][kSmallBlock];
    const int i = threadIdx.x & 3, base = threadIdx.x & ~3, kk = i < 3 ? i : 2;
    const int e_ = e0 + (int)(blockIdx.x * kSmallBlock + threadIdx.x) / 4;
    const Consts &K = *d.K;
    const bool live = e_ < d.nelem;
    const int e = live ? e_ : d.nelem - 1;
    const bool dt_step = (K.fixed_dt == 0) && (d.clk->steps % 10 == 0);
    const double step_dt = d.clk->step_dt;
    if (e_ == 0 && i == 0) d.clk->mass_valid = 0;
    const size_t E = d.nelem;
    const int n = reinterpret_cast<const int *>(d.conn)[4 * (size_t)e + i];
    const Mix &x = K.M.mix[d.mix[e]];
    const bool rotate = K.rheol & 1;
    // the rotation's operands of both fields, early: s_A s_B (times w_k), the
    // two other terms of the off-diagonal component, those of the normal one
    const int cA = two(0x10, kk), cB = two(0x29, kk);                  // 0 0 1 | 1 2 2
    const int cC = four(0x334, kk), cD = four(0x455, kk);              // 4 3 3 | 5 5 4
    const int cP = four(0x433, kk), cQ = four(0x554, kk);              // 3 3 4 | 4 5 5
    double r[2][8];
    if (rotate) {
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            const double *a = (f ? d.strain : d.stress) + e;
            r[f][0] = a[cA * E];
            r[f][1] = a[cB * E];
            r[f][2] = a[cC * E];
            r[f][3] = a[cD * E];
            r[f][4] = a[cP * E];
            r[f][5] = a[cQ * E];
            r[f][6] = a[kk * E];
            r[f][7] = a[(3 + kk) * E];
        }
    }
    const double T = d.T[n], v[3] = {d.vx[n], d.vy[n], d.vz[n]}, vol_was = d.vol[e];
    s_x[0][threadIdx.x] = d.x[n];
    s_x[1][threadIdx.x] = d.y[n];
    s_x[2][threadIdx.x] = d.z[n];
    __syncwarp();
    auto edge = [&](int k, int p, int q) { return s_x[k][base + p] - s_x[k][base + q]; };
    // compute_volume: lane k < 3 its k-th term
    double vol;
    {
        // x edge 01 12 23; (u, v) = (23, 12) (01, 23) (12, 01)
        const int xp = kk, up = two(0x12, kk), vp = two(0x09, kk);     // first nodes: 2 0 1 | 1 2 0
        const double xe = edge(0, xp, xp + 1), uy = edge(1, up, up + 1), uz = edge(2, up, up + 1),
                     vy = edge(1, vp, vp + 1), vz = edge(2, vp, vp + 1);
        double p[2], t[1];
        products<2>({uy, vy}, {vz, uz}, p);
        products<1>({xe}, {p[0] - p[1]}, t);
        vol = sf::div6(quad_get(t[0], 0) + quad_get(t[0], 1) + quad_get(t[0], 2));
    }
    if (live && i == 0) {
        d.vol_old[e] = vol_was;
        d.vol[e] = vol;
        if (not_positive(vol)) atomicOr(&d.clk->status, 0x4u);
    }
    double minh = 0;
    if (dt_step) {
        // min_height: lane f one facet: e01 x e02, e01 x e03, e02 x e23, e12 x e23
        const int p0 = two(0x40, i), p1 = two(0xa5, i);               // 0 0 0 1 | 1 1 2 2
        const int q0 = two(0xa0, i), q1 = two(0xfe, i);               // 0 0 2 2 | 2 3 3 3
        double a[3], b[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a[k] = edge(k, p0, p1);
            b[k] = edge(k, q0, q1);
        }
        const double c0 = a[1] * b[2] - a[2] * b[1], c1 = a[2] * b[0] - a[0] * b[2], c2 = a[0] * b[1] - a[1] * b[0];
        const double a2 = c0 * c0 + c1 * c1 + c2 * c2;
        const double m2 = smax(smax(quad_get(a2, 0), quad_get(a2, 1)), smax(quad_get(a2, 2), quad_get(a2, 3)));
        minh = 3 * vol / (sqrt(m2) / 2);
    }
    // compute_shape_fn: edges (13, 12) (02, 23) (13, 03) (01, 02)
    double g[3];
    {
        const int p0 = two(0x11, i), p1 = two(0x7b, i);               // 1 0 1 0 | 3 2 3 1
        const int q0 = two(0x09, i), q1 = two(0xbe, i);               // 1 2 0 0 | 2 3 3 2
        double a[3], b[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a[k] = edge(k, p0, p1);
            b[k] = edge(k, q0, q1);
        }
        const double iv = sf::div(1.0, sf::mul(6.0, vol));
        double p[6];
        products<6>({a[1], a[2], a[2], a[0], a[0], a[1]}, {b[2], b[1], b[0], b[2], b[1], b[0]}, p);
        products<3>({iv, iv, iv}, {p[0] - p[1], p[2] - p[3], p[4] - p[5]}, g);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s_g[k][threadIdx.x] = g[k];
        if (live) d.shp[(size_t)(4 * k + i) * E + e] = g[k];
    }
    const double Tn[4] = {quad_get(T, 0), quad_get(T, 1), quad_get(T, 2), quad_get(T, 3)};
    // compute_mass's element half
    {
        const double rT = mat_rho(K.M, x, elem_mean4(Tn[0], Tn[1], Tn[2], Tn[3]));
        if (live && i == 0) d.c_mass[e] = sf::quarter(sf::mul(K.is_qs ? x.rho_qs : rT, vol));
        if (live && i == 1 && K.thermal) d.c_tmass[e] = sf::quarter(sf::mul(sf::mul(rT, x.cp), vol));
    }
    // spin and next strain rate (as k_ea_rotate forms them: half the brackets'
    // sum, exact while every operand of the element is in sf::unpack's range)
    double D[3], u[3];
    {
        uint32_t far = 0;
        sf::Op ov[3], og[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            ov[k] = sf::unpack(v[k], far);
            og[k] = sf::unpack(g[k], far);
        }
        far = max(far, __shfl_xor_sync(0xffffffffu, far, 1, 4));
        far = max(far, __shfl_xor_sync(0xffffffffu, far, 2, 4));
        const double xy = sf::prod(ov[0], og[1]), yx = sf::prod(ov[1], og[0]), xz = sf::prod(ov[0], og[2]),
                     zx = sf::prod(ov[2], og[0]), yz = sf::prod(ov[1], og[2]), zy = sf::prod(ov[2], og[1]);
        __syncwarp();                    // (the coordinates have been read)
#pragma unroll
        for (int k = 0; k < 3; ++k) s_x[k][threadIdx.x] = sf::prod(ov[k], og[k]);
        s_x[3][threadIdx.x] = xy + yx;
        s_x[4][threadIdx.x] = xz + zx;
        s_x[5][threadIdx.x] = yz + zy;
        s_x[6][threadIdx.x] = xy - yx;
        s_x[7][threadIdx.x] = xz - zx;
        s_x[8][threadIdx.x] = yz - zy;
        __syncwarp();
        double Dk = sf::add0(s_x[kk][base]), tk = sf::add0(s_x[3 + kk][base]), uk = sf::add0(s_x[6 + kk][base]);
#pragma unroll
        for (int j = 1; j < 4; ++j) {
            Dk += s_x[kk][base + j];
            tk += s_x[3 + kk][base + j];
            uk += s_x[6 + kk][base + j];
        }
        tk = sf::half(tk);
        if (live && !sf::in_range(far)) {
            double r[9];
            ea_rates_exact(d, e, r);
            Dk = kk == 0 ? r[0] : kk == 1 ? r[1] : r[2];
            tk = kk == 0 ? r[3] : kk == 1 ? r[4] : r[5];
            uk = 2 * (kk == 0 ? r[6] : kk == 1 ? r[7] : r[8]);
        }
        if (live && i < 3) {
            d.srate_next[kk * E + e] = Dk;
            d.srate_next[(3 + kk) * E + e] = tk;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            D[k] = quad_get(Dk, k);
            u[k] = quad_get(uk, k);
        }
    }
    if (live && i == 3) d.c_trdv[e] = sf::mul(D[0] + D[1] + D[2], vol);
    // rotate_stress with u = 2 w (k_ea_rotate), lane k < 3 the components k and 3 + k
    if (rotate) {
        uint32_t farw = 0;
        const sf::Op ow[3] = {sf::unpack(u[0], farw), sf::unpack(u[1], farw), sf::unpack(u[2], farw)};
        const sf::Op odt = sf::unpack(step_dt, farw), hdt = half_op(odt);
        const sf::Op wk = kk == 0 ? ow[0] : kk == 1 ? ow[1] : ow[2];
        const sf::Op wC = kk == 2 ? ow[1] : ow[2], wD = kk == 0 ? ow[1] : ow[0];       // w5 w5 w4 | w4 w3 w3
        const sf::Op wP = kk == 2 ? ow[1] : ow[0], wQ = kk == 0 ? ow[1] : ow[2];       // w3 w3 w4 | w4 w5 w5
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            double *arr = f ? d.strain : d.stress;
            uint32_t far = farw;
            const double off = sf::prod(sf::unpack(r[f][0], far), wk) - sf::prod(sf::unpack(r[f][1], far), wk) +
                               signed_by(sf::prod(sf::unpack(r[f][2], far), wC), kk == 0) +
                               signed_by(sf::prod(sf::unpack(r[f][3], far), wD), kk != 2);
            const double nrm = signed_by(sf::prod(sf::unpack(r[f][4], far), wP), kk == 0) +
                               signed_by(sf::prod(sf::unpack(r[f][5], far), wQ), kk != 2);
            const double sn = r[f][6] + sf::prod(odt, sf::unpack(nrm, far));
            const double so = r[f][7] + sf::prod(hdt, sf::unpack(off, far));
            const unsigned bad = __ballot_sync(0xffffffffu, !sf::in_range(far));
            if (!live) continue;
            if ((bad >> (base & 31)) & 15u) {
                if (i == 0) ea_rotate_exact(d, e, arr, step_dt, 0.5 * u[0], 0.5 * u[1], 0.5 * u[2]);
            } else if (i < 3) {
                arr[kk * E + e] = sn;
                arr[(3 + kk) * E + e] = so;
            }
        }
    }
    // the conduction vector's row i
    if (K.thermal) {
        double gj[4][3], p[12], q[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < 3; ++k) gj[j][k] = s_g[k][base + j];
        products<12>({g[0], g[1], g[2], g[0], g[1], g[2], g[0], g[1], g[2], g[0], g[1], g[2]},
                     {gj[0][0], gj[0][1], gj[0][2], gj[1][0], gj[1][1], gj[1][2], gj[2][0], gj[2][1], gj[2][2], gj[3][0],
                      gj[3][1], gj[3][2]},
                     p);
        products<4>({p[0] + p[1] + p[2], p[3] + p[4] + p[5], p[6] + p[7] + p[8], p[9] + p[10] + p[11]},
                    {Tn[0], Tn[1], Tn[2], Tn[3]}, q);
        const double diffusion = sf::add0(q[0]) + q[1] + q[2] + q[3];
        if (live) d.tmp[(size_t)i * E + e] = sf::mul(diffusion, sf::mul(x.k, vol));
    }
    if (dt_step) dt_reduce_and_finalize(d, minh, live && i == 0, nblocks);
}

// E-C (k_fe_c): lane i has node i's force
__global__ void __launch_bounds__(kSmallBlock) k_fe_c_quad(Dev d)
{
    const int i = threadIdx.x & 3, e_ = (int)(blockIdx.x * kSmallBlock + threadIdx.x) / 4;
    const Consts &K = *d.K;
    const bool live = e_ < d.nelem;
    const int e = live ? e_ : d.nelem - 1;
    const size_t E = d.nelem;
    const int n = reinterpret_cast<const int *>(d.conn)[4 * (size_t)e + i];
    // lane k < 3 has the k-th normal stress to itself: it is corrected in place,
    // so no other lane may read it from memory (lanes of a warp run in any order
    // between barriers); the shear stresses are not written
    const bool mine = live && i < 3;
    double sn = mine ? d.stress[i * E + e] : 0.0;
    double s[6];
#pragma unroll
    for (int k = 3; k < 6; ++k) s[k] = d.stress[k * E + e];
    const double g[3] = {d.shp[(size_t)i * E + e], d.shp[(size_t)(4 + i) * E + e], d.shp[(size_t)(8 + i) * E + e]};
    const double vol = d.vol[e], dp = d.dp[e], a = d.ntmp[n], T = d.T[n];
    const double dpe = sf::add0(quad_get(a, 0)) + quad_get(a, 1) + quad_get(a, 2) + quad_get(a, 3);
    const double ddp = sf::div3(-dp + sf::quarter(dpe));
    sn += ddp;
    if (mine) d.stress[i * E + e] = sn;
#pragma unroll
    for (int k = 0; k < 3; ++k) s[k] = quad_get(sn, k);
    const double Tm = elem_mean4(quad_get(T, 0), quad_get(T, 1), quad_get(T, 2), quad_get(T, 3));
    double buoy = 0;
    if (K.gravity != 0) buoy = sf::quarter(sf::mul(mat_rho(K.M, K.M.mix[d.mix[e]], Tm), K.gravity));
    double p[9], q[3];
    products<9>({s[0], s[3], s[4], s[3], s[1], s[5], s[4], s[5], s[2]},
                {g[0], g[1], g[2], g[0], g[1], g[2], g[0], g[1], g[2]}, p);
    products<3>({p[0] + p[1] + p[2], p[3] + p[4] + p[5], p[6] + p[7] + p[8] + buoy}, {vol, vol, vol}, q);
    if (!live) return;
    d.tmp[(size_t)i * E + e] = q[0];
    d.tmp[(size_t)(4 + i) * E + e] = q[1];
    d.tmp[(size_t)(8 + i) * E + e] = q[2];
}

}  // namespace des
