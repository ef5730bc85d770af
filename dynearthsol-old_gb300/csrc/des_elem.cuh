// Element passes of the FP64 step, one thread per element: E-A (update_mesh's
// element half, rotate_stress, the next step's contributions, the dt minimum)
// as three kernels (geometry, rates and rotation, conduction), and E-C (NMD
// correction, force vectors).
//
// What bounds them: GB300's FP64 pipe.  It retires 502 G instructions/s (a
// warp's instruction every 20 clocks of an SM, measured with chains of DADD,
// DMUL or DFMA at 4 to 32 warps per SM; one warp alone gets one per 68
// clocks), and the reference's arithmetic for E-A is 385 of them per element.
// Every product and quotient is on the integer pipes here (sf::prod on
// operands taken apart once, sf::div), and one of the rotation's three
// sum-and-difference pairs, which leaves 154 (41 + 81 + 32 over the three
// kernels; E-C 41).
// Three kernels rather than one: the fused pass was limited by instruction
// fetch (its 2,800 instructions of loop bodies exceed what the instruction
// caches hold for warps at different places: a quarter of the warps' time
// was "no instruction"), and the split bodies are 700 to 1,100 each.  The
// gradients' way through memory that the split costs (192 B per element) is
// cheap for a pass at a fifth of the DRAM rate.  Loops over nodes stay rolled for
// the same reason.
// On a 100x100x40 box (2.4M elements): E-A 1,248 us before (one kernel, 92
// products on the integer pipes, 260 FP64 instructions), 971 us fused with
// all products on them, 796 us split (geometry 231, rates and rotation 386
// at the FP64 pipe's peak, conduction 175; 829 in the mean over steps, of which
// every tenth forms dt); E-C 258 -> 211 us.
#pragma once

#include "des_kernels.cuh"

namespace des {

constexpr int kEaBlock = 128;     // threads of a block, in E-A's kernels and E-C

// Products are on the integer pipes (sf::prod), exact while the stage's
// operands are in sf::unpack's range; an element with one outside is formed
// again on the FP64 unit, out of line.

// an operand in shared memory: an 8-byte column and a 4-byte column per thread
__device__ __forceinline__ void put_op(double *w, uint32_t *x, const sf::Op &a)
{
    *w = __hiloint2double((int)a.hi, (int)a.lo);
    *x = a.ex;
}
__device__ __forceinline__ sf::Op get_op(const double *w, const uint32_t *x)
{
    const double v = *w;
    sf::Op a;
    a.lo = (uint32_t)__double2loint(v);
    a.hi = (uint32_t)__double2hiint(v);
    a.ex = *x;
    return a;
}
// a / 2 (an operand in range)
__device__ __forceinline__ sf::Op half_op(sf::Op a)
{
    a.ex -= a.hi ? 1u << 20 : 0u;
    return a;
}

// ---- geometry ---------------------------------------------------------------

// The edges X[i] - X[j] of the vertex pairs 01 02 03 12 13 23 in shared
// memory, three components each, a column per thread.
constexpr int kE01 = 0, kE02 = 3, kE03 = 6, kE12 = 9, kE13 = 12, kE23 = 15, kEdgeCols = 18;

__device__ __forceinline__ void load_edge(const double *se, int c, double a[3])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) a[k] = se[(c + k) * kEaBlock];
}

// the squared norm of a x b (tri_area2's terms: the facet's cross product up
// to the sign of both factors or of the whole, which the squares do not see)
__device__ __forceinline__ double edge_norm2(const double *se, int ca, int cb)
{
    double a[3], b[3];
    load_edge(se, ca, a);
    load_edge(se, cb, b);
    const double d0 = a[1] * b[2] - a[2] * b[1], d1 = a[2] * b[0] - a[0] * b[2], d2 = a[0] * b[1] - a[1] * b[0];
    return d0 * d0 + d1 * d1 + d2 * d2;
}

// min_height (geometry.cxx:280-293) from the edges: facets (0,1,2): e01 x e02,
// (0,1,3): e01 x e03, (2,3,0): e02 x e23, (2,3,1): e12 x e23.  Out of line:
// every tenth step calls it, and its registers stay out of the pass's own.
static __device__ __noinline__ double edge_min_height(const double *se, double vol)
{
    const double m2 = smax(smax(edge_norm2(se, kE01, kE02), edge_norm2(se, kE01, kE03)),
                           smax(edge_norm2(se, kE02, kE23), edge_norm2(se, kE12, kE23)));
    return 3 * vol / (sqrt(m2) / 2);
}

// The stages on the FP64 unit, for an element with an operand outside
// sf::unpack's range (a subnormal or huge number, an infinity, NaN); out of
// line, each from what the stage started from.
static __device__ __noinline__ double ea_volume_exact(const double *se)
{
    double a[3], b[3], c[3];                 // e01, e12, e23
    load_edge(se, kE01, a);
    load_edge(se, kE12, b);
    load_edge(se, kE23, c);
    return sf::div6(a[0] * (c[1] * b[2] - b[1] * c[2]) + b[0] * (a[1] * c[2] - c[1] * a[2]) +
                    c[0] * (b[1] * a[2] - a[1] * b[2]));
}

static __device__ __noinline__ void ea_gradients_exact(const Dev &d, int e, double vol)
{
    double X[4][3], dx[4], dy[4], dz[4];
    load_xyz4(d, d.conn[e], X);
    shape_fn(X, vol, dx, dy, dz);
    store_shp(d, e, dx, dy, dz);
}

// volume, shape functions, mass contributions, dt minimum.  FP64 pipe 70 % and
// integer ALU 70 % busy; 10 blocks of 128 per SM (8 or 12: the same within 1 %)
//
// PARTS: what the kernel does.  kStep is E-A's; the others are the reference's
// functions: compute_volume (vol_old taken along with kSaveOld), compute_mass's
// element half into tmp[0..2] (temperatures from Tsrc, NULL for 0),
// compute_shape_fn.
enum { kVolume = 1, kSaveOld = 2, kMass = 4, kShape = 8, kStep = 16 };
constexpr int kStepGeometry = kStep | kVolume | kSaveOld | kShape;

template <int PARTS>
__global__ void __launch_bounds__(kEaBlock, 10) k_ea_geometry(Dev d, int e0, unsigned nblocks, const double *Tsrc)
{
    using sf::Op;
    using sf::prod;
    using sf::unpack;
    __shared__ double s_edge[kEdgeCols * kEaBlock];
    const int e = e0 + blockIdx.x * kEaBlock + threadIdx.x;
    const Consts &K = *d.K;
    const bool live = e < d.nelem;
    const int4 c = live ? d.conn[e] : int4{0, 0, 0, 0};
    const bool dt_step = (PARTS & kStep) && (K.fixed_dt == 0) && (d.clk->steps % 10 == 0);
    if ((PARTS & kStep) && e == 0) d.clk->mass_valid = 0;
    double minh = 0;
    if (live) {
        const size_t E = d.nelem;
        double *se = s_edge + threadIdx.x;
        double e01[3], e12[3], e23[3];
        if (PARTS & (kVolume | kShape)) {
            double X[4][3];
            load_xyz4(d, c, X);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                e01[k] = X[0][k] - X[1][k];
                e12[k] = X[1][k] - X[2][k];
                e23[k] = X[2][k] - X[3][k];
                se[(kE01 + k) * kEaBlock] = e01[k];
                se[(kE12 + k) * kEaBlock] = e12[k];
                se[(kE23 + k) * kEaBlock] = e23[k];
                if (PARTS & kShape) {
                    se[(kE02 + k) * kEaBlock] = X[0][k] - X[2][k];
                    se[(kE03 + k) * kEaBlock] = X[0][k] - X[3][k];
                    se[(kE13 + k) * kEaBlock] = X[1][k] - X[3][k];
                }
            }
        }
        double vol;
        if (PARTS & kVolume) {
            // compute_volume (geometry.cxx:29-49)
            uint32_t far = 0;
            Op a[3], b[3], g[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                a[k] = unpack(e01[k], far);
                b[k] = unpack(e12[k], far);
                g[k] = unpack(e23[k], far);
            }
            const double c0 = prod(g[1], b[2]) - prod(b[1], g[2]);
            const double c1 = prod(a[1], g[2]) - prod(g[1], a[2]);
            const double c2 = prod(b[1], a[2]) - prod(a[1], b[2]);
            vol = sf::div6(prod(a[0], unpack(c0, far)) + prod(b[0], unpack(c1, far)) + prod(g[0], unpack(c2, far)));
            if (!sf::in_range(far)) vol = ea_volume_exact(se);
            if (PARTS & kSaveOld) d.vol_old[e] = d.vol[e];
            d.vol[e] = vol;
            if (not_positive(vol)) atomicOr(&d.clk->status, 0x4u);
        } else {
            vol = d.vol[e];
        }
        if (dt_step) minh = edge_min_height(se, vol);
        if (PARTS & (kMass | kStep)) {
            // compute_mass's element half (geometry.cxx:354-365)
            const Mix &x = K.M.mix[d.mix[e]];
            const double *Ts = (PARTS & kStep) ? d.T : Tsrc;
            double Tn[4] = {0, 0, 0, 0};
            if ((PARTS & kStep) || Ts) load_nodal4(Ts, c, Tn);
            const double rT = mat_rho(K.M, x, elem_mean4(Tn[0], Tn[1], Tn[2], Tn[3]));
            const double rho = K.is_qs ? x.rho_qs : rT;
            ((PARTS & kStep) ? d.c_mass : d.tmp + E)[e] = sf::quarter(sf::mul(rho, vol));
            if (K.thermal)
                ((PARTS & kStep) ? d.c_tmass : d.tmp + 2 * E)[e] = sf::quarter(sf::mul(sf::mul(rT, x.cp), vol));
            if (!(PARTS & kStep)) d.tmp[e] = vol;
        }
        if (PARTS & kShape) {
            // compute_shape_fn (geometry.cxx:410-452): node i's gradient is
            // (a x b) / 6V with the edges (a, b) = (13, 12) (02, 23) (13, 03) (01, 02)
            uint32_t far = 0;
            const Op oiv = unpack(sf::div(1.0, sf::mul(6.0, vol)), far);
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
                double ea[3], eb[3], g[3];
                load_edge(se, (0x0c3c >> (4 * i)) & 15, ea);
                load_edge(se, (0x36f9 >> (4 * i)) & 15, eb);
                Op a[3], b[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    a[k] = unpack(ea[k], far);
                    b[k] = unpack(eb[k], far);
                }
                g[0] = prod(a[1], b[2]) - prod(a[2], b[1]);
                g[1] = prod(a[2], b[0]) - prod(a[0], b[2]);
                g[2] = prod(a[0], b[1]) - prod(a[1], b[0]);
#pragma unroll
                for (int k = 0; k < 3; ++k) d.shp[(size_t)(4 * k + i) * E + e] = prod(oiv, unpack(g[k], far));
            }
            if (!sf::in_range(far)) ea_gradients_exact(d, e, vol);
        }
    }
    if (dt_step) dt_reduce_and_finalize(d, minh, live, nblocks);
}

// ---- rates and rotation --------------------------------------------------------

static __device__ __noinline__ void ea_rates_exact(const Dev &d, int e, double *out)
{
    double V[4][3], dx[4], dy[4], dz[4];
    load_vel4(d, d.conn[e], V);
    load_shp(d, e, dx, dy, dz);
    strain_rate(V, dx, dy, dz, out);
    spin(V, dx, dy, dz, out[6], out[7], out[8]);
}

static __device__ __noinline__ void ea_rotate_exact(const Dev &d, int e, double *arr, double dt, double w3, double w4,
                                                    double w5)
{
    double s[6];
    load6(arr, d.nelem, e, s);
    jaumann(s, dt, w3, w4, w5);
    store6(arr, d.nelem, e, s);
}

// the next strain rate, its dvoldt contribution, rotate_stress.  81 FP64
// instructions per element, the pipe near its measured peak; 8 blocks of 128
// per SM
//
// PARTS: kRates the strain rate into out, kDvoldt its dvoldt contribution,
// kRotate the rotation with the current dt, kStepRotate the same with the
// running step's, where the rheology has it.
enum { kRates = 1, kDvoldt = 2, kRotate = 4, kStepRotate = 8 };
constexpr int kStepRates = kRates | kDvoldt | kStepRotate;

template <int PARTS>
__global__ void __launch_bounds__(kEaBlock, 8) k_ea_rotate(Dev d, int e0, double *out)
{
    using sf::Op;
    using sf::prod;
    using sf::unpack;
    const int e = e0 + blockIdx.x * kEaBlock + threadIdx.x;
    if (e >= d.nelem) return;
    const size_t E = d.nelem;
    const int4 c = d.conn[e];
    // The spin (fields.cxx:483-504) and the next strain rate
    // (fields.cxx:193-241) of the same velocities and gradients share
    // their products V_i,a dN_i/db.  Both sum 0.5 (bracket) over the four
    // nodes; scaling by 0.5 is exact and commutes with rounding, so 0.5
    // times the sum of the brackets equals the reference's sum bit for
    // bit (for terms above the subnormal range).  A sum's first addition,
    // 0 + x, is an integer select (sf::add0).
    double D[6], u[3];
    {
        uint32_t far = 0;
        bool rare = false;
        double t[3];
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
            const int n = i == 0 ? c.x : i == 1 ? c.y : i == 2 ? c.z : c.w;
            const double *gp = d.shp + (size_t)i * E + e;
            const Op v0 = unpack(d.vx[n], far), v1 = unpack(d.vy[n], far), v2 = unpack(d.vz[n], far);
            Op g[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) g[k] = unpack(gp[4 * k * E], far);
            const double xx = prod(v0, g[0]), yy = prod(v1, g[1]), zz = prod(v2, g[2]);
            double tp[3], um[3];
            // (one pair of the three on the integer pipes: E-A takes 861 us on
            // 2.4M elements with none, 830 with one, 833 with two, 858 with all)
            const double xy = prod(v0, g[1]), yx = prod(v1, g[0]), xz = prod(v0, g[2]), zx = prod(v2, g[0]);
            tp[0] = xy + yx;
            um[0] = xy - yx;
            tp[1] = xz + zx;
            um[1] = xz - zx;
            sf::sum_diff(prod(v1, g[2]), prod(v2, g[1]), tp[2], um[2], rare);
            if (i == 0) {
                D[0] = sf::add0(xx);
                D[1] = sf::add0(yy);
                D[2] = sf::add0(zz);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    t[k] = sf::add0(tp[k]);
                    u[k] = sf::add0(um[k]);
                }
            } else {
                D[0] += xx;
                D[1] += yy;
                D[2] += zz;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    t[k] += tp[k];
                    u[k] += um[k];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) D[3 + k] = sf::half(t[k]);
        if (rare || !sf::in_range(far)) {
            double r[9];
            ea_rates_exact(d, e, r);
#pragma unroll
            for (int k = 0; k < 6; ++k) D[k] = r[k];
#pragma unroll
            for (int k = 0; k < 3; ++k) u[k] = 2 * r[6 + k];
        }
    }
    if (PARTS & kRates) store6(out, E, e, D);
    if (PARTS & kDvoldt) d.c_trdv[e] = sf::mul(tr3(D), d.vol[e]);
    // rotate_stress (fields.cxx:419-433) with u = 2 w, twice the spin:
    // powers of two move through the products and sums exactly (the
    // operands are in range), so dt inc is dt (sum with u) for the normal
    // components, where the reference has 2 s_ab w, and (dt / 2) (sum
    // with u) for the others
    if (!(PARTS & (kRotate | kStepRotate)) || ((PARTS & kStepRotate) && !(d.K->rheol & 1))) return;
    uint32_t farw = 0;
    const Op w3 = unpack(u[0], farw), w4 = unpack(u[1], farw), w5 = unpack(u[2], farw);
    const double dt = (PARTS & kStepRotate) ? d.clk->step_dt : d.clk->dt;
    const Op odt = unpack(dt, farw), hdt = half_op(odt);
#pragma unroll 1
    for (int f = 0; f < 2; ++f) {
        double *arr = f ? d.strain : d.stress;
        double s[6];
        load6(arr, E, e, s);
        uint32_t far = farw;
        Op o[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) o[k] = unpack(s[k], far);
        const double p3 = prod(o[3], w3), p4 = prod(o[4], w4), p5 = prod(o[5], w5);
        s[0] += prod(odt, unpack(-p3 - p4, far));
        s[1] += prod(odt, unpack(p3 - p5, far));
        s[2] += prod(odt, unpack(p4 + p5, far));
        s[3] += prod(hdt, unpack(prod(o[0], w3) - prod(o[1], w3) - prod(o[4], w5) - prod(o[5], w4), far));
        s[4] += prod(hdt, unpack(prod(o[0], w4) - prod(o[2], w4) + prod(o[3], w5) - prod(o[5], w3), far));
        s[5] += prod(hdt, unpack(prod(o[1], w5) - prod(o[2], w5) + prod(o[3], w4) + prod(o[4], w3), far));
        if (sf::in_range(far))
            store6(arr, E, e, s);
        else
            ea_rotate_exact(d, e, arr, dt, 0.5 * u[0], 0.5 * u[1], 0.5 * u[2]);
    }
}

// ---- conduction -------------------------------------------------------------------

static __device__ __noinline__ void ea_conduction_exact(const Dev &d, int e, double kv)
{
    const size_t E = d.nelem;
    double Tn[4], tr[4], dx[4], dy[4], dz[4];
    load_shp(d, e, dx, dy, dz);
    load_nodal4(d.T, d.conn[e], Tn);
    conduction(dx, dy, dz, Tn, kv, tr);
    for (int i = 0; i < 4; ++i) d.tmp[i * E + e] = tr[i];
}

// the conduction vector (fields.cxx:130-143) tr[i] = kv sum_j
// (gradNi.gradNj) T_j.  gradNi.gradNj and gradNj.gradNi round
// identically (the products commute and are summed in the same
// order), so the 10 distinct dot products are formed once: those of
// pairs go through shared memory, a node's own stays in its row.  The rows
// are unrolled (190 -> 174 us for 2.4M elements; the pairs too: 175; the other
// kernels' loops over nodes unrolled: geometry 229 -> 289, E-C 212 -> 259, for
// the spills and the longer code).
__global__ void __launch_bounds__(kEaBlock, 8) k_ea_conduction(Dev d, int e0)
{
    using sf::Op;
    using sf::prod;
    using sf::unpack;
    __shared__ double s_col[18 * kEaBlock];       // the gradients, then the dot products of pairs 01 02 03 12 13 23
    __shared__ uint32_t s_ex[12 * kEaBlock];
    const int e = e0 + blockIdx.x * kEaBlock + threadIdx.x;
    if (e >= d.nelem) return;
    const size_t E = d.nelem;
    const int4 c = d.conn[e];
    double *sg = s_col + threadIdx.x, *sd = sg + 12 * kEaBlock;
    uint32_t *sx = s_ex + threadIdx.x;
    uint32_t far = 0;
#pragma unroll
    for (int k = 0; k < 12; ++k) put_op(sg + k * kEaBlock, sx + k * kEaBlock, unpack(d.shp[k * E + e], far));   // 4 k + i: dN_i/dx_k
#pragma unroll 1
    for (int q = 0; q < 6; ++q) {
        const int i = (0x211000 >> (4 * q)) & 3, j = (0x332321 >> (4 * q)) & 3;
        double p[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
            p[k] = prod(get_op(sg + (4 * k + i) * kEaBlock, sx + (4 * k + i) * kEaBlock),
                          get_op(sg + (4 * k + j) * kEaBlock, sx + (4 * k + j) * kEaBlock));
        sd[q * kEaBlock] = p[0] + p[1] + p[2];
    }
    const double kv = sf::mul(d.K->M.mix[d.mix[e]].k, d.vol[e]);
    const Op okv = unpack(kv, far);
    double Tn[4];
    load_nodal4(d.T, c, Tn);
    Op oT[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) oT[j] = unpack(Tn[j], far);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        // the pair number of (i, j), j = 0..3 (the diagonal's nibble unused)
        const unsigned pairs = i == 0 ? 0x2100u : i == 1 ? 0x4300u : i == 2 ? 0x5031u : 0x0542u;
        double p[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const Op g = get_op(sg + (4 * k + i) * kEaBlock, sx + (4 * k + i) * kEaBlock);
            p[k] = prod(g, g);
        }
        const double dii = p[0] + p[1] + p[2];
        double diffusion = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double off = sd[((pairs >> (4 * j)) & 15) * kEaBlock];
            const double pj = prod(unpack(i == j ? dii : off, far), oT[j]);
            diffusion = j == 0 ? sf::add0(pj) : diffusion + pj;
        }
        d.tmp[(size_t)i * E + e] = prod(unpack(diffusion, far), okv);
    }
    if (!sf::in_range(far)) ea_conduction_exact(d, e, kv);
}

// ---- E-C: NMD correction, element force vectors ---------------------------------

static __device__ __noinline__ void ec_force_exact(const Dev &d, int e)
{
    double s[6];
    load6(d.stress, d.nelem, e, s);
    force_elem_body(d, e, d.conn[e], s);
}

// 12 blocks of 128 per SM (8: 349 us on 3.84M elements, 10: 332, 12: 330)
// NMD: E-C; without it the force vectors alone (update_force's element half)
template <bool NMD>
__global__ void __launch_bounds__(kEaBlock, 12) k_fe_c(Dev d)
{
    using sf::Op;
    using sf::prod;
    using sf::unpack;
    const int e = blockIdx.x * kEaBlock + threadIdx.x;
    if (e >= d.nelem) return;
    const size_t E = d.nelem;
    const Consts &K = *d.K;
    const int4 c = d.conn[e];
    double s[6];
    load6(d.stress, E, e, s);
    if (NMD) {
        double a[4];
        load_nodal4(d.ntmp, c, a);
        double dpe = sf::add0(a[0]);            // 0 + a0, then the rest; / 4, / 3
        for (int i = 1; i < 4; ++i) dpe += a[i];
        const double ddp = sf::div3(-d.dp[e] + sf::quarter(dpe));
        for (int i = 0; i < 3; ++i) {
            s[i] += ddp;
            d.stress[i * E + e] = s[i];
        }
    }
    double buoy = 0;
    if (K.gravity != 0) {
        double Tn[4];
        load_nodal4(d.T, c, Tn);
        buoy = sf::quarter(sf::mul(mat_rho(K.M, K.M.mix[d.mix[e]], elem_mean4(Tn[0], Tn[1], Tn[2], Tn[3])), K.gravity));
    }
    // fields.cxx:321-346, a node of the element per turn
    uint32_t far = 0;
    Op o[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) o[k] = unpack(s[k], far);
    const Op ov = unpack(d.vol[e], far);
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const Op gx = unpack(d.shp[(size_t)i * E + e], far), gy = unpack(d.shp[(size_t)(4 + i) * E + e], far),
                 gz = unpack(d.shp[(size_t)(8 + i) * E + e], far);
        const double fx = prod(o[0], gx) + prod(o[3], gy) + prod(o[4], gz);
        const double fy = prod(o[3], gx) + prod(o[1], gy) + prod(o[5], gz);
        const double fz = prod(o[4], gx) + prod(o[5], gy) + prod(o[2], gz) + buoy;
        d.tmp[(size_t)i * E + e] = prod(unpack(fx, far), ov);
        d.tmp[(size_t)(4 + i) * E + e] = prod(unpack(fy, far), ov);
        d.tmp[(size_t)(8 + i) * E + e] = prod(unpack(fz, far), ov);
    }
    if (!sf::in_range(far)) ec_force_exact(d, e);
}

}  // namespace des
