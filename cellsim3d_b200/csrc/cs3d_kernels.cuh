// cs3d_kernels.cuh -- the per-timestep kernels of libcs3d.so (sm_100a).
//
// One CTA of 192 threads (six warps) owns one cell at a time and draws the
// next one from a counter; thread i owns node i.  The cell's 180 positions
// and velocities are staged in shared memory; the 540 bond angles are
// evaluated once each (the reference evaluates every angle twice, from the
// vertex and from the arm end) and their arm-end forces are gathered from
// shared memory in the reference's summation order.
//
// The neighbour list (per cell: candidate cells; per node: the nodes of
// candidate cells within the list radius, as slot << 8 | node) is rebuilt
// on the device whenever the accumulated displacement bound reaches the
// skin, or after a division.  Every step the reference's own contact
// predicates -- stale grid bin of the node, stale bounding box of the
// neighbour cell, strict (conservative) and non-strict (dissipative)
// cut-offs in float -- are evaluated on every list entry, so the contact
// pairs are exactly the reference's.  Partner nodes are read straight from
// global memory: the few hundred partners of a cell stay in L1/L2.
//
// Times in the comments below that name 100,000 packed cells are averages of
// steps 11 to 40 from a jittered fcc lattice at volume fraction 0.5, where a
// node has at most 9 entries; they rise as the cells settle against each other
// (steps 201 to 230, up to 18 entries: S1 1.62 -> 2.69 ms, S2 0.53 -> 0.66 ms).
#pragma once
#include "cs3d_dev.cuh"

namespace cs3d {

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ float3 f3(float4 a) { return make_float3(a.x, a.y, a.z); }

template <typename T>
__device__ __forceinline__ T warp_sum(T v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_min(float v)
{
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ void atomic_or_err(InstState *st, unsigned bits) { atomicOr(&st->err, bits); }

// Block-wide exclusive scan (NT threads, NT a multiple of 32); wsum[32].
template <int NT>
__device__ __forceinline__ int block_excl_scan(int v, int *wsum, int &total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int s = lane < NT / 32 ? wsum[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        wsum[lane] = s;
    }
    __syncthreads();
    const int r = (wid > 0 ? wsum[wid - 1] : 0) + x - v;
    total = wsum[NT / 32 - 1];
    __syncthreads();
    return r;
}


// Partner data: read-only for the length of a step's own kernel, but written
// by other CTAs between the phases of k_steps (COOP), which must not read it
// through the read-only path.
template <bool COOP>
__device__ __forceinline__ float4 ld_partner(const float4 *p)
{
    return COOP ? *p : __ldg(p);
}

// Active cells: the identity for a single instance, else the work table.
__device__ __forceinline__ int n_work(const Dev &d) { return d.single ? d.st[0].n : *d.work_n; }
__device__ __forceinline__ int cell_of(const Dev &d, int w) { return d.single ? w : d.work[w]; }
__device__ __forceinline__ int inst_of(const Dev &d, int a) { return d.single ? 0 : d.cell_inst[a]; }

// Cells of a phase dealt out to the CTAs one by one: a CTA begins with the
// cell of its index and draws the next one while it works.  A cell next to a
// division takes three times as long as another, so that with a fixed stride
// the last CTA of S1 ended 60 % after the mean one (2500 growing cells); S1
// takes the newest cells first, a further 2 % of the step.
// next[]: two words of the CTA's shared memory; the counter is zero at the
// start of the phase (step_begin).
struct Dealer {
    int *counter, *next;
    int w, turn;

    __device__ __forceinline__ Dealer(int *counter_, int *next_) : counter(counter_), next(next_), w(blockIdx.x), turn(0) {}
    // at the start of a cell's work, before a barrier
    __device__ __forceinline__ void draw()
    {
        if (threadIdx.x == 0) next[turn] = (int)gridDim.x + atomicAdd(counter, 1);
    }
    // after a barrier that follows draw()
    __device__ __forceinline__ void advance()
    {
        w = next[turn];
        turn ^= 1;
    }
};
enum { DEAL_S1, DEAL_S2, DEAL_LISTS, DEALS };

// Kick of the split velocity Verlet with the reference's mixed precision:
// the float sum is scaled by the double literal 0.5 and divided by the mass
// in double, then stored as float (src/propagate.cu:698-705, 721-723, 732-734).
// a / m, the integrator's division by the particle mass, correctly rounded
// as the IEEE double division the reference evaluates: with im = 1/m
// correctly rounded (set on the host), q = a * im is within one ulp of a/m,
// the remainder a - q m is exact in one FMA, and q + (a - q m) im rounded
// once is the correctly rounded quotient (Markstein's theorem); three FP64
// operations instead of a full division.  Checked against the IEEE division
// on 1.03e9 operand pairs of the integrator's shapes and random masses.
__device__ __forceinline__ double div_m(double a, const InstParams &P)
{
    const double q = a * P.inv_m;
    return fma(fma(-q, P.mass_d, a), P.inv_m, q);
}

// v + 0.5 fsum / m (double arithmetic, stored as float), src/propagate.cu:681-736.
__device__ __forceinline__ float kick(float v, float fsum, const InstParams &P)
{
    return (float)((double)v + div_m(0.5 * (double)fsum, P));
}

// Langevin random force (src/propagate.cu:668-678): rand_scale_factor times
// three standard normals per node and step.  The reference draws them from
// per-node curand XORWOW states; here they come from the counter-based
// Philox4x32-10 generator (Salmon, Moraes, Dror and Shaw, "Parallel random
// numbers: as easy as 1, 2, 3", SC'11; round multipliers and Weyl key
// increments as published there) keyed by the instance's rand_seed and
// counted by (node, step), with the Box-Muller transform on 24-bit uniforms.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const unsigned hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        const unsigned hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}

__device__ __forceinline__ float unit_open(unsigned r)
{
    return ((float)(r >> 8) + 0.5f) * (1.0f / 16777216.0f);  // (0, 1), exact in float
}

__device__ __forceinline__ float3 random_force(const InstParams &P, int a, int i, int step)
{
    const unsigned node = (unsigned)((a - P.base) * SLOTS + i);
    const uint4 r = philox4x32_10(make_uint4(node, (unsigned)step, 0u, 0u), make_uint2(P.rseed, 0x2545F491u));
    const float ra = sqrtf(-2.0f * logf(unit_open(r.x))), ta = 6.28318531f * unit_open(r.y);
    const float rb = sqrtf(-2.0f * logf(unit_open(r.z))), tb = 6.28318531f * unit_open(r.w);
    return make_float3(P.rscale * (ra * cosf(ta)), P.rscale * (ra * sinf(ta)), P.rscale * (rb * cosf(tb)));
}

// 1/sqrt(x) and 1/x of positive doubles: the hardware's FP64
// approximations (rsqrt.approx.ftz.f64, rcp.approx.ftz.f64; relative error
// below 1e-6 on B200) refined by one Newton step in FP64.  Measured over
// 1e-4..1e4 on B200: relative error below 1.3e-12, far below what the forces
// need (their float rounding is 6e-8), with no float conversions.  The
// arguments are never subnormal (squared lengths of at least ~1e-8).
__device__ __forceinline__ double rsqrt_nr(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y * (1.5 - 0.5 * x * y * y);
}
__device__ __forceinline__ double rcp_nr(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r * (2.0 - x * r);
}

// Bond-angle term for one angle at a vertex with arms P (to the p-end node)
// and Q (to the q-end node); Fp/Fq are GetAngleForce(P, Q) and
// GetAngleForce(Q, P) of src/propagate.cu:26-60 (k = 1000, :335), with the
// same 1e-3 regularisers.  The force is proportional to theta - theta0, a
// difference of two angles near 2 rad whose float rounding alone (1.2e-7)
// would exceed the 1e-5 relative force bar, so it is formed without
// rounding theta.  u = cos(theta) (the reference's regularised ratio) is
// formed in FP64; with c0, s0 = cos, sin of theta0 in FP64,
//   sin(dth / 2) = (c0 - u) / (2 sin(theta0 + dth / 2)),   dth = theta - theta0.
// A float estimate of dth from acosf is refined by one Newton step of this
// equation in FP64 (sin/cos of dth/2 by their Taylor series, |dth/2| < 0.4
// for |dth/2| up to ~1.2 rad), which leaves dth accurate to ~1e-12.
__device__ __forceinline__ void sincos_small(double x, double &s, double &c)
{
    const double x2 = x * x;
    s = x * (1.0 + x2 * (-1.0 / 6 + x2 * (1.0 / 120 + x2 * (-1.0 / 5040 + x2 * (1.0 / 362880 +
            x2 * (-1.0 / 39916800 + x2 * (1.0 / 6227020800.0 - x2 / 1307674368000.0)))))));
    c = 1.0 + x2 * (-0.5 + x2 * (1.0 / 24 + x2 * (-1.0 / 720 + x2 * (1.0 / 40320 + x2 * (-1.0 / 3628800 +
            x2 * (1.0 / 479001600 + x2 * (-1.0 / 87178291200.0 + x2 / 20922789888000.0)))))));
}

// One arm of a vertex: the exact FP64 difference p of two node positions,
// its squared length, length, and inverse length and its square (from one rsqrt).
struct Arm {
    double x, y, z, r2, len, ir2, ir;
};

__device__ __forceinline__ Arm make_arm(const double3 &to, const double3 &from)
{
    Arm a;
    a.x = to.x - from.x;
    a.y = to.y - from.y;
    a.z = to.z - from.z;
    a.r2 = a.x * a.x + a.y * a.y + a.z * a.z;
    const double r = rsqrt_nr(a.r2);
    a.len = a.r2 * r;
    a.ir2 = r * r;
    a.ir = r;
    return a;
}

// The angle between arms p and q: GetAngleForce(P, Q) (Fp) and
// GetAngleForce(Q, P) (Fq).  |p||q| is the product of the two lengths, as the
// reference forms it (sqrtf(ri_2) * sqrtf(rk_2)).
__device__ __forceinline__ void angle_term(const Arm &p, const Arm &q, float th0f, double c0, double s0, double3 &Fp,
                                           double3 &Fq)
{
    const double idk = p.x * q.x + p.y * q.y + p.z * q.z;
    const double u = idk * rcp_nr(p.len * q.len + 1e-3);
    // float estimate, then one Newton step on g(h) = sin(h) sin(theta0 + h) - (c0 - u)/2, h = dth/2
    double h = 0.5 * (double)(acosf((float)u) - th0f);
    double sh, ch;
    sincos_small(h, sh, ch);
    const double s1 = s0 * ch + c0 * sh, c1t = c0 * ch - s0 * sh;  // sin, cos of theta0 + h
    const double g = sh * s1 - 0.5 * (c0 - u);
    const double dg = ch * s1 + sh * c1t;                            // d/dh of sin(h) sin(theta0 + h)
    h -= g * rcp_nr(dg);
    const double dth = 2.0 * h;
    const double c1 = -rsqrt_nr(p.r2 * q.r2 - idk * idk + 1e-3);
    const double f = -1000.0 * c1 * dth;
    const double cp = idk * p.ir2, cq = idk * q.ir2;
    Fp = make_double3(f * (q.x - cp * p.x), f * (q.y - cp * p.y), f * (q.z - cp * p.z));
    Fq = make_double3(f * (p.x - cq * q.x), f * (p.y - cq * q.y), f * (p.z - cq * q.z));
}

// Shared per-CTA data of the contact sweep: candidate cells with their stale
// boxes and stale insertion bin ranges.
struct SlotData {
    int cell[MAXC];
    float4 lo[MAXC], hi[MAXC];   // w: lowest, highest bin along z (int bits)
    int4 range[MAXC];            // lowest and highest bin along x and y
    float mn[3];
    int div[3];
};

// Candidate cells and stale grid of cell a (independent loads only, so they
// overlap with the caller's own-node loads; a __syncthreads() follows).
__device__ __forceinline__ void slots_load(const Dev &d, int a, const InstState *st, int par, SlotData &sd)
{
    const int t = threadIdx.x;
    // read in full whatever the count, so that no load waits for another
    // (entries past the count are never used)
    if (t < MAXC) sd.cell[t] = d.cand[(size_t)a * MAXC + t];
    // thread 0 has the drawing of the next cell to do
    if (t >= 160 && t < 163) {
        const int q = t - 160;
        const int *mm = st->mm[par];
        float mn = fminf(o2f(mm[2 * q]), 1.0e8f);
        float mx = fmaxf(o2f(mm[2 * q + 1]), -1.0e8f);
        sd.mn[q] = mn;
        sd.div[q] = grid_div(mn, mx);
    }
}

// Stale boxes / insertion ranges of the candidates (slots_load visible).
__device__ __forceinline__ void slots_boxes(const Dev &d, const InstParams &P, int par, SlotData &sd, int nc)
{
    int t = threadIdx.x;
    if (t < nc) {
        int c = sd.cell[t];
        float4 lo = d.aabb[par][2 * c], hi = d.aabb[par][2 * c + 1];
        int st, en;
        int4 rg;
        bin_range_axis(lo.x, hi.x, P.ra, sd.mn[0], sd.div[0], rg.x, rg.y);
        bin_range_axis(lo.y, hi.y, P.ra, sd.mn[1], sd.div[1], rg.z, rg.w);
        bin_range_axis(lo.z, hi.z, P.ra, sd.mn[2], sd.div[2], st, en);
        lo.w = __int_as_float(st);
        hi.w = __int_as_float(en);
        sd.lo[t] = lo;
        sd.hi[t] = hi;
        sd.range[t] = rg;
    }
}

// The reference's cell-level contact filter for one node, cached per
// candidate slot (the entries are sorted by slot): the node's stale grid bin
// lies in the slot cell's stale insertion range (the cell is in the node's
// bin list, src/propagatebound.cu:209-256) and the node is within the
// cut-off of the slot cell's stale box (src/propagate.cu:382-392).
struct NodeBins {
    int b0, b1, b2;   // the node's stale grid bin
};

__device__ __forceinline__ NodeBins node_bins(const SlotData &sd, float3 x)
{
    return {node_bin_axis(x.x, sd.mn[0], sd.div[0]), node_bin_axis(x.y, sd.mn[1], sd.div[1]),
            node_bin_axis(x.z, sd.mn[2], sd.div[2])};
}

__device__ __forceinline__ bool slot_ok(const SlotData &sd, const InstParams &P, float3 x, NodeBins nb, int s)
{
    const int4 g = sd.range[s];
    const float4 lo = sd.lo[s], hi = sd.hi[s];
    return nb.b0 >= g.x && nb.b0 <= g.y && nb.b1 >= g.z && nb.b1 <= g.w && nb.b2 >= __float_as_int(lo.w) &&
           nb.b2 <= __float_as_int(hi.w) && aabb_keep(lo, hi, x.x, x.y, x.z, P.ra2);
}

// ---------------------------------------------------------------------------
// The contact sweep of S1 shares a warp's entries among its lanes.  A node has
// one or two entries on average and the nodes next to another cell five to
// forty: with a lane walking its own node's entries, a warp took as many
// rounds as its busiest node has entries and most lanes waited.  Here the
// entries of the warp's 32 nodes (eight of each node at a time, the first of
// every node, then the second, ...) are laid out back to back, a round takes
// 32 of them, one to a lane, and the owners then add up the results of their
// entries in entry order, so that a node's sums do not depend on the sharing.
// An owner seldom has more than two entries in a round, and adds them to its
// running force exactly as a lane walking its own entries would.  S1 of 100,000
// packed cells 2.01 -> 1.86 ms, of 3000 growing ones 97 -> 85 us (with an
// owner's entries side by side, up to 32 to a round, 1.89 ms and 95 us); S2's
// sweep, two loads and three additions a pair, is slower this way (0.62 ->
// 0.65 ms).
// ---------------------------------------------------------------------------
constexpr int EPRE = 8;    // entries of a node laid out at a time

struct alignas(16) SweepSmem {
    double res[7][32];           // results of a round: force over distance, distance, velocity difference
    uint32_t item[EPRE * 32];    // owner lane << 16 | slot << 8 | node
    unsigned own[32];            // results of the round that are the node's
};

// S1 contact sweep of the warp's nodes (i: this lane's): conservative contact
// force (strict cut-off, src/propagate.cu:406-442) added to F, sum of the
// velocity differences v_i - v_j of the dissipative pairs (non-strict cut-off,
// src/propagate.cu:600-656) in vsum (its tangential part is taken once, by
// tangential()).  Lists the dissipative pairs for S2 (positions do not change
// before S2) and returns their number.
// Partner positions and velocities are read from global memory (L1/L2
// resident: the partners of a cell are a few hundred nodes).
template <bool COOP>
__device__ __forceinline__ int sweep_s1(const Dev &d, const InstParams &P, const SlotData &sd, SweepSmem &ss, int a,
                                        int i, float3 x, float3 v, int ne, const uint32_t (&pre)[EPRE / 2], double &FX,
                                        double &FY, double &FZ, double3 &vsum)
{
    const int lane = i & 31;
    const int most = __reduce_max_sync(0xffffffffu, ne);
    if (most == 0) return 0;   // uniform in the warp
    const uint16_t *ep = d.ent + (size_t)a * MAXE * SLOTS + i;
    uint16_t *dl = d.dlist + (size_t)a * MAXD * SLOTS + i;
    const NodeBins nb = node_bins(sd, x);
    const unsigned below = (1u << lane) - 1u;
    uint32_t w[EPRE / 2] = {pre[0], pre[1], pre[2], pre[3]};
    int nd = 0;
    ss.own[lane] = 0u;
    for (int k0 = 0; k0 < most; k0 += EPRE) {
        int m = 0;
#pragma unroll
        for (int k = 0; k < EPRE; ++k) {
            const bool has = k0 + k < ne;
            const unsigned b = __ballot_sync(0xffffffffu, has);
            if (has)
                ss.item[m + __popc(b & below)] = (unsigned)lane << 16 | (k & 1 ? w[k / 2] >> 16 : w[k / 2] & 0xffffu);
            m += __popc(b);
        }
        __syncwarp();
        // the next eight, in flight during the rounds
        if (k0 + EPRE < most) {
#pragma unroll
            for (int k = 0; k < EPRE; ++k) {
                const int q = k0 + EPRE + k;
                const unsigned e = q < ne ? ep[(size_t)q * SLOTS] : 0u;
                w[k / 2] = k & 1 ? w[k / 2] | e << 16 : e;
            }
        }
        for (int b = 0; b < m; b += 32) {
            const bool act = b + lane < m;
            const unsigned it = act ? ss.item[b + lane] : (unsigned)lane << 16;
            const int o = it >> 16, s = (it >> 8) & 255u, j = it & 255u;
            const float3 xo = make_float3(__shfl_sync(0xffffffffu, x.x, o), __shfl_sync(0xffffffffu, x.y, o),
                                          __shfl_sync(0xffffffffu, x.z, o));
            const float3 vo = make_float3(__shfl_sync(0xffffffffu, v.x, o), __shfl_sync(0xffffffffu, v.y, o),
                                          __shfl_sync(0xffffffffu, v.z, o));
            const NodeBins no = {__shfl_sync(0xffffffffu, nb.b0, o), __shfl_sync(0xffffffffu, nb.b1, o),
                                 __shfl_sync(0xffffffffu, nb.b2, o)};
            bool pass = act && slot_ok(sd, P, xo, no, s);
            const int id = pass ? sd.cell[s] * SLOTS + j : 0;
            float4 xj = make_float4(0.f, 0.f, 0.f, 0.f), vj = xj;
            if (pass) {
                xj = ld_partner<COOP>(&d.X[id]);
                vj = ld_partner<COOP>(&d.V[id]);
            }
            const float r2 = r2_ref(__fsub_rn(xo.x, xj.x), __fsub_rn(xo.y, xj.y), __fsub_rn(xo.z, xj.z));
            pass = pass && !(r2 > P.ra2);
            if (pass) {
                atomicOr(&ss.own[o], 1u << lane);
                if (d.record_pairs) {
                    const unsigned long long slot = atomicAdd(d.n_pairs, 1ull);
                    if ((long long)slot < d.pair_cap)
                        d.pairs[slot] = make_int4((a << 8) | (i - lane + o), ((id / SLOTS) << 8) | (id % SLOTS),
                                                  r2 < P.ra2 ? 3 : 2, 0);
                }
                // distance in FP64 from the exact difference of the float
                // positions: (rr - R) cancels for stiff repulsion
                const double ex = (double)xo.x - xj.x, ey = (double)xo.y - xj.y, ez = (double)xo.z - xj.z;
                const double R2 = ex * ex + ey * ey + ez * ez;
                const double iR = rsqrt_nr(R2);
                const double R = R2 * iR;
                double k = 0.0;
                if (r2 < P.ra2) {
                    if (R < (double)P.ra) k += -(double)P.asE * ((double)P.ra - R) * iR;
                    if (R <= (double)P.rr) k += (double)P.rsE * ((double)P.rr - R) * iR;
                }
                ss.res[0][lane] = k;
                ss.res[1][lane] = ex; ss.res[2][lane] = ey; ss.res[3][lane] = ez;
                // a pair with a node that is no number counts for the friction only
                // and must not get into F: k = 0 times 0 (the owner leaving out pairs
                // with k = 0 makes the steps of 8 cells 1.3 % slower, zeros chosen
                // before the stores S1 of packed cells 1 %)
                if (r2 != r2) ss.res[1][lane] = ss.res[2][lane] = ss.res[3][lane] = 0.0;
                // velocity differences of floats are exact in FP64
                ss.res[4][lane] = (double)vo.x - vj.x;
                ss.res[5][lane] = (double)vo.y - vj.y;
                ss.res[6][lane] = (double)vo.z - vj.z;
            }
            __syncwarp();
            unsigned mine = ss.own[lane];
            ss.own[lane] = 0u;
            while (mine) {
                const int q = __ffs(mine) - 1;
                mine &= mine - 1u;
                if (nd < MAXD) dl[(size_t)nd * SLOTS] = (uint16_t)ss.item[b + q];
                ++nd;
                const double k = ss.res[0][q];
                FX = fma(k, ss.res[1][q], FX);
                FY = fma(k, ss.res[2][q], FY);
                FZ = fma(k, ss.res[3][q], FZ);
                vsum.x += ss.res[4][q]; vsum.y += ss.res[5][q]; vsum.z += ss.res[6][q];
            }
            __syncwarp();
        }
    }
    return nd;
}

constexpr int SB = 4;      // pairs whose partner loads are in flight together

// S2 sweep: sum of the velocity differences over the dissipative pairs found
// by S1 (their list, in column layout), with the velocities after the half
// kicks; tangential() takes its tangential part.
template <bool COOP>
__device__ __forceinline__ double3 sweep_s2(const Dev &d, const int *cell, int a, int i, float3 v, int nd)
{
    const uint16_t *dl = d.dlist + (size_t)a * MAXD * SLOTS + i;
    double3 vt = make_double3(0.0, 0.0, 0.0);
    for (int k0 = 0; k0 < nd; k0 += SB) {
        unsigned e[SB];
#pragma unroll
        for (int q = 0; q < SB; ++q) e[q] = k0 + q < nd ? dl[(size_t)(k0 + q) * SLOTS] : 0xffffu;
        float4 vj[SB];
#pragma unroll
        for (int q = 0; q < SB; ++q)
            vj[q] = e[q] != 0xffffu ? ld_partner<COOP>(&d.Vb[cell[e[q] >> 8] * SLOTS + (int)(e[q] & 255u)])
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int q = 0; q < SB; ++q) {
            if (e[q] == 0xffffu) continue;
            vt.x += (double)v.x - vj[q].x;
            vt.y += (double)v.y - vj[q].y;
            vt.z += (double)v.z - vj[q].z;
        }
    }
    return vt;
}

// Tangential part of the friction sum, src/propagate.cu:558-656: the
// reference adds v_ij - (v_ij . n) n over the dissipative pairs of node i, with
// n the unit normal of the surface at i, sign * unit((x_N2 - x_N1) x (x_N3 -
// x_N1)).  The projection is linear in v_ij, so the sweeps sum the velocity
// differences alone (S) and this applies it once: S - (S . n) n.  The normal
// is formed in FP64 from exact differences of the float positions.
__device__ __forceinline__ double3 as_d3(const float4 &a) { return make_double3(a.x, a.y, a.z); }

// xs: the cell's positions.
__device__ __forceinline__ double3 tangential(const float4 *xs, int n0, int n1, int n2, float sgn, double3 S)
{
    const double3 p0 = as_d3(xs[n0]), p1 = as_d3(xs[n1]), p2 = as_d3(xs[n2]);
    const double ax = p1.x - p0.x, ay = p1.y - p0.y, az = p1.z - p0.z;
    const double bx = p2.x - p0.x, by = p2.y - p0.y, bz = p2.z - p0.z;
    const double cx = ay * bz - az * by, cy = az * bx - ax * bz, cz = ax * by - ay * bx;
    const double s = (double)sgn * rsqrt_nr(cx * cx + cy * cy + cz * cz);
    const double nx = s * cx, ny = s * cy, nz = s * cz;
    const double dn = S.x * nx + S.y * ny + S.z * nz;
    return make_double3(S.x - dn * nx, S.y - dn * ny, S.z - dn * nz);
}

// Dissipative force, src/propagate.cu:546-658: bond damping with the three
// neighbours, tangential friction sum vt, viscous drag, on the cell's
// velocities vs.  FP64: the damping
// term is a sum of velocity differences that can cancel.
__device__ __forceinline__ float3 dis_force(const InstParams &P, const float4 *vs, int i, int n0, int n1, int n2,
                                           double3 vt)
{
    const double3 v = as_d3(vs[i]);
    double dx = 0.0, dy = 0.0, dz = 0.0;
    const int nbr[3] = {n0, n1, n2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double3 vn = as_d3(vs[nbr[k]]);
        dx += v.x - vn.x; dy += v.y - vn.y; dz += v.z - vn.z;
    }
    const double gi = P.gint, ge = P.gext, go = P.go;
    return make_float3((float)(-gi * dx - ge * vt.x - go * v.x), (float)(-gi * dy - ge * vt.y - go * v.y),
                       (float)(-gi * dz - ge * vt.z - go * v.z));
}

// PressureUpdate, src/PressureKernels.cu:4-40, for the step `step` being
// taken: with variable stiffness, from step phase_count on a cell whose
// stiffness is not stiffness1 has pressure 0; every other cell grows by the
// growth rate up to maxPressure.  The reference runs it after Integrate and
// ForwardTime and before the forces; here S1 applies it to its cell before
// the pressure force (nothing in between reads the pressure), so that the
// stored pressures are always those of the last finished step.
__device__ __forceinline__ float pressure_update(const Dev &d, const InstParams &P, int a, int step)
{
    const float p = d.press[a];
    if (P.diffE && step >= P.phase && d.E[a] != P.stiff1) return 0.0f;
    if (p < P.maxp) return p + P.growth;
    return p;
}

// ---------------------------------------------------------------------------
// K1: first half kick + drift of a step (Integrate + ForwardTime,
// src/propagate.cu:681-763).  The step's PressureUpdate is S1's.
// ---------------------------------------------------------------------------
// One cell, called by the whole block (it synchronises).
__device__ __forceinline__ void integrate_cell(const Dev &d, int a, float *smax)
{
    {
        int inst = inst_of(d, a);
        const InstParams &P = d.prm[inst];
        int i = threadIdx.x;
        float disp = 0.0f;
        if (i < NODES) {
            size_t g = (size_t)a * SLOTS + i;
            float4 x = d.X[g], v = d.V[g], fc = d.FC[g], fd = d.FD[g];
            const float dt = P.dt;
            float sx = __fadd_rn(__fmul_rn(dt, fc.x), __fmul_rn(dt, fd.x));
            float sy = __fadd_rn(__fmul_rn(dt, fc.y), __fmul_rn(dt, fd.y));
            float sz = __fadd_rn(__fmul_rn(dt, fc.z), __fmul_rn(dt, fd.z));
            if (P.rands) {  // + sqrt(dt) Fr of the previous step
                const float4 fr = d.FR[g];
                sx = __fadd_rn(sx, __fmul_rn(P.rdt, fr.x));
                sy = __fadd_rn(sy, __fmul_rn(P.rdt, fr.y));
                sz = __fadd_rn(sz, __fmul_rn(P.rdt, fr.z));
            }
            v.x = kick(v.x, sx, P);
            v.y = kick(v.y, sy, P);
            v.z = kick(v.z, sz, P);
            float4 xn = make_float4(__fmaf_rn(v.x, dt, x.x), __fmaf_rn(v.y, dt, x.y), __fmaf_rn(v.z, dt, x.z), 0.0f);
            // displacement since the last neighbour-list build
            const float4 xb = d.Xb[g];
            float ddx = xn.x - xb.x, ddy = xn.y - xb.y, ddz = xn.z - xb.z;
            disp = sqrtf(ddx * ddx + ddy * ddy + ddz * ddz);
            d.X[g] = xn;
            d.V[g] = v;
        }
        disp = warp_max(disp);
        if ((i & 31) == 0) smax[i >> 5] = disp;
        __syncthreads();
        if (i == 0) {
            float m = smax[0];
            for (int q = 1; q < SLOTS / 32; ++q) m = fmaxf(m, smax[q]);
            d.cdisp[a] = m;
            atomicMax(&d.st[inst].disp_step, __float_as_uint(m));
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(SLOTS) k_integrate(Dev d)
{
    const int W = n_work(d);
    __shared__ float smax[SLOTS / 32];
    for (int w = blockIdx.x; w < W; w += gridDim.x) integrate_cell(d, cell_of(d, w), smax);
}

// ---------------------------------------------------------------------------
// Per-step bookkeeping (one block): step counter, rebuild decision, reset of
// the accumulators that this step fills.
// ---------------------------------------------------------------------------
// Slices of the cell table of the list build: every rebuilding instance gets
// its own power-of-two range of bins (at least twice its cells), laid out
// back to back.  Whole block (NT threads), after the rebuild decisions.
template <int NT>
__device__ __forceinline__ void assign_hash_slices(const Dev &d)
{
    __shared__ int wsum[32];
    __shared__ unsigned carry;
    if (threadIdx.x == 0) carry = 0u;
    __syncthreads();
    for (int k0 = 0; k0 < d.n_inst; k0 += NT) {
        const int k = k0 + threadIdx.x;
        int size = 0;
        if (k < d.n_inst) {
            InstState *st = &d.st[k];
            int bits = 0;
            if (st->rebuild) {
                bits = 6;
                while ((1ll << bits) < 2ll * st->n) ++bits;
                for (int q = 0; q <= st->top; ++q) st->hmax[q][0] = st->hmax[q][1] = st->hmax[q][2] = 0u;
                st->top = st->n_large = st->n_giant = 0;
                size = 1 << bits;
            }
            st->hbits = bits;
        }
        int tot;
        const int off = block_excl_scan<NT>(size, wsum, tot);
        if (k < d.n_inst) d.st[k].hbase = carry + (unsigned)off;
        if (threadIdx.x == 0) carry += (unsigned)tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) *d.epoch += 1u;   // empties the table
}

template <int NT>
__device__ __forceinline__ void step_begin(const Dev &d, int par_next)
{
    __shared__ int any;
    if (threadIdx.x == 0) {
        any = 0;
        *d.n_build = 0;
        for (int q = 0; q < DEALS; ++q) d.deal[q] = 0;
        *d.div_prev = *d.div_total;   // the divisions the lists are rebuilt around
        *d.div_total = 0;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < d.n_inst; k += blockDim.x) {
        InstState *st = &d.st[k];
        const InstParams &P = d.prm[k];
        st->step += 1;
        // ds: the largest distance of any node from its anchor (Xb, its
        // position at a build).  A list built at time tb stays complete
        // while all nodes stay within skin/2 of their anchors, if it holds
        // the pairs within ra + skin + D(a) + D(b), D the largest such
        // distance at tb among the nodes of each of the two cells: a pair
        // within ra now was within ra + (skin/2 + D(a)) + (skin/2 + D(b)) at
        // tb.  Whole-instance builds (D reset to 0) use ra + skin; the 1e-3
        // slack covers float rounding.  After divisions, only the divided
        // cells (anchors reset) and the cells within the list radius of them
        // are rebuilt, unless many cells divided: a division concerns some
        // dozen cells, so that from one cell in 16 on most would be built.
        const float ds = __uint_as_float(st->disp_step);
        st->disp_step = 0u;
        if (P.sk_n > 0) {
            // the skin of the instance's population range; a change is a
            // whole-instance rebuild with the new list radius
            float want = P.skin_base;
            for (int q = 0; q < P.sk_n; ++q)
                if (st->n >= P.sk_min[q]) want = P.sk_val[q];
            if (want != P.skin) {
                InstParams *Pw = &d.prm[k];
                Pw->skin = want;
                Pw->rlist = Pw->ra + want;
                st->force_rebuild = 1;
            }
        }
        const bool by_disp = st->force_rebuild || !(2.0f * ds + 1e-3f < P.skin);
        const bool by_div = st->div_count > 0 && 16 * st->div_count > st->n;
        const bool full = by_disp || by_div;
        if (by_div && !by_disp) st->rebuilds_div += 1;
        const bool part = !full && st->div_count > 0;
        st->rebuild = full ? 2 : part ? 1 : 0;
        st->ds = full ? 0.0f : ds;
        st->force_rebuild = 0;
        st->div_count = 0;
        if (full || part) {
            if (full) st->rebuilds += 1;
            any = 1;
        }
        for (int q = 0; q < 3; ++q) {
            st->mm[par_next][2 * q] = f2o(1.0e30f);
            st->mm[par_next][2 * q + 1] = f2o(-1.0e30f);
        }
    }
    __syncthreads();
    if (any) assign_hash_slices<NT>(d);
    if (threadIdx.x == 0) {
        d.flags[0] = any;
        d.flags[1] = 0;
        *d.n_pairs = 0ull;
    }
}

__global__ void __launch_bounds__(256) k_step_begin(Dev d, int par_next)
{
    step_begin<256>(d, par_next);
}

// Whole-instance list rebuild of every instance at the next step.
__global__ void k_force_rebuild(Dev d)
{
    for (int k = threadIdx.x; k < d.n_inst; k += blockDim.x) d.st[k].force_rebuild = 1;
}

// Init variant: rebuild everything, reset the grid accumulators.
__global__ void __launch_bounds__(256) k_init_begin(Dev d)
{
    for (int k = threadIdx.x; k < d.n_inst; k += blockDim.x) {
        InstState *st = &d.st[k];
        st->rebuild = 2;
        st->ds = 0.0f;
        st->force_rebuild = 0;
        st->disp_step = 0u;
        st->flagged = 0;   // not zero after a step left half done
        st->div_count = 0;
        for (int p = 0; p < 2; ++p)
            for (int q = 0; q < 3; ++q) {
                st->mm[p][2 * q] = f2o(1.0e30f);
                st->mm[p][2 * q + 1] = f2o(-1.0e30f);
            }
    }
    __syncthreads();
    assign_hash_slices<256>(d);
    if (threadIdx.x == 0) {
        d.flags[0] = 1;
        *d.n_build = 0;
        for (int q = 0; q < DEALS; ++q) d.deal[q] = 0;
        *d.div_total = 0;
        *d.div_prev = 0;
        *d.n_pairs = 0ull;
    }
}

// ---------------------------------------------------------------------------
// Block reductions over the 180 nodes of a cell.
// ---------------------------------------------------------------------------
struct GeomScratch {
    double sum[SLOTS / 32][3];
    float mn[SLOTS / 32][3], mx[SLOTS / 32][3];
    double vol[SLOTS / 32], area[SLOTS / 32];
    double fc[CS3D_FACES][3];   // face centres relative to the cell's centre of mass
};

// t / 180, correctly rounded by Markstein's method as div_m; an infinity stays
// one (its remainder is no number).
__device__ __forceinline__ double div_nodes(double t)
{
    constexpr double r = 1.0 / NODES;
    const double q = t * r;
    const double e = fma(-q, (double)NODES, t);
    return e == e ? fma(e, r, q) : q;
}

// Centre of mass (FP64 sum, src/centermass.cu:8-50) and bounding box
// (src/propagatebound.cu:10-141) of the cell staged in xs: first the warps'
// sums and extents, then, after the barrier, whoever needs them adds them up.
__device__ __forceinline__ void cell_geom(const float4 *xs, GeomScratch &gs)
{
    const int i = threadIdx.x, w = i >> 5, l = i & 31;
    const bool real = i < NODES;
    const float4 p = xs[real ? i : 0];
    const double sx = warp_sum(real ? (double)p.x : 0.0), sy = warp_sum(real ? (double)p.y : 0.0),
                 sz = warp_sum(real ? (double)p.z : 0.0);
    const float mnx = warp_min(p.x), mny = warp_min(p.y), mnz = warp_min(p.z);
    const float mxx = warp_max(p.x), mxy = warp_max(p.y), mxz = warp_max(p.z);
    if (l == 0) {
        gs.sum[w][0] = sx; gs.sum[w][1] = sy; gs.sum[w][2] = sz;
        gs.mn[w][0] = mnx; gs.mn[w][1] = mny; gs.mn[w][2] = mnz;
        gs.mx[w][0] = mxx; gs.mx[w][1] = mxy; gs.mx[w][2] = mxz;
    }
    __syncthreads();
}

__device__ __forceinline__ float3 geom_centre(const GeomScratch &gs)
{
    double tx = 0, ty = 0, tz = 0;
    for (int q = 0; q < SLOTS / 32; ++q) { tx += gs.sum[q][0]; ty += gs.sum[q][1]; tz += gs.sum[q][2]; }
    return make_float3((float)div_nodes(tx), (float)div_nodes(ty), (float)div_nodes(tz));
}

__device__ __forceinline__ void geom_box(const GeomScratch &gs, float4 &lo, float4 &hi)
{
    lo = make_float4(1e30f, 1e30f, 1e30f, 0.0f);
    hi = make_float4(-1e30f, -1e30f, -1e30f, 0.0f);
    for (int q = 0; q < SLOTS / 32; ++q) {
        lo.x = fminf(lo.x, gs.mn[q][0]); lo.y = fminf(lo.y, gs.mn[q][1]); lo.z = fminf(lo.z, gs.mn[q][2]);
        hi.x = fmaxf(hi.x, gs.mx[q][0]); hi.y = fmaxf(hi.y, gs.mx[q][1]); hi.z = fmaxf(hi.z, gs.mx[q][2]);
    }
}

// sqrt(x) to half an ulp: the approximate inverse root, refined once (to 1e-12),
// then Heron's step by the exact remainder.  Zero, values that the approximation
// does not reach and those that are no finite numbers take the full root.
__device__ __forceinline__ double sqrt_full(double x)
{
    if (!(x > 1e-280 && x < 1e280)) return sqrt(x);
    const double r = rsqrt_nr(x), s = x * r;
    return fma(0.5 * r, fma(-s, s, x), s);
}

// Volume, area and the division test, src/volume.cu:5-163, in FP64.  Each
// face (12 pentagons, 80 hexagons, vertices relative to the cell's centre of
// mass) is cut into triangles at its vertex average; the volume is the sum
// of |det| / 6 of the tetrahedra (centre of mass, triangle) and the area the
// sum of the triangle areas.  The face centres first (one thread per face)
// , then the 552 triangles dealt out to all threads.
__device__ __noinline__ void cell_volume(const uint8_t *faces, const uint32_t *tris, const float4 *xs, float3 cm,
                                         GeomScratch &gs, bool sph, double &vol, double &area)
{
    const int t = threadIdx.x, w = t >> 5, l = t & 31;
    const double cx = cm.x, cy = cm.y, cz = cm.z;
    uint32_t tri[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) tri[k] = t + k * SLOTS < CS3D_FACES * 6 ? __ldg(&tris[t + k * SLOTS]) : 0u;
    if (t < CS3D_FACES) {
        const uint8_t *F = faces + 7 * t;
        double ax = 0, ay = 0, az = 0;
        for (int q = 0; q < 5; ++q) {
            const float4 p = xs[F[q]];
            ax += (double)p.x - cx; ay += (double)p.y - cy; az += (double)p.z - cz;
        }
        double fac = (double)0.166666667f;
        if (t < 12) fac = (double)0.2f;
        else {
            const float4 p = xs[F[5]];
            ax += (double)p.x - cx; ay += (double)p.y - cy; az += (double)p.z - cz;
        }
        gs.fc[t][0] = ax * fac; gs.fc[t][1] = ay * fac; gs.fc[t][2] = az * fac;
    }
    __syncthreads();
    double tv = 0, fa = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (t + k * SLOTS >= CS3D_FACES * 6) break;
        const float4 p0 = xs[tri[k] & 255u], p1 = xs[(tri[k] >> 8) & 255u];
        const int f = tri[k] >> 16;
        const double x0 = (double)p0.x - cx, y0 = (double)p0.y - cy, z0 = (double)p0.z - cz;
        const double x1 = (double)p1.x - cx, y1 = (double)p1.y - cy, z1 = (double)p1.z - cz;
        const double ax = gs.fc[f][0], ay = gs.fc[f][1], az = gs.fc[f][2];
        const double n1 = (y1 * az - ay * z1) * x0;
        const double n2 = (z1 * ax - az * x1) * y0;
        const double n3 = (x1 * ay - ax * y1) * z0;
        tv += fabs(n1 + n2 + n3);
        if (sph) {
            const double u1 = x0 - ax, v1 = y0 - ay, w1 = z0 - az;
            const double u2 = x1 - ax, v2 = y1 - ay, w2 = z1 - az;
            const double xx = v1 * w2 - w1 * v2, yy = w1 * u2 - u1 * w2, zz = u1 * v2 - v1 * u2;
            fa += 0.5 * sqrt_full(xx * xx + yy * yy + zz * zz);
        }
    }
    tv = warp_sum(tv);
    fa = warp_sum(fa);
    if (l == 0) { gs.vol[w] = tv; gs.area[w] = fa; }
    __syncthreads();
    vol = 0; area = 0;
    for (int q = 0; q < SLOTS / 32; ++q) { vol += gs.vol[q]; area += gs.area[q]; }
    vol = vol / 6.0;
}

// ---------------------------------------------------------------------------
// S1: conservative force (src/propagate.cu:183-520), first dissipative force
// (:523-665 with v after Integrate) and VelocityUpdateA/B (:714-736).
// INIT = true evaluates the initial forces of src/GPUbounce.cu:978-1004
// (no velocity update; Fd written to FD).
// ---------------------------------------------------------------------------
// Arm forces of the angles at each vertex, summed by destination: entry
// vertex*3 + k goes to the vertex's k-th neighbour.
struct ArmForces {
    double x[SLOTS * 3], y[SLOTS * 3], z[SLOTS * 3];
};

// The next cell's nodes and first entries towards L2: a system of more than
// some 20,000 cells does not stay there between steps.  With the bins of a
// node by multiplication (div_dl), a candidate's bin ranges in two 16-byte
// words with its box and the cell's set-up spread over the warps: S1 of 100,000 packed
// cells 1.86 -> 1.68 ms, of 3000 growing ones 85 -> 80 us.
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void prefetch_cell(const Dev &d, int a)
{
    const int t = threadIdx.x;
    constexpr int LINES = SLOTS * 16 / 128;   // a cell's positions, and as much of its entries (8 a node)
    if (t < LINES) prefetch_l2((const char *)(d.X + (size_t)a * SLOTS) + 128 * t);
    else if (t < 2 * LINES) prefetch_l2((const char *)(d.V + (size_t)a * SLOTS) + 128 * (t - LINES));
    else if (t < 3 * LINES) prefetch_l2((const char *)(d.ent + (size_t)a * MAXE * SLOTS) + 128 * (t - 2 * LINES));
}

struct S1Smem {
    // The cell's positions and velocities as floats, converted where they are
    // read: with FP64 copies the gathers of the neighbours kept the L1 pipe 70 %
    // busy, with floats the conversions share the XU pipe's 32 % (S1 of 100,000
    // packed cells 1.66 -> 1.61 ms; with positions in both forms 1.69).
    float4 xs[SLOTS], vs[SLOTS];
    SlotData sd;
    union {                         // the angles' arms are read before the sweep begins: the
        SweepSmem sweep[SLOTS / 32];  // room is worth more as L1 (S1 of 100,000 packed
        ArmForces arm;                // cells 1.76 -> 1.73 ms, a barrier included)
    };
    float press;         // the cell's pressure of this step
    int next[2];
};

template <bool INIT, bool COOP>
__device__ __forceinline__ void s1_cells(const Dev &d, int par, S1Smem &sm)
{
    const int W = n_work(d);
    const int i = threadIdx.x;
    const uint32_t nnp = (i < NODES) ? __ldg(&d.topo.nnpack[i]) : 0u;
    const int n0 = nnp & 255, n1 = (nnp >> 8) & 255, n2 = (nnp >> 16) & 255;
    const float sgn = (float)(int8_t)(nnp >> 24);
    Dealer deal(&d.deal[DEAL_S1], sm.next);
    while (deal.w < W) {
        // the newest cells first: fresh daughters take longest
        const int a = cell_of(d, W - 1 - deal.w);
        deal.draw();
        const int inst = inst_of(d, a);
        const InstParams &P = d.prm[inst];
        const size_t g = (size_t)a * SLOTS + i;
        const int nc = d.ncand[a];
        float4 x4 = make_float4(0, 0, 0, 0), v4 = make_float4(0, 0, 0, 0);
        if (i < NODES) { x4 = d.X[g]; v4 = d.V[g]; }
        const int ne = d.nent[g];
        uint32_t pre[EPRE / 2];
#pragma unroll
        for (int q = 0; q < EPRE / 2; ++q)
            pre[q] = (uint32_t)d.ent[((size_t)a * MAXE + 2 * q) * SLOTS + i] |
                     ((uint32_t)d.ent[((size_t)a * MAXE + 2 * q + 1) * SLOTS + i] << 16);
        sm.xs[i] = x4;
        sm.vs[i] = v4;
        slots_load(d, a, &d.st[inst], par, sm.sd);
        if (i == 128) {
            // this step's PressureUpdate (none before the initial forces)
            const float pr = INIT ? d.press[a] : pressure_update(d, P, a, d.st[inst].step);
            if (!INIT) d.press[a] = pr;
            sm.press = pr;
        }
        __syncthreads();
        slots_boxes(d, P, par, sm.sd, nc);
        const int wn = sm.next[deal.turn];
        if (wn < W) prefetch_cell(d, cell_of(d, W - 1 - wn));
        const float3 x = f3(x4);
        const float3 v = f3(v4);
        // The node force is accumulated in FP64: its terms (pressure up
        // to ~1e3, stiff contact repulsion up to ~1e4) can cancel to a
        // net force orders of magnitude smaller, and the sum is rounded to
        // float once, as the reference stores it.
        double FX = 0.0, FY = 0.0, FZ = 0.0;
        if (i < NODES) {
            const double3 xi = as_d3(x4);
            const Arm pa = make_arm(as_d3(sm.xs[n0]), xi), pb = make_arm(as_d3(sm.xs[n1]), xi),
                      pc = make_arm(as_d3(sm.xs[n2]), xi);
            // springs, src/propagate.cu:298-314, along the angles' arms:
            // k (R - R0) / R0 * d / R = k (1/R0 - 1/R) d
            const double stiff = d.E[a];
            const auto spring = [&](const Arm &p, int k) {
                const double c = stiff * (__ldg(&d.topo.r0i[3 * i + k]) - p.ir);
                FX += c * p.x; FY += c * p.y; FZ += c * p.z;
            };
            spring(pa, 0);
            spring(pb, 1);
            spring(pc, 2);
            // internal pressure, src/propagate.cu:318-330 (CM of the previous step)
            {
                const float4 cm = d.CM[a];
                const double rx = xi.x - cm.x, ry = xi.y - cm.y, rz = xi.z - cm.z;
                const double c = 3.0 * (double)sm.press * rsqrt_nr(rx * rx + ry * ry + rz * rz);
                FX += c * rx; FY += c * ry; FZ += c * rz;
            }
            // bond angles: thread = vertex, three angles each
            if (P.angles) {
                const double2 *cs0 = d.topo.cs0 + 3 * i;
                const float4 th = __ldg(&d.topo.th0[i]);
                // angles (n0, n1), (n1, n2), (n0, n2); arm ends summed by destination
                double3 F01p, F01q, F12p, F12q, F02p, F02q;
                double2 t0 = __ldg(&cs0[0]);
                angle_term(pa, pb, th.x, t0.x, t0.y, F01p, F01q);
                t0 = __ldg(&cs0[1]);
                angle_term(pb, pc, th.y, t0.x, t0.y, F12p, F12q);
                t0 = __ldg(&cs0[2]);
                angle_term(pa, pc, th.z, t0.x, t0.y, F02p, F02q);
                const int o = i * 3;
                sm.arm.x[o] = F01p.x + F02p.x; sm.arm.y[o] = F01p.y + F02p.y; sm.arm.z[o] = F01p.z + F02p.z;
                sm.arm.x[o + 1] = F01q.x + F12p.x; sm.arm.y[o + 1] = F01q.y + F12p.y; sm.arm.z[o + 1] = F01q.z + F12p.z;
                sm.arm.x[o + 2] = F12q.x + F02q.x; sm.arm.y[o + 2] = F12q.y + F02q.y; sm.arm.z[o + 2] = F12q.z + F02q.z;
            }
        }
        __syncthreads();
        if (i < NODES) {
            if (isnan(x.x) || isnan(x.y) || isnan(x.z)) atomic_or_err(&d.st[inst], CS3D_ERRBIT_NAN);
            // bond angles, src/propagate.cu:81-181: the vertex terms (minus
            // the arm forces of the angles at i) and the arm terms (the arm
            // forces that the angles at the three neighbours send to i)
            if (P.angles) {
                const int o = i * 3;
                const uint4 am = __ldg(&d.topo.arm[i]);
                FX += sm.arm.x[am.x] + sm.arm.x[am.y] + sm.arm.x[am.z] - (sm.arm.x[o] + sm.arm.x[o + 1] + sm.arm.x[o + 2]);
                FY += sm.arm.y[am.x] + sm.arm.y[am.y] + sm.arm.y[am.z] - (sm.arm.y[o] + sm.arm.y[o + 1] + sm.arm.y[o + 2]);
                FZ += sm.arm.z[am.x] + sm.arm.z[am.y] + sm.arm.z[am.z] - (sm.arm.z[o] + sm.arm.z[o + 1] + sm.arm.z[o + 2]);
            }
        }
        __syncthreads();
        // contacts, src/propagate.cu:356-442 and the first dissipative sweep
        double3 vsum = make_double3(0.0, 0.0, 0.0);
        const int nd = sweep_s1<COOP>(d, P, sm.sd, sm.sweep[i >> 5], a, i, x, v, ne, pre, FX, FY, FZ, vsum);
        if (i < NODES) {
            const double3 vt = tangential(sm.xs, n0, n1, n2, sgn, vsum);
            if (nd > MAXD) atomic_or_err(&d.st[inst], CS3D_ERRBIT_ENTRY_OVERFLOW);
            // rigid box walls, src/propagate.cu:474-510 (float gap tests)
            if (P.rigid) {
                const double wk = P.wallk, th = P.thresh;
                float g1 = x.x, g2 = __fsub_rn(P.box[0], x.x);
                if (g1 < P.thresh) FX += -wk * ((double)g1 - th);
                if (g2 < P.thresh) FX += wk * ((double)g2 - th);
                g1 = x.y; g2 = __fsub_rn(P.box[1], x.y);
                if (g1 < P.thresh) FY += -wk * ((double)g1 - th);
                if (g2 < P.thresh) FY += wk * ((double)g2 - th);
                g1 = x.z; g2 = __fsub_rn(P.box[2], x.z);
                if (g1 < P.thresh) FZ += -wk * ((double)g1 - th);
                if (g2 < P.thresh) FZ += wk * ((double)g2 - th);
            }
            const float3 fd = dis_force(P, sm.vs, i, n0, n1, n2, vt);
            d.FC[g] = make_float4((float)FX, (float)FY, (float)FZ, 0.f);
            d.ndis[g] = (uint8_t)(nd < MAXD ? nd : MAXD);
            if (INIT) {
                d.FD[g] = make_float4(fd.x, fd.y, fd.z, 0.f);
                d.FR[g] = make_float4(0.f, 0.f, 0.f, 0.f);  // no random force before the first step
            } else {
                const float dt = P.dt;
                // random force of this step (CalculateRanForce, GPUbounce.cu:1133-1137)
                float3 fr = make_float3(0.f, 0.f, 0.f);
                if (P.rands) {
                    fr = random_force(P, a, i, d.st[inst].step);
                    d.FR[g] = make_float4(fr.x, fr.y, fr.z, 0.f);
                }
                // VelocityUpdateA reads the stored (float) conservative force:
                // 0.5 (dt Fc + sqrt(dt) Fr) / m
                float vx = kick(v.x, __fadd_rn(__fmul_rn(dt, (float)FX), __fmul_rn(P.rdt, fr.x)), P);
                float vy = kick(v.y, __fadd_rn(__fmul_rn(dt, (float)FY), __fmul_rn(P.rdt, fr.y)), P);
                float vz = kick(v.z, __fadd_rn(__fmul_rn(dt, (float)FZ), __fmul_rn(P.rdt, fr.z)), P);
                const double hdt = 0.5 * (double)dt;
                vx = (float)((double)vx + div_m(hdt * (double)fd.x, P));
                vy = (float)((double)vy + div_m(hdt * (double)fd.y, P));
                vz = (float)((double)vz + div_m(hdt * (double)fd.z, P));
                d.Vb[g] = make_float4(vx, vy, vz, 0.f);
            }
        }
        __syncthreads();
        deal.advance();
    }
}

template <bool INIT>
__global__ void __launch_bounds__(SLOTS, 4) k_s1(Dev d, int par)
{
    extern __shared__ __align__(16) unsigned char s1_raw[];  // sizeof(S1Smem)
    s1_cells<INIT, false>(d, par, *reinterpret_cast<S1Smem *>(s1_raw));
}

// ---------------------------------------------------------------------------
// S2: second dissipative force with the updated velocities
// (src/GPUbounce.cu:1151), centre of mass (:1164), volumes and division
// flags (:1172, DIV only), bounding boxes and grid extents for the next step
// (:1312-1334).  The dissipative pairs are those S1 listed (same positions).
// ---------------------------------------------------------------------------
struct S2Smem {
    float4 xs[SLOTS];
    float4 vs[SLOTS];
    int cell[MAXC];
    GeomScratch gs;
    int dflag;   // the cell divides (division steps)
    float smax[SLOTS / 32];
    int next[2];
};

// Integrate + ForwardTime of the next step (src/propagate.cu:681-763) on the
// node's force and velocity after this step; returns the node's distance from
// its list anchor.  The same operations as k_integrate.
__device__ __forceinline__ float next_kick(const Dev &d, const InstParams &P, size_t g, float4 x4, float4 v4,
                                           float3 fd)
{
    const float4 fc = d.FC[g];
    const float dt = P.dt;
    float sx = __fadd_rn(__fmul_rn(dt, fc.x), __fmul_rn(dt, fd.x));
    float sy = __fadd_rn(__fmul_rn(dt, fc.y), __fmul_rn(dt, fd.y));
    float sz = __fadd_rn(__fmul_rn(dt, fc.z), __fmul_rn(dt, fd.z));
    if (P.rands) {
        const float4 fr = d.FR[g];
        sx = __fadd_rn(sx, __fmul_rn(P.rdt, fr.x));
        sy = __fadd_rn(sy, __fmul_rn(P.rdt, fr.y));
        sz = __fadd_rn(sz, __fmul_rn(P.rdt, fr.z));
    }
    float4 vn = v4;
    vn.x = kick(v4.x, sx, P);
    vn.y = kick(v4.y, sy, P);
    vn.z = kick(v4.z, sz, P);
    const float4 xn = make_float4(__fmaf_rn(vn.x, dt, x4.x), __fmaf_rn(vn.y, dt, x4.y),
                                  __fmaf_rn(vn.z, dt, x4.z), 0.0f);
    const float4 xb = d.Xb[g];
    const float ddx = xn.x - xb.x, ddy = xn.y - xb.y, ddz = xn.z - xb.z;
    d.X[g] = xn;
    d.V[g] = vn;
    return sqrtf(ddx * ddx + ddy * ddy + ddz * ddz);
}

__device__ __forceinline__ void flush_mm(const Dev &d, int inst, int pn, const float *acc)
{
    int *mm = d.st[inst].mm[pn];
    for (int q = 0; q < 3; ++q) {
        atomicMin(&mm[2 * q], f2o(acc[2 * q]));
        atomicMax(&mm[2 * q + 1], f2o(acc[2 * q + 1]));
    }
}

__device__ __forceinline__ void prefetch_cell_s2(const Dev &d, int a)
{
    const int t = threadIdx.x;
    constexpr int LINES = SLOTS * 16 / 128;
    const size_t o = (size_t)a * SLOTS;
    const float4 *p = t < LINES ? d.X + o : t < 2 * LINES ? d.Vb + o : t < 3 * LINES ? d.FC + o : d.Xb + o;
    if (t < 4 * LINES) prefetch_l2((const char *)p + 128 * (t % LINES));
    else if (t < 4 * LINES + 12) prefetch_l2((const char *)(d.dlist + o * MAXD) + 128 * (t - 4 * LINES));
}

// FUSE: the first half kick and drift of the next step (k_integrate) are
// done here, on the force and velocity in registers: FUSE 1 when the next
// step follows in the same launch sequence, FUSE 2 on the last step of a
// cs3d_step call, which also keeps the step-end positions (Xe; the step-end
// velocities are Vb) for the state read-back, so that the next call starts
// without a k_integrate pass.  A stream over X, Vb, FC and Xb with the
// partners' velocities gathered: S2 of 100,000 packed cells 0.62 -> 0.52 ms with
// the next cell prefetched, extents by redux, one thread's box and centre, the
// centre's division by 180 as a product, and no store of forces nobody reads.
template <bool DIV, bool COOP>
__device__ __forceinline__ void s2_cells(const Dev &d, int par, const int FUSE, S2Smem &sm)
{
    float *smax = sm.smax;
    const int W = n_work(d);
    const int i = threadIdx.x;
    const int pn = par ^ 1;
    const uint32_t nnp = (i < NODES) ? __ldg(&d.topo.nnpack[i]) : 0u;
    const int n0 = nnp & 255, n1 = (nnp >> 8) & 255, n2 = (nnp >> 16) & 255;
    const float sgn = (float)(int8_t)(nnp >> 24);
    int acc_inst = -1;
    float acc[6];
    Dealer deal(&d.deal[DEAL_S2], sm.next);
    while (deal.w < W) {
        const int a = cell_of(d, deal.w);
        deal.draw();
        const int inst = inst_of(d, a);
        const InstParams &P = d.prm[inst];
        InstState *st = &d.st[inst];
        const size_t g = (size_t)a * SLOTS + i;
        float4 x4 = make_float4(0, 0, 0, 0), v4 = make_float4(0, 0, 0, 0);
        int nd = 0;
        if (i < NODES) { x4 = d.X[g]; v4 = d.Vb[g]; nd = d.ndis[g]; }
        if (i < MAXC) sm.cell[i] = d.cand[(size_t)a * MAXC + i];
        sm.xs[i] = x4;
        sm.vs[i] = v4;
        __syncthreads();
        float disp = 0.0f;

        float3 fdk = make_float3(0.f, 0.f, 0.f);
        if (i < NODES) {
            const double3 vt = tangential(sm.xs, n0, n1, n2, sgn, sweep_s2<COOP>(d, sm.cell, a, i, f3(v4), nd));
            const float3 fd = dis_force(P, sm.vs, i, n0, n1, n2, vt);

            // between fused steps only the two cells of a division still need
            // the force: it went into the next kick
            if (FUSE != 1) d.FD[g] = make_float4(fd.x, fd.y, fd.z, 0.f);
            fdk = fd;
            if (FUSE == 2 && !DIV) d.Xe[g] = x4;
            if (FUSE && !DIV) disp = next_kick(d, P, g, x4, v4, fd);
            else d.V[g] = v4;
        }
        if (FUSE && !DIV) {
            disp = warp_max(disp);
            if ((i & 31) == 0) smax[i >> 5] = disp;
        }
        if (i == 0) sm.dflag = 0;
        cell_geom(sm.xs, sm.gs);
        const int wn = sm.next[deal.turn];
        if (wn < W) prefetch_cell_s2(d, cell_of(d, wn));
        float3 cm;
        if (DIV || i == 0) cm = geom_centre(sm.gs);
        if (DIV) {
            if (st->step <= P.div_steps && P.growth > 0.0f) {
                double vol, area;
                cell_volume(d.topo.faces, d.topo.tri, sm.xs, cm, sm.gs, P.check_sph != 0, vol, area);
                if (i == 0) {
                    d.vol[a] = (float)vol;
                    if (!isfinite(vol)) { atomic_or_err(st, CS3D_ERRBIT_NONFINITE_VOL); vol = 1.0; }
                    int flag = vol > (double)P.divvol;
                    if (P.check_sph) {
                        d.area[a] = (float)area;
                        if (flag) {
                            double cb = cbrt(vol);
                            double psi = 4.835975862049408 * cb * cb / area;
                            if (fabs(1.0 - psi) > 0.05) flag = 0;
                        }
                    }
                    d.divflag[a] = (uint8_t)flag;
                    sm.dflag = flag;
                    if (flag) {
                        d.flagged[P.base + atomicAdd(&st->flagged, 1)] = a;
                        d.flags[1] = 1;
                    }
                }
            }
        }
        if (FUSE && DIV) {
            // With the division decision known: a cell that does not divide
            // takes the next step's half kick and drift here, the two cells of
            // a division after their placement (k_div_apply).
            __syncthreads();
            const bool divides = sm.dflag != 0;   // uniform
            if (FUSE == 2 && !divides && i < NODES) d.Xe[g] = x4;
            if (!divides && i < NODES) disp = next_kick(d, P, g, x4, v4, fdk);
            if (FUSE == 1 && divides && i < NODES) d.FD[g] = make_float4(fdk.x, fdk.y, fdk.z, 0.f);
            disp = warp_max(disp);
            if ((i & 31) == 0) smax[i >> 5] = disp;
            __syncthreads();
        }
        if (i == 0) {
            if (FUSE && (!DIV || sm.dflag == 0)) {
                float mx = smax[0];  // visible: cell_geom (and the division decision) synchronise the block
                for (int q = 1; q < SLOTS / 32; ++q) mx = fmaxf(mx, smax[q]);
                d.cdisp[a] = mx;
                atomicMax(&st->disp_step, __float_as_uint(mx));
            }
            float4 lo, hi;
            geom_box(sm.gs, lo, hi);
            d.CM[a] = make_float4(cm.x, cm.y, cm.z, 0.f);
            d.aabb[pn][2 * a] = lo;
            d.aabb[pn][2 * a + 1] = hi;
            if (DIV && sm.dflag) {
                // the boxes of its two cells enter the extents after their placement
            } else if (inst != acc_inst) {
                if (acc_inst >= 0) flush_mm(d, acc_inst, pn, acc);
                acc_inst = inst;
                acc[0] = lo.x; acc[1] = hi.x; acc[2] = lo.y; acc[3] = hi.y; acc[4] = lo.z; acc[5] = hi.z;
            } else {
                acc[0] = fminf(acc[0], lo.x); acc[1] = fmaxf(acc[1], hi.x);
                acc[2] = fminf(acc[2], lo.y); acc[3] = fmaxf(acc[3], hi.y);
                acc[4] = fminf(acc[4], lo.z); acc[5] = fmaxf(acc[5], hi.z);
            }
        }
        __syncthreads();
        deal.advance();
    }
    if (threadIdx.x == 0 && acc_inst >= 0) flush_mm(d, acc_inst, pn, acc);
}

template <bool DIV, int FUSE>
__global__ void __launch_bounds__(SLOTS, 5) k_s2(Dev d, int par)
{
    __shared__ S2Smem sm;
    s2_cells<DIV, false>(d, par, FUSE, sm);
}

// Centre of mass, bounding boxes and grid extents only (initialisation,
// src/GPUbounce.cu:739-763).
__global__ void __launch_bounds__(SLOTS) k_geom(Dev d, int par)
{
    __shared__ float4 xs[SLOTS];
    __shared__ GeomScratch gs;
    const int W = n_work(d);
    const int i = threadIdx.x;
    for (int w = blockIdx.x; w < W; w += gridDim.x) {
        const int a = cell_of(d, w);
        const int inst = inst_of(d, a);
        xs[i] = (i < NODES) ? d.X[(size_t)a * SLOTS + i] : make_float4(0, 0, 0, 0);
        __syncthreads();
        cell_geom(xs, gs);
        if (i == 0) {
            const float3 cm = geom_centre(gs);
            float4 lo, hi;
            geom_box(gs, lo, hi);
            d.CM[a] = make_float4(cm.x, cm.y, cm.z, 0.f);
            d.aabb[par][2 * a] = lo;
            d.aabb[par][2 * a + 1] = hi;
            int *mm = d.st[inst].mm[par];
            atomicMin(&mm[0], f2o(lo.x)); atomicMax(&mm[1], f2o(hi.x));
            atomicMin(&mm[2], f2o(lo.y)); atomicMax(&mm[3], f2o(hi.y));
            atomicMin(&mm[4], f2o(lo.z)); atomicMax(&mm[5], f2o(hi.z));
        }
        __syncthreads();
    }
}

// calc_sys_CM, src/GPUbounce.cu:2504-2520: the float mean of the first n
// centres of mass, summed in cell order; recorded as the instance's system
// centre.
__device__ __forceinline__ float3 sys_centre(const Dev &d, const InstParams &P, InstState *st, int n)
{
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    for (int c = 0; c < n; ++c) {
        const float4 cm = d.CM[P.base + c];
        sx = __fadd_rn(sx, cm.x);
        sy = __fadd_rn(sy, cm.y);
        sz = __fadd_rn(sz, cm.z);
    }
    sx = __fdiv_rn(sx, (float)n);
    sy = __fdiv_rn(sy, (float)n);
    sz = __fdiv_rn(sz, (float)n);
    st->syscm[0] = sx;
    st->syscm[1] = sy;
    st->syscm[2] = sz;
    return make_float3(sx, sy, sz);
}

__device__ __forceinline__ float dist2(float4 cm, float3 o)
{
    const float dx = __fsub_rn(cm.x, o.x), dy = __fsub_rn(cm.y, o.y), dz = __fsub_rn(cm.z, o.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// getRmax2, src/GPUbounce.cu:2523-2536: the largest squared distance of the
// first n centres of mass from the recorded system centre.
__device__ __forceinline__ float rmax2_from(const Dev &d, const InstParams &P, const InstState *st, int n)
{
    const float3 o = make_float3(st->syscm[0], st->syscm[1], st->syscm[2]);
    float r2 = 0.0f;
    for (int c = 0; c < n; ++c) {
        const float v = dist2(d.CM[P.base + c], o);
        r2 = r2 < v ? v : r2;   // std::max
    }
    return r2;
}

// num_cells_far, src/GPUbounce.cu:1288-1290 and :2538-2565, after the
// divisions of a step (count_only_internal_cells): the newest div_count cells
// whose centre of mass lies farther than radius_cutoff x the largest distance
// from the system's centre are not counted as dividing.  The daughters'
// centres of mass are still 0 here (computed in their first step), as in the
// reference.  One thread per instance (k).
__device__ __forceinline__ void far_count(const Dev &d, int k)
{
    const InstParams &P = d.prm[k];
    InstState *st = &d.st[k];
    if (!(P.far_r > 0.0f) || !(st->step <= P.div_steps && P.growth > 0.0f)) return;
    const int n = st->n, nd = st->div_count;
    if (nd == 0 || n < 50) return;
    const float3 o = sys_centre(d, P, st, n);
    const float thr = __fmul_rn(__fmul_rn(P.far_r, P.far_r), rmax2_from(d, P, st, n));
    int far = 0;
    for (int c = n - nd; c < n; ++c)
        if (dist2(d.CM[P.base + c], o) > thr) ++far;
    if (far) {
        const int q = atomicAdd(d.n_far, 1);
        if (q < d.far_cap) d.farlog[q] = make_int4(k, st->step, far, 0);
    }
}

// ---------------------------------------------------------------------------
// Division (src/GPUbounce.cu:1210-1286, src/postscriptinit.cu:148-256).
// D1: one block per instance, dividers in ascending index order, one RANMAR
// normal each (bit-exact float arithmetic of src/RandomVector.h:8-24).  S2
// left the flagged cells of each instance in a list, in no order.  The
// generator's state is staged in shared memory: its draws are one dependent
// chain, which took 4 us a division from global memory.
// ---------------------------------------------------------------------------
template <typename S>   // InstState or DivRng
__device__ void ranmar_dev(S *st, float *out, int len)
{
    for (int v = 0; v < len; ++v) {
        float uni = __fsub_rn(st->u[st->i97], st->u[st->j97]);
        if (uni < 0.0f) uni = __fadd_rn(uni, 1.0f);
        st->u[st->i97] = uni;
        if (--st->i97 == 0) st->i97 = 97;
        if (--st->j97 == 0) st->j97 = 97;
        st->rc = __fsub_rn(st->rc, st->rcd);
        if (st->rc < 0.0f) st->rc = __fadd_rn(st->rc, st->rcm);
        uni = __fsub_rn(uni, st->rc);
        if (uni < 0.0f) uni = __fadd_rn(uni, 1.0f);
        out[v] = uni;
    }
}

template <typename S>
__device__ void random_vector_dev(S *st, float n[3])
{
    float r[2], s;
    do {
        ranmar_dev(st, r, 2);
        r[0] = __fsub_rn(__fmul_rn(2.0f, r[0]), 1.0f);
        r[1] = __fsub_rn(__fmul_rn(2.0f, r[1]), 1.0f);
        s = __fadd_rn(__fmul_rn(r[0], r[0]), __fmul_rn(r[1], r[1]));
    } while (s >= 1.0f);
    float x1 = r[0], x2 = r[1];
    float q = __fsqrt_rn(__fsub_rn(__fsub_rn(1.0f, __fmul_rn(x1, x1)), __fmul_rn(x2, x2)));
    n[0] = __fmul_rn(__fmul_rn(2.0f, x1), q);
    n[1] = __fmul_rn(__fmul_rn(2.0f, x2), q);
    n[2] = __fsub_rn(1.0f, __fmul_rn(2.0f, __fadd_rn(__fmul_rn(x1, x1), __fmul_rn(x2, x2))));
}

// Cell a's box of this step (aabb[pn]) into its instance's grid extents.
__device__ __forceinline__ void add_extents(const Dev &d, InstState *st, int pn, int a)
{
    const float4 lo = d.aabb[pn][2 * a], hi = d.aabb[pn][2 * a + 1];
    int *mm = st->mm[pn];
    atomicMin(&mm[0], f2o(lo.x)); atomicMax(&mm[1], f2o(hi.x));
    atomicMin(&mm[2], f2o(lo.y)); atomicMax(&mm[3], f2o(hi.y));
    atomicMin(&mm[4], f2o(lo.z)); atomicMax(&mm[5], f2o(hi.z));
}

struct DivRng {
    float u[98];
    float rc, rcd, rcm;
    int i97, j97;
};

struct DivSmem {
    DivRng rng;
    int warp_cnt[32];
    int base;
};

// NT threads; k: the instance; far: some instance counts internal cells.
template <int NT>
__device__ __forceinline__ void div_select(const Dev &d, int par, int k, bool far, DivSmem &sm)
{
    InstState *st = &d.st[k];
    const InstParams &P = d.prm[k];
    if (!(st->step <= P.div_steps && P.growth > 0.0f)) return;
    const int total = st->flagged, t = threadIdx.x;
    if (total == 0) return;
    const int n0 = st->n;
    const int room = P.cap - n0;
    const int ndiv = total < room ? total : room;
    __syncthreads();   // all have read the count
    if (t == 0) {
        if (total > room) atomicOr(&st->err, CS3D_ERRBIT_CAPACITY);
        sm.base = atomicAdd(d.div_total, ndiv);
        st->div_count = ndiv;
        st->flagged = 0;
    }
    for (int q = t; q < 98; q += NT) sm.rng.u[q] = st->u[q];
    if (t == 0) {
        sm.rng.rc = st->rc; sm.rng.rcd = st->rcd; sm.rng.rcm = st->rcm;
        sm.rng.i97 = st->i97; sm.rng.j97 = st->j97;
    }
    __syncthreads();
    const int base = sm.base;
    if (total <= NT) {
        // rank of each flagged cell among them
        if (t < total) {
            const int *f = d.flagged + P.base;
            const int a = f[t];
            int r = 0;
            for (int q = 0; q < total; ++q) r += f[q] < a;
            if (r < ndiv) {
                DivEntry &e = d.divtab[base + r];
                e.parent = a;
                e.daughter = P.base + n0 + r;
                e.inst = k;
            } else add_extents(d, st, par ^ 1, a);
        }
        __syncthreads();
    } else {
        // many: ascending compaction of the flags in chunks of NT
        int done = 0;
        for (int c0 = 0; c0 < n0 && done < total; c0 += NT) {
            const int c = c0 + t;
            const int f = (c < n0) ? (d.divflag[P.base + c] ? 1 : 0) : 0;
            const unsigned b = __ballot_sync(0xffffffffu, f);
            const int lane = t & 31, wid = t >> 5;
            if (lane == 0) sm.warp_cnt[wid] = __popc(b);
            __syncthreads();
            int off = done;
            for (int q = 0; q < wid; ++q) off += sm.warp_cnt[q];
            off += __popc(b & ((1u << lane) - 1u));
            if (f && off < ndiv) {
                DivEntry &e = d.divtab[base + off];
                e.parent = P.base + c;
                e.daughter = P.base + n0 + off;
                e.inst = k;
            } else if (f) add_extents(d, st, par ^ 1, P.base + c);
            int tot = 0;
            for (int q = 0; q < NT / 32; ++q) tot += sm.warp_cnt[q];
            done += tot;
            __syncthreads();
        }
    }
    // normals in ascending order (one serial RNG stream per instance)
    if (t == 0) {
        const int ev0 = atomicAdd(d.n_events, ndiv);
        const int w0 = d.single ? 0 : atomicAdd(d.work_n, ndiv);
        for (int q = 0; q < ndiv; ++q) {
            DivEntry &e = d.divtab[base + q];
            float n[3];
            random_vector_dev(&sm.rng, n);
            e.n[0] = n[0]; e.n[1] = n[1]; e.n[2] = n[2];
            float nn = sqrtf(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
            if (fabsf(nn - 1.0f) > 1e-3f) atomicOr(&st->err, CS3D_ERRBIT_BAD_NORMAL);
            if (ev0 + q < d.ev_cap) d.events[ev0 + q] = make_int4(k, st->step, e.parent - P.base, e.daughter - P.base);
            if (!d.single) d.work[w0 + q] = e.daughter;
        }
        st->n = n0 + ndiv;
        st->rc = sm.rng.rc; st->i97 = sm.rng.i97; st->j97 = sm.rng.j97;
        if (far) far_count(d, k);
    }
    __syncthreads();
    for (int q = t; q < 98; q += NT) st->u[q] = sm.rng.u[q];
    __syncthreads();
}

__global__ void __launch_bounds__(256) k_div_select(Dev d, int par, int far)
{
    __shared__ DivSmem sm;
    if (d.flags[1] && (int)blockIdx.x < d.n_inst) div_select<256>(d, par, blockIdx.x, far != 0, sm);
}

// D2: one block per division: the two daughters by half-space projection
// through CM + n*gap/2 (FP64 geometry), velocities, pressures, stiffness.
// With fuse also their next half kick and drift, which S2 gave every other cell.
__device__ __forceinline__ void div_apply(const Dev &d, int par, bool fuse, float4 *xs, GeomScratch &gs, float *smax)
{
    const int T = *d.div_total;
    const int pn = par ^ 1;
    const int i = threadIdx.x;
    for (int q = blockIdx.x; q < T; q += gridDim.x) {
        DivEntry e = d.divtab[q];
        const InstParams &P = d.prm[e.inst];
        const int a = e.parent, b = e.daughter;
        float4 cm4 = d.CM[a];
        double half = (double)(0.5f * P.rr);
        double cm[3] = {cm4.x, cm4.y, cm4.z};
        float4 xa = make_float4(0, 0, 0, 0), xb = make_float4(0, 0, 0, 0);
        if (i < NODES) {
            float4 x = d.X[(size_t)a * SLOTS + i];
            double px[3] = {x.x, x.y, x.z};
            // separate roundings (no DFMA) so the result is bit-identical to
            // the oracle's FP64 restatement of CalcAndUpdateDaughtPos
            for (int s = 0; s < 2; ++s) {
                double sg = s == 0 ? 1.0 : -1.0;
                double n[3] = {sg * e.n[0], sg * e.n[1], sg * e.n[2]};
                double o[3], y[3];
                for (int q = 0; q < 3; ++q) {
                    o[q] = __dadd_rn(cm[q], __dmul_rn(half, n[q]));
                    y[q] = __dsub_rn(px[q], o[q]);
                }
                double dn = __dadd_rn(__dadd_rn(__dmul_rn(y[0], n[0]), __dmul_rn(y[1], n[1])), __dmul_rn(y[2], n[2]));
                if (dn <= 0.0)
                    for (int q = 0; q < 3; ++q) y[q] = __dsub_rn(y[q], __dmul_rn(dn, n[q]));
                float4 r = make_float4((float)__dadd_rn(y[0], o[0]), (float)__dadd_rn(y[1], o[1]),
                                       (float)__dadd_rn(y[2], o[2]), 0.f);
                if (s == 0) xa = r; else xb = r;
            }
        }
        __syncthreads();
        xs[i] = xa;
        __syncthreads();
        float4 lo, hi;
        cell_geom(xs, gs);
        if (i == 0) {
            geom_box(gs, lo, hi);
            d.aabb[pn][2 * a] = lo;
            d.aabb[pn][2 * a + 1] = hi;
            add_extents(d, &d.st[e.inst], pn, a);
        }
        __syncthreads();
        xs[i] = xb;
        __syncthreads();
        cell_geom(xs, gs);
        if (i == 0) {
            geom_box(gs, lo, hi);
            d.aabb[pn][2 * b] = lo;
            d.aabb[pn][2 * b + 1] = hi;
            add_extents(d, &d.st[e.inst], pn, b);
            d.press[a] = P.minp;
            d.press[b] = P.minp;
            d.E[b] = P.daught_same ? d.E[a] : P.stiff1;
            d.cell_inst[b] = e.inst;
        }
        if (i < NODES) {
            size_t ga = (size_t)a * SLOTS + i, gb = (size_t)b * SLOTS + i;
            d.X[ga] = xa;
            d.X[gb] = xb;
            d.Xb[ga] = xa;   // new anchors of the displacement test
            d.Xb[gb] = xb;
            d.Xe[ga] = xa;   // step-end state of the two cells (read back after a fused last step)
            d.Xe[gb] = xb;
            d.Vb[gb] = d.Vb[ga];
            d.V[gb] = d.V[ga];
            d.FC[gb] = make_float4(0, 0, 0, 0);
            d.FD[gb] = make_float4(0, 0, 0, 0);
            // no random force before the daughter's first step: the slot may hold
            // that of a cell of an earlier load
            d.FR[gb] = make_float4(0, 0, 0, 0);
        }
        __syncthreads();
        if (fuse) {   // a thread's own nodes
            integrate_cell(d, a, smax);
            integrate_cell(d, b, smax);
        }
    }
}

__global__ void __launch_bounds__(SLOTS) k_div_apply(Dev d, int par, int fuse)
{
    __shared__ float4 xs[SLOTS];
    __shared__ GeomScratch gs;
    __shared__ float smax[SLOTS / 32];
    div_apply(d, par, fuse != 0, xs, gs, smax);
}

// CoM correction at the end of a step (correct_com, src/GPUbounce.cu:1430-1440
// with calc_sys_CM :2504-2520 and CorrectCoMMotion, src/propagate.cu:766-776):
// the mean of the cells' centres of mass (a float sum in cell order, as the
// host loop does; a daughter's entry is still 0 in its first step) is
// subtracted from every node.  The centres of mass, boxes and grid of this
// step keep their unshifted values, as in the reference; the list anchors
// move with the nodes (a uniform shift changes no distance).
//
// The order of the sum makes it a chain of n dependent float additions per
// component.  The block stages the centres in shared memory, so the chain
// waits for shared memory and the adder only; three threads take one
// component each.  One block per instance.
template <int NT>
__device__ __forceinline__ void com_centre(const Dev &d, int k, float (*stage)[NT])
{
    const InstParams &P = d.prm[k];
    if (!P.correct_com) return;   // uniform
    const int n = d.st[k].n, t = threadIdx.x;
    float s = 0.0f;
    for (int c0 = 0; c0 < n; c0 += NT) {
        __syncthreads();
        if (c0 + t < n) {
            const float4 cm = d.CM[P.base + c0 + t];
            stage[0][t] = cm.x; stage[1][t] = cm.y; stage[2][t] = cm.z;
        }
        __syncthreads();
        const int m = n - c0 < NT ? n - c0 : NT;
        if (t < 3) {
            const float *p = stage[t];
#pragma unroll 8
            for (int c = 0; c < m; ++c) s = __fadd_rn(s, p[c]);
        }
    }
    if (t < 3) d.st[k].syscm[t] = __fdiv_rn(s, (float)n);
}

__global__ void __launch_bounds__(256) k_com_centre(Dev d)
{
    __shared__ float stage[3][256];
    if ((int)blockIdx.x < d.n_inst) com_centre<256>(d, blockIdx.x, stage);
}

// The shift of the nodes and their anchors, all 192 slots of a cell: a stream
// over the active cells, bound by memory (64 B a node).  One block per
// instance took 300 us a step at 1023 cells, with the centre's sum from
// global memory.
__device__ __forceinline__ void com_shift(const Dev &d)
{
    const int W = n_work(d);
    for (int w = blockIdx.x; w < W; w += gridDim.x) {
        const int a = cell_of(d, w);
        const int inst = inst_of(d, a);
        if (!d.prm[inst].correct_com) continue;
        const float *o = d.st[inst].syscm;
        const float ox = o[0], oy = o[1], oz = o[2];
        const size_t g = (size_t)a * SLOTS + threadIdx.x;
        float4 x = d.X[g], b = d.Xb[g];
        x.x = __fsub_rn(x.x, ox); x.y = __fsub_rn(x.y, oy); x.z = __fsub_rn(x.z, oz);
        b.x = __fsub_rn(b.x, ox); b.y = __fsub_rn(b.y, oy); b.z = __fsub_rn(b.z, oz);
        d.X[g] = x;
        d.Xb[g] = b;
    }
}

__global__ void __launch_bounds__(SLOTS) k_com_shift(Dev d) { com_shift(d); }

// Cells softened when growth ends, src/GPUbounce.cu:1340-1429 (duringGrowth
// off): at the end of step div_time_steps + 2, after the step's grid and
// before its CoM correction.  One thread per instance runs the reference's
// host loops in their order.
__global__ void k_soften(Dev d, int step)
{
    const int k = blockIdx.x;
    if (k >= d.n_inst || threadIdx.x != 0) return;
    const InstParams &P = d.prm[k];
    InstState *st = &d.st[k];
    if (!P.soften || st->step != step || P.div_steps + 2 != step) return;
    const int n = st->n;
    int count = P.soft_n;
    if (P.soft_frac > 0.0f) count = (int)roundf(__fmul_rn(P.soft_frac, (float)n));
    float *E = d.E + P.base;
    if (P.soft_rand) {
        // distinct picks roundf(u * n) in [0, n]; n itself names no cell
        if (count > n + 1) { atomicOr(&st->err, CS3D_ERRBIT_SOFT_CELLS); return; }
        uint8_t *pick = d.pick + P.base + k;
        for (int c = 0; c <= n; ++c) pick[c] = 0;
        long long draws = 0;
        for (int got = 0; got < count;) {
            if (++draws > 64ll * (n + 1) + (1ll << 20)) { atomicOr(&st->err, CS3D_ERRBIT_SOFT_CELLS); break; }
            float u;
            ranmar_dev(st, &u, 1);
            const int ind = (int)roundf(__fmul_rn(u, (float)n));
            if (!pick[ind]) { pick[ind] = 1; ++got; }
        }
        for (int c = 0; c < n; ++c)
            if (pick[c]) E[c] = P.E2;
        return;
    }
    // getRmax2 runs before calc_sys_CM here (src/GPUbounce.cu:1399-1402), so
    // it measures from the previously recorded system centre
    const float r2max = rmax2_from(d, P, st, n);
    const float3 o = sys_centre(d, P, st, n);
    const float f = __fsub_rn(1.0f, P.closeness);
    const float thr = __fmul_rn(__fmul_rn(f, f), r2max);
    for (int c = 0, got = 0; got < count && c < n; ++c)
        if (dist2(d.CM[P.base + c], o) <= thr) { E[c] = P.E2; ++got; }
}

// Volume histogram of one instance's cells at the current positions (the
// analysis scripts/pop.py and the statistical checks do offline): one block
// per cell computes the centre of mass and the volume of src/volume.cu:5-163
// in FP64 (the division test's arithmetic) and counts it into one of nbins
// equal bins over [lo, hi), counts[0] below, counts[nbins + 1] at or above.
__global__ void __launch_bounds__(SLOTS) k_vol_hist(Dev d, int inst, float lo, float hi, int nbins,
                                                    unsigned long long *counts, float *vols)
{
    __shared__ float4 xs[SLOTS];
    __shared__ GeomScratch gs;
    const InstParams &P = d.prm[inst];
    const int n = d.st[inst].n;
    for (int c = blockIdx.x; c < n; c += gridDim.x) {
        const int a = P.base + c;
        const int i = threadIdx.x;
        xs[i] = i < NODES ? d.X[(size_t)a * SLOTS + i] : make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        cell_geom(xs, gs);
        double vol, area;
        cell_volume(d.topo.faces, d.topo.tri, xs, geom_centre(gs), gs, false, vol, area);
        if (i == 0) {
            const float v = (float)vol;
            if (vols) vols[c] = v;
            int b;
            if (!(v >= lo)) b = 0;
            else if (!(v < hi)) b = nbins + 1;
            else {
                b = 1 + (int)((double)(v - lo) / ((double)hi - (double)lo) * nbins);
                b = b > nbins ? nbins : b;
            }
            atomicAdd(&counts[b], 1ull);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Neighbour-list build (instances whose displacement bound reached the skin,
// or that divided): every cell's box at the current positions, a table of the
// cells by the bin of their box centre, then one CTA per cell that collects
// the cells whose boxes come within the list radius of its own and, of their
// nodes, those within the list radius of its nodes.
//
// A form that binned the nodes instead (a counting sort of all nodes into
// bins of the list radius, every thread walking the 27 bins around its node)
// went at the pace of the fullest node of a warp: next to the plane of a fresh
// division a bin holds tens of nodes, and the build of one cell there took
// 50 to 80 us.  Boxes cut the neighbours' nodes down to a few hundred that lie
// near the cell, the warps test those against a patch of 30 nodes each, and
// the entries come in their final order (ascending cell, then node).  Bound by
// the latency of one cell's chain in partial builds (11 us a cell alone on its
// SM) and by instruction issue in whole ones.  With
// this form a step of 2500 to 3200 growing cells went from 350 to 237 us (all
// of it list build), one of 301 from 98 to 69 us; a whole build of 30,000
// packed cells takes 0.70 ms (ncu) against 1.27 and the sort.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int bin_coord(float v, float inv)
{
    return (int)floorf(fminf(fmaxf(__fmul_rn(v, inv), -1.0e9f), 1.0e9f));
}

// Bin of a box along one axis: the bin of its centre.
__device__ __forceinline__ int box_bin(float lo, float hi, float inv)
{
    return bin_coord(__fmul_rn(0.5f, __fadd_rn(lo, hi)), inv);
}

// k: the size class.
__device__ __forceinline__ unsigned bin_slot(const InstState &st, int k, int ix, int iy, int iz)
{
    unsigned h = (unsigned)ix * 0x8da6b343u ^ (unsigned)iy * 0xd8163841u ^ (unsigned)iz * 0xcb1ab31fu ^
                 (unsigned)k * 0x85ebca6bu;
    h ^= h >> 15;
    h *= 0x9e3779b1u;
    return st.hbase + (h >> (32 - st.hbits));
}

// Gap of two intervals (negative: they overlap).
__device__ __forceinline__ float gap(float lo1, float hi1, float lo2, float hi2)
{
    return fmaxf(lo1 - hi2, lo2 - hi1);
}

__device__ __forceinline__ bool boxes_near(float4 l1, float4 h1, float4 l2, float4 h2, float r)
{
    return gap(l1.x, h1.x, l2.x, h2.x) <= r && gap(l1.y, h1.y, l2.y, h2.y) <= r && gap(l1.z, h1.z, l2.z, h2.z) <= r;
}

// List radius of two cells whose nodes are at most da and db from their
// anchors (both 0 at whole-instance builds), and the same for the box tests,
// which it enlarges by more than their rounding.
__device__ __forceinline__ float list_radius(const InstParams &P, bool full, float da, float db)
{
    return full ? P.rlist + 1e-4f : P.rlist + da + db + 1.1e-3f;
}
constexpr float BOX_REACH = 1.0001f;

// Size classes.  The extent of the largest cell widens the search of every
// cell, so that cells out of all proportion are kept apart: class 0 holds those
// with half extents of up to LARGE bins (a cell at rest has 0.7, one that
// divides 0.9), the next ones up to 2, 4, ... LARGE, in bins of 2, 4, ... the
// edge.  The first MAXL larger cells go into a list that every cell looks
// through, cheaper for a few than a class of their own; so do those beyond the
// last class.  One cell of 12 times the size among 40,000 sent all of them
// through all others: a whole build took 8.9 ms, 0.89 ms now, as without it.
// All 40,000 of 4 times the size: 0.98 ms before, 0.39 now; of 8 times 7.4 ms, 0.41.
constexpr float LARGE = 2.5f;
constexpr int MAXL = 64;

// 1 / bin edge of class k.
__device__ __forceinline__ float class_inv(float inv, int k) { return inv * __int_as_float((127 - k) << 23); }

// Class of a box (LEVELS: none).
__device__ __forceinline__ int box_level(float4 lo, float4 hi, float inv)
{
    const float h = 0.5f * fmaxf(hi.x - lo.x, fmaxf(hi.y - lo.y, hi.z - lo.z)) * inv;
    int k = 0;
    while (k < LEVELS && !(h <= LARGE * (float)(1 << k))) ++k;
    return k;
}

// B1: boxes at the current positions and the cell table, one warp per cell;
// and the cells to build into d.build: all cells of whole builds, and those
// that partial builds concern (the divided ones and those whose boxes come
// within the list radius of one).  The divided cells' own boxes are not needed
// for that: they lie within those of their placement (aabb[par], of the step
// before) and the kick since, which is their distance from their anchors.
__device__ __forceinline__ void nb_boxes(const Dev &d, int par)
{
    const int W = n_work(d), T = *d.div_prev;
    const int lane = threadIdx.x & 31, nw = SLOTS / 32;
    const unsigned epoch = *d.epoch;
    float half[3] = {0.f, 0.f, 0.f};   // largest half extents of this warp's cells (one instance)
    // the cells of a CTA's warps are listed with one atomic
    __shared__ int listed[SLOTS / 32];
    for (int w0 = blockIdx.x * nw; w0 < W; w0 += gridDim.x * nw) {
        const int w = w0 + (threadIdx.x >> 5);
        const int a = w < W ? cell_of(d, w) : 0;
        const int inst = inst_of(d, a);
        InstState *st = &d.st[inst];
        const int rb = w < W ? st->rebuild : 0;
        if (lane == 0) listed[threadIdx.x >> 5] = -1;
        if (rb) {
            const InstParams &P = d.prm[inst];
            const float4 *X = d.X + (size_t)a * SLOTS;
            float lx = 1e30f, ly = 1e30f, lz = 1e30f, hx = -1e30f, hy = -1e30f, hz = -1e30f;
#pragma unroll
            for (int k = 0; k < (NODES + 31) / 32; ++k) {
                const int i = lane + 32 * k;
                if (i < NODES) {
                    const float4 x = X[i];
                    lx = fminf(lx, x.x); hx = fmaxf(hx, x.x);
                    ly = fminf(ly, x.y); hy = fmaxf(hy, x.y);
                    lz = fminf(lz, x.z); hz = fmaxf(hz, x.z);
                }
            }
            lx = warp_min(lx); ly = warp_min(ly); lz = warp_min(lz);
            hx = warp_max(hx); hy = warp_max(hy); hz = warp_max(hz);
            const float4 lo = make_float4(lx, ly, lz, 0.f), hi = make_float4(hx, hy, hz, 0.f);
            int m = 0;
            if (rb == 1) {
                const float da = d.cdisp[a];
                for (int q = lane; q < T; q += 32) {
                    const DivEntry &e = d.divtab[q];
                    if (e.inst != inst) continue;
                    const int cs[2] = {e.parent, e.daughter};
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int c = cs[k];
                        float r = d.cdisp[c];
                        r += list_radius(P, false, da, r);
                        float4 pl = d.aabb[par][2 * c], ph = d.aabb[par][2 * c + 1];
                        if (P.correct_com) {   // the correction moved the nodes, not the boxes
                            const float *o = st->syscm;
                            pl = make_float4(pl.x - o[0], pl.y - o[1], pl.z - o[2], 0.f);
                            ph = make_float4(ph.x - o[0], ph.y - o[1], ph.z - o[2], 0.f);
                            r += 1e-3f;
                        }
                        if (a == c) m |= 2;
                        else if (boxes_near(lo, hi, pl, ph, r * BOX_REACH)) m |= 1;
                    }
                }
                m = __reduce_or_sync(0xffffffffu, m);
            }
            if (lane == 0) {
                d.nbox[2 * a] = lo;
                d.nbox[2 * a + 1] = hi;
                d.mark[a] = (uint8_t)m;
                if (rb == 2 || m) listed[threadIdx.x >> 5] = a;
                if (lx <= hx && ly <= hy && lz <= hz) {   // some node is a number, along each axis
                    const float inv = P.inv_bin;
                    const int k = box_level(lo, hi, inv);
                    bool listed_apart = false;
                    if (k == LEVELS) {
                        listed_apart = true;
                        d.large[P.base + P.cap - 1 - atomicAdd(&st->n_giant, 1)] = a;
                    } else if (k > 0 && __ldcg(&st->n_large) < MAXL) {
                        const int at = atomicAdd(&st->n_large, 1);
                        listed_apart = at < MAXL;
                        if (listed_apart) d.large[P.base + at] = a;
                    }
                    if (!listed_apart) {
                        // positive, which shows that the class is in use (a NaN, of a
                        // cell at infinity, would be the largest of all)
                        const float hq[3] = {fmaxf(0.5f * (hx - lx), 1e-30f), fmaxf(0.5f * (hy - ly), 1e-30f),
                                             fmaxf(0.5f * (hz - lz), 1e-30f)};
#pragma unroll
                        for (int q = 0; q < 3; ++q) {
                            if (d.single && k == 0) half[q] = fmaxf(half[q], hq[q]);
                            // a look first: most cells are smaller than one already in
                            else if (__float_as_uint(hq[q]) > __ldcg(&st->hmax[k][q]))
                                atomicMax(&st->hmax[k][q], __float_as_uint(hq[q]));
                        }
                        if (k > 0 && __ldcg(&st->top) < k) atomicMax(&st->top, k);
                        const float inv_k = class_inv(inv, k);
                        const unsigned b =
                            bin_slot(*st, k, box_bin(lx, hx, inv_k), box_bin(ly, hy, inv_k), box_bin(lz, hz, inv_k));
                        const unsigned long long old =
                            atomicExch(&d.bins[b], ((unsigned long long)epoch << 32) | (unsigned)a);
                        d.bnext[a] = (unsigned)(old >> 32) == epoch ? (int)(unsigned)old : -1;
                    }
                }
            }
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const int c = lane < nw ? listed[lane] : -1;
            const unsigned b = __ballot_sync(0xffffffffu, c >= 0);
            int at = 0;
            if (lane == 0 && b) at = atomicAdd(d.n_build, __popc(b));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (c >= 0) d.build[at + __popc(b & ((1u << lane) - 1u))] = c;
        }
        __syncthreads();
    }
    if (d.single) {
        // one atomic for a CTA: one for each cell of the only instance took 8 us at 3000 cells
        __shared__ unsigned most[3];
        if (threadIdx.x < 3) most[threadIdx.x] = 0u;
        __syncthreads();
        if (lane == 0)
            for (int q = 0; q < 3; ++q) atomicMax(&most[q], __float_as_uint(half[q]));
        __syncthreads();
        if (threadIdx.x < 3 && most[threadIdx.x]) atomicMax(&d.st[0].hmax[0][threadIdx.x], most[threadIdx.x]);
    }
}

__global__ void __launch_bounds__(SLOTS) k_nb_boxes(Dev d, int par)
{
    if (d.flags[0]) nb_boxes(d, par);
}

constexpr int NBW = SLOTS / 32;   // warps of a CTA, and cells whose nodes are staged together
constexpr int MAXB = SLOTS;       // cells with boxes in reach that one pass takes
constexpr int WL = 64;            // nodes of a warp's list

// Nodes in reach of a warp's patch: minus their coordinates (the distance
// tests are packed additions and multiplications of two nodes), the squared
// list radius of their cell and slot << 8 | node.
struct alignas(16) PatchList {
    float x[WL], y[WL], z[WL], r2[WL];
    uint16_t id[WL];
};

struct ListSmem {
    float4 node[NBW][SLOTS];       // nodes in reach of the cell, by staged cell: x, y, z, node
    PatchList list[NBW];
    int count[NBW];
    float rad[NBW];                // their list radii
    int raw[MAXB], cell[MAXB];     // cells in reach: as found, ascending
    unsigned touched[MAXC][6];     // partner nodes with an entry, by slot (CS3D_OPT_HALO_STATS)
    uint8_t used[MAXB];
    int n, hsum, next[2];
    // statistics of the instance st_inst, not yet in its state
    int st_inst, built, searches, max_cand, max_entries, max_halo;
};

// The nodes of cell c in reach (r) of the box lo, hi, in ascending order into
// seg; returns their number.  One warp.
__device__ __forceinline__ int stage_nodes(const Dev &d, int c, float4 lo, float4 hi, float r, float4 *seg)
{
    const int lane = threadIdx.x & 31;
    const float4 *X = d.X + (size_t)c * SLOTS;
    float4 x[(NODES + 31) / 32];
#pragma unroll
    for (int k = 0; k < (NODES + 31) / 32; ++k)
        x[k] = lane + 32 * k < NODES ? X[lane + 32 * k] : make_float4(1e30f, 1e30f, 1e30f, 0.f);
    int m = 0;
#pragma unroll
    for (int k = 0; k < (NODES + 31) / 32; ++k) {
        const bool in = boxes_near(lo, hi, x[k], x[k], r);
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in)
            seg[m + __popc(b & ((1u << lane) - 1u))] =
                make_float4(x[k].x, x[k].y, x[k].z, __int_as_float(lane + 32 * k));
        m += __popc(b);
    }
    return m;
}

__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b)
{
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c)
{
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long both(float v)
{
    return ((unsigned long long)__float_as_uint(v) << 32) | __float_as_uint(v);
}

// One thread's node in the list build: position (twice, for packed
// arithmetic), its entry column and the entries so far.
struct NodeEntries {
    unsigned long long x, y, z;
    uint16_t *ep;
    int cnt;
};

// The n nodes of the warp's list against the node of every lane; with store,
// entries for those within the radius.  Eight nodes at a time: the loads are
// broadcasts and the distances independent.  Returns whether this lane's node
// has any.
__device__ __forceinline__ bool patch_flush(PatchList &L, int n, NodeEntries &e, bool store, ListSmem &sm, bool halo)
{
    const int lane = threadIdx.x & 31;
    const int np = (n + 7) & ~7;
    if (lane < np - n) L.r2[n + lane] = -1.0f;   // no distance is below
    __syncwarp();
    bool any = false;
    for (int k = 0; k < np; k += 8) {
        unsigned m = 0;
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
            const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&L.x[k + h]);
            const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&L.y[k + h]);
            const ulonglong2 Z = *reinterpret_cast<const ulonglong2 *>(&L.z[k + h]);
            const float4 r2 = *reinterpret_cast<const float4 *>(&L.r2[k + h]);
            const unsigned long long dx0 = add2(e.x, X.x), dx1 = add2(e.x, X.y), dy0 = add2(e.y, Y.x),
                                     dy1 = add2(e.y, Y.y), dz0 = add2(e.z, Z.x), dz1 = add2(e.z, Z.y);
            const unsigned long long d0 = fma2(dz0, dz0, fma2(dy0, dy0, fma2(dx0, dx0, 0ull)));
            const unsigned long long d1 = fma2(dz1, dz1, fma2(dy1, dy1, fma2(dx1, dx1, 0ull)));
            if (__uint_as_float((unsigned)d0) < r2.x) m |= 1u << h;
            if (__uint_as_float((unsigned)(d0 >> 32)) < r2.y) m |= 2u << h;
            if (__uint_as_float((unsigned)d1) < r2.z) m |= 4u << h;
            if (__uint_as_float((unsigned)(d1 >> 32)) < r2.w) m |= 8u << h;
        }
        any |= m != 0u;
        if (!store) continue;
        while (m) {
            const unsigned id = L.id[k + __ffs(m) - 1];
            m &= m - 1u;
            sm.used[id >> 8] = 1;
            if (halo) atomicOr(&sm.touched[id >> 8][(id & 255u) >> 5], 1u << (id & 31u));
            if (e.cnt < MAXE) e.ep[(size_t)e.cnt * SLOTS] = (uint16_t)id;
            ++e.cnt;
        }
    }
    __syncwarp();
    return any;
}

// The m staged nodes of one cell (slot s, list radius rad) that are in reach
// of the box of the warp's patch, onto the warp's list; a list with more than
// 32 nodes is flushed.  n: its length.
__device__ __forceinline__ bool patch_add(PatchList &L, int &n, const float4 *seg, int m, int s, float rad, float4 plo,
                                          float4 phi, NodeEntries &e, bool store, ListSmem &sm, bool halo)
{
    const int lane = threadIdx.x & 31;
    bool any = false;
    for (int q0 = 0; q0 < m; q0 += 32) {
        float4 y = make_float4(1e30f, 1e30f, 1e30f, 0.f);
        if (q0 + lane < m) y = seg[q0 + lane];
        const bool in = boxes_near(plo, phi, y, y, rad * BOX_REACH);
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int k = n + __popc(b & ((1u << lane) - 1u));
            L.x[k] = -y.x; L.y[k] = -y.y; L.z[k] = -y.z;
            L.r2[k] = rad * rad;
            L.id[k] = (uint16_t)((s << 8) | __float_as_int(y.w));
        }
        n += __popc(b);
        if (n > WL - 32) {
            any |= patch_flush(L, n, e, store, sm, halo);
            n = 0;
        }
    }
    return any;
}

// Cell c (box l, h) in reach of cell a (box lo, hi).
__device__ __forceinline__ bool cell_near(const Dev &d, const InstParams &P, int a, float4 lo, float4 hi, bool full,
                                          float da, int c, float4 l, float4 h)
{
    return c != a && boxes_near(lo, hi, l, h, list_radius(P, full, da, full ? 0.0f : d.cdisp[c]) * BOX_REACH);
}

// Cells of the instance with a box in reach of the CTA's cell (a, box lo, hi)
// into sm.raw, through the table and the lists of large cells.  sm.n may exceed
// MAXB, also where the table would be no help.
__device__ __forceinline__ void cells_in_reach(const Dev &d, const InstParams &P, const InstState *st, int a, float4 lo,
                                               float4 hi, bool full, float da, unsigned epoch, ListSmem &sm)
{
    const int t = threadIdx.x;
    const auto take = [&](int c) {
        const int k = atomicAdd(&sm.n, 1);
        if (k < MAXB) sm.raw[k] = c;
    };
    const auto take_if_near = [&](int c) {
        if (cell_near(d, P, a, lo, hi, full, da, c, d.nbox[2 * c], d.nbox[2 * c + 1])) take(c);
    };
    const float r = list_radius(P, full, da, st->ds) * BOX_REACH;
    const int top = st->top, nl = min(st->n_large, MAXL), ng = st->n_giant;
    // largest half extents of the class
    unsigned hx = st->hmax[0][0], hy = st->hmax[0][1], hz = st->hmax[0][2];
    for (int k = 0;;) {
        if (hx != 0u) {   // some cells
            // the centre of a box in reach lies within r + its half extent of this
            // box; a thousandth more covers the rounding of the bounds
            const float inv = class_inv(P.inv_bin, k);
            const float ex = (r + __uint_as_float(hx)) * 1.001f, ey = (r + __uint_as_float(hy)) * 1.001f,
                        ez = (r + __uint_as_float(hz)) * 1.001f;
            const int x0 = bin_coord(lo.x - ex, inv), y0 = bin_coord(lo.y - ey, inv), z0 = bin_coord(lo.z - ez, inv);
            const long long nx = bin_coord(hi.x + ex, inv) - x0 + 1ll, ny = bin_coord(hi.y + ey, inv) - y0 + 1ll,
                            nz = bin_coord(hi.z + ez, inv) - z0 + 1ll;
            // A cell whose nodes are all NaN along an axis has no box (lo 1e30, hi
            // -1e30) and reaches nothing: the bins of its ranges come out negative,
            // and their product wraps to some 1e9.
            if (nx <= 0 || ny <= 0 || nz <= 0) return;
            if (nx > 64 || ny > 64 || nz > 64 || nx * ny * nz > 4096) {   // far larger than the class
                if (t == 0) atomicAdd(&sm.n, MAXB + 1);
                return;
            }
            const int nyz = (int)(ny * nz), nb = (int)nx * nyz;
            for (int q = t; q < nb; q += SLOTS) {
                const int ix = x0 + q / nyz, iy = y0 + (q % nyz) / (int)nz, iz = z0 + q % (int)nz;
                const unsigned long long h = d.bins[bin_slot(*st, k, ix, iy, iz)];
                int c = (unsigned)(h >> 32) == epoch ? (int)(unsigned)h : -1;
                while (c >= 0) {
                    const int nxt = d.bnext[c];
                    const float4 l = d.nbox[2 * c], g = d.nbox[2 * c + 1];
                    // bins share table entries: only the cells of this very bin
                    if (cell_near(d, P, a, lo, hi, full, da, c, l, g) && box_bin(l.x, g.x, inv) == ix &&
                        box_bin(l.y, g.y, inv) == iy && box_bin(l.z, g.z, inv) == iz &&
                        (top == 0 || box_level(l, g, P.inv_bin) == k))
                        take(c);
                    c = nxt;
                }
            }
        }
        if (++k > top) break;
        hx = st->hmax[k][0]; hy = st->hmax[k][1]; hz = st->hmax[k][2];
    }
    for (int q = t; q < nl; q += SLOTS) take_if_near(d.large[P.base + q]);
    for (int q = t; q < ng; q += SLOTS) take_if_near(d.large[P.base + P.cap - 1 - q]);
}

// sm.raw[0 .. n) ascending into sm.cell (n <= MAXB).  Whole CTA; synchronises before and after.
__device__ __forceinline__ void sort_reach(ListSmem &sm, int n)
{
    const int t = threadIdx.x;
    if (t < n) {
        const int key = sm.raw[t];
        int k = 0;
        for (int q = 0; q < n; ++q) k += sm.raw[q] < key;
        sm.cell[k] = key;
    }
    __syncthreads();
}

// Statistics of the lists built so far into their instance's state (thread 0).
__device__ __forceinline__ void list_stats(const Dev &d, ListSmem &sm)
{
    if (sm.st_inst < 0) return;
    InstState *st = &d.st[sm.st_inst];
    atomicAdd(&st->built, sm.built);
    if (sm.searches) atomicAdd(&st->searches, sm.searches);
    atomicMax(&st->max_cand, sm.max_cand);
    atomicMax(&st->max_entries, sm.max_entries);
    if (d.halo_stats) atomicMax(&st->max_halo, sm.max_halo);
}

// B2: the lists of cell a, with the radius of whole builds (full) or with the
// cells' displacements.  The whole CTA; its warps take a patch of 30
// neighbouring nodes each.  False, without full only, if some node has more
// entries than it has room for, or the cell more candidates.
__device__ __forceinline__ bool nb_cell(const Dev &d, int a, int node, unsigned epoch, bool full, ListSmem &sm)
{
    const int t = threadIdx.x, wid = t >> 5, lane = t & 31;
    const bool real = node < NODES;
    const bool halo = d.halo_stats != 0;
    const int inst = inst_of(d, a);
    InstState *st = &d.st[inst];
    const InstParams &P = d.prm[inst];
    const float da = full ? 0.0f : d.cdisp[a];
    const bool fresh = st->rebuild == 2 || (d.mark[a] & 2);   // new anchors
    const float4 lo = d.nbox[2 * a], hi = d.nbox[2 * a + 1];
    const size_t g = (size_t)a * SLOTS + node;
    const float4 x = real ? d.X[g] : make_float4(-1e30f, -1e30f, -1e30f, 0.f);
    __syncthreads();
    if (t == 0) {
        sm.n = 0;
        if (sm.st_inst != inst) {
            list_stats(d, sm);
            sm.st_inst = inst;
            sm.built = sm.searches = sm.max_cand = sm.max_entries = sm.max_halo = 0;
        }
    }
    sm.used[t] = 0;
    if (halo && t < MAXC)
        for (int q = 0; q < 6; ++q) sm.touched[t][q] = 0u;
    __syncthreads();
    cells_in_reach(d, P, st, a, lo, hi, full, da, epoch, sm);
    // box of the warp's patch
    float4 plo, phi;
    plo.x = warp_min(real ? x.x : 1e30f); phi.x = warp_max(real ? x.x : -1e30f);
    plo.y = warp_min(real ? x.y : 1e30f); phi.y = warp_max(real ? x.y : -1e30f);
    plo.z = warp_min(real ? x.z : 1e30f); phi.z = warp_max(real ? x.z : -1e30f);
    NodeEntries e = {both(x.x), both(x.y), both(x.z), d.ent + (size_t)a * MAXE * SLOTS + node, 0};
    PatchList &L = sm.list[wid];
    int nslot = 0, nl = 0, searched = 0;
    __syncthreads();
    const int nr = sm.n;   // uniform
    if (nr <= MAXC) {
        // usual case: every cell in reach gets a slot, six at a time
        sort_reach(sm, nr);
        nslot = nr;
        if (t < nr) d.cand[(size_t)a * MAXC + t] = sm.cell[t];
        for (int c0 = 0; c0 < nr; c0 += NBW) {
            if (c0 + wid < nr) {
                const int c = sm.cell[c0 + wid];
                const float rad = list_radius(P, full, da, full ? 0.0f : d.cdisp[c]);
                const int m = stage_nodes(d, c, lo, hi, rad * BOX_REACH, sm.node[wid]);
                if (lane == 0) { sm.count[wid] = m; sm.rad[wid] = rad; }
            }
            __syncthreads();
            const int nc = min(NBW, nr - c0);
            for (int c = 0; c < nc; ++c)
                patch_add(L, nl, sm.node[c], sm.count[c], c0 + c, sm.rad[c], plo, phi, e, true, sm, halo);
            __syncthreads();
        }
        patch_flush(L, nl, e, true, sm, halo);
    } else {
        // more cells in reach than slots: a slot only for a cell with an
        // entry, one cell at a time, in ascending order
        const auto use = [&](int nw) {   // the nw cells in sm.raw
            sort_reach(sm, nw);
            for (int c = 0; c < nw; ++c) {
                const float rad = list_radius(P, full, da, full ? 0.0f : d.cdisp[sm.cell[c]]);
                if (wid == 0) {
                    const int m = stage_nodes(d, sm.cell[c], lo, hi, rad * BOX_REACH, sm.node[0]);
                    if (lane == 0) sm.count[0] = m;
                }
                __syncthreads();
                nl = 0;
                bool any = patch_add(L, nl, sm.node[0], sm.count[0], 0, rad, plo, phi, e, false, sm, false);
                any |= patch_flush(L, nl, e, false, sm, false);
                if (__syncthreads_or(any)) {
                    if (nslot < MAXC) {
                        nl = 0;
                        patch_add(L, nl, sm.node[0], sm.count[0], nslot, rad, plo, phi, e, true, sm, halo);
                        patch_flush(L, nl, e, true, sm, halo);
                        if (t == 0) d.cand[(size_t)a * MAXC + nslot] = sm.cell[c];
                    }
                    ++nslot;
                }
                __syncthreads();
            }
        };
        if (nr <= MAXB) use(nr);
        else {
            // all cells of the instance, MAXB of them to a window and WIN windows
            // to a look, most of which find nothing
            constexpr int WIN = 4;
            searched = 1;
            const int n = st->n;
            for (int c0 = 0; c0 < n; c0 += WIN * MAXB) {
                unsigned hit = 0;
#pragma unroll
                for (int k = 0; k < WIN; ++k) {
                    const int q = c0 + k * MAXB + t, c = P.base + q;
                    if (q < n && cell_near(d, P, a, lo, hi, full, da, c, d.nbox[2 * c], d.nbox[2 * c + 1])) hit |= 1u << k;
                }
                if (!__syncthreads_or(hit)) continue;
                for (int k = 0; k < WIN; ++k) {
                    if (t == 0) sm.n = 0;
                    __syncthreads();
                    if (hit >> k & 1u) sm.raw[atomicAdd(&sm.n, 1)] = P.base + c0 + k * MAXB + t;
                    __syncthreads();
                    use(sm.n);
                    __syncthreads();   // all have read the count
                }
            }
        }
    }
    if (!full && __syncthreads_or(e.cnt > MAXE || nslot > MAXC)) return false;
    if (real) {
        d.nent[g] = (uint8_t)(e.cnt < MAXE ? e.cnt : MAXE);
        // new anchors, except for the neighbours of divided cells: other
        // cells' lists rely on their old anchors
        if (fresh) d.Xb[g] = x;
        if (e.cnt > MAXE) atomicOr(&st->err, CS3D_ERRBIT_ENTRY_OVERFLOW);
    }
    // the padding slots have no entries
    if (t >= NODES) d.nent[(size_t)a * SLOTS + t] = 0;
    const int wm = __reduce_max_sync(0xffffffffu, e.cnt);
    if (lane == 0) atomicMax(&sm.max_entries, wm);
    const int nused = __syncthreads_count(sm.used[t] != 0);
    int nh = 0;
    if (halo) {
        if (t == 0) sm.hsum = 0;
        __syncthreads();
        if (t < MAXC) {
            for (int q = 0; q < 6; ++q) nh += __popc(sm.touched[t][q]);
            atomicAdd(&sm.hsum, nh);
        }
        __syncthreads();
        nh = sm.hsum;
    }
    if (t == 0) {
        if (nslot > MAXC) atomicOr(&st->err, CS3D_ERRBIT_CAND_OVERFLOW);
        d.ncand[a] = nslot < MAXC ? nslot : MAXC;
        sm.built += 1;
        sm.searches += searched;
        sm.max_cand = max(sm.max_cand, nslot > MAXC ? nslot : nused);
        sm.max_halo = max(sm.max_halo, nh);
    }
    return true;
}

// The listed cells.  Where a partial build's radius gives a node more entries
// than it has room for, or the cell more candidates (cells far from their
// anchors in a crowd), the cell's lists are built with the radius of a whole build, which covers this step, and
// the instance is rebuilt whole in the next one.
__device__ __forceinline__ void nb_lists(const Dev &d, ListSmem &sm)
{
    const int t = threadIdx.x;
    const unsigned epoch = *d.epoch;
    const int node = __ldg(&d.topo.patch[t]);
    if (t == 0) sm.st_inst = -1;
    const int N = *d.n_build;
    Dealer deal(&d.deal[DEAL_LISTS], sm.next);
    while (deal.w < N) {
        const int a = d.build[deal.w];
        deal.draw();
        InstState *st = &d.st[inst_of(d, a)];
        bool full = st->rebuild == 2;
        while (!nb_cell(d, a, node, epoch, full, sm)) {
            full = true;
            if (t == 0) {
                st->force_rebuild = 1;
                atomicAdd(&st->fallbacks, 1);
            }
        }
        deal.advance();
    }
    __syncthreads();
    if (t == 0) list_stats(d, sm);
}

__global__ void __launch_bounds__(SLOTS, 6) k_nb_lists(Dev d)
{
    __shared__ ListSmem sm;
    if (d.flags[0]) nb_lists(d, sm);
}

// ---------------------------------------------------------------------------
// Whole steps in one kernel (cooperative launch, all CTAs resident): the
// phases of the launch sequence with grid barriers between them.  For small
// systems, most of whose kernels find little or nothing to do: a step of the
// sequence is five launches, seven where cells may divide, and an empty one
// takes some 2 us, a barrier 1.5 us.
// ---------------------------------------------------------------------------
union StepsSmem {
    S1Smem s1;
    S2Smem s2;
    ListSmem lists;
    DivSmem div;
    float com[3][SLOTS];
};

// Polls for the other CTAs at a barrier (about a microsecond each) by default.
constexpr unsigned SYNC_POLLS = 1u << 22;

// Polls until *p >= v.  Relaxed loads: an acquiring one empties the SM's L1,
// which the CTAs still at work beside this one need (S1 of 440 cells took 38 us
// beside acquiring polls, 24 without).  False if the others did not come: the
// CTA must return.  It has counted itself in, so that those still to come pass
// this barrier, do the next phase's work among themselves and give up at its
// end, where the arrivals no longer add up.  Nothing of that state is stepped
// again: the host refuses until the instances are loaded.  One thread.
__device__ __forceinline__ bool poll_until(const Dev &d, const unsigned *p, unsigned v)
{
    for (unsigned polls = 0; polls < d.polls; ++polls) {
        unsigned u;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(u) : "l"(p) : "memory");
        if (u >= v) {
            __threadfence();
            return true;
        }
        __nanosleep(20);
    }
    for (int k = 0; k < d.n_inst; ++k) atomic_or_err(&d.st[k], CS3D_ERRBIT_SYNC);
    return false;
}

// Barriers of the grid, every CTA in the same order.  b: barriers and serial
// sections so far.
struct GridBar {
    unsigned arrived = 0, serials = 0;
};

__device__ __forceinline__ bool grid_sync(const Dev &d, GridBar &b)
{
    b.arrived += gridDim.x;
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&d.bar[0], 1u);
        ok = poll_until(d, &d.bar[0], b.arrived);
    }
    return !__syncthreads_or(!ok);
}

// The same, with `serial` run by the last CTA to arrive (all its threads)
// before the others go on.
template <typename F>
__device__ __forceinline__ bool grid_sync(const Dev &d, GridBar &b, F serial)
{
    __shared__ int last;
    b.arrived += gridDim.x;
    b.serials += 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&d.bar[0], 1u) == b.arrived - 1u;
        if (last) __threadfence();
    }
    __syncthreads();
    bool ok = true;
    if (last) {
        serial();
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(&d.bar[1]), "r"(b.serials) : "memory");
        }
    } else if (threadIdx.x == 0) ok = poll_until(d, &d.bar[1], b.serials);
    return !__syncthreads_or(!ok);
}

// n steps from the kicked state (X, V hold the first step's half kick and
// drift); the first n_div of them test for division.  last: the call ends with
// them (S2 mode 2 on the last one).  com: some instance corrects its
// centre-of-mass motion, so that S2 leaves the kick to the phase that shifts
// the nodes; far: some instance counts internal cells.
__global__ void __launch_bounds__(SLOTS, 4) k_steps(Dev d, int par, int n, int n_div, int last, int com, int far)
{
    extern __shared__ __align__(16) unsigned char steps_raw[];
    StepsSmem &sm = *reinterpret_cast<StepsSmem *>(steps_raw);
    GridBar bar;
    if (!grid_sync(d, bar, [&] { step_begin<SLOTS>(d, par ^ 1); })) return;
    for (int k = 0; k < n; ++k, par ^= 1) {
        const bool div = k < n_div, end = k + 1 == n;
        const int fuse = com ? 0 : end && last ? 2 : 1;
        const auto next = [&] { if (!end) step_begin<SLOTS>(d, par); };
        if (d.flags[0]) {
            nb_boxes(d, par);
            if (!grid_sync(d, bar)) return;
            nb_lists(d, sm.lists);
            if (!grid_sync(d, bar)) return;
        }
        s1_cells<false, true>(d, par, sm.s1);
        if (!grid_sync(d, bar)) return;
        if (div) s2_cells<true, true>(d, par, fuse, sm.s2);
        else s2_cells<false, true>(d, par, fuse, sm.s2);
        // the next step begins at the last barrier of this one
        const auto centres = [&] {
            for (int q = 0; q < d.n_inst; ++q) com_centre<SLOTS>(d, q, sm.com);
        };
        if (!grid_sync(d, bar, [&] {
                if (d.flags[1]) return;
                if (com) centres();
                else next();
            }))
            return;
        if (div && d.flags[1]) {
            for (int q = blockIdx.x; q < d.n_inst; q += gridDim.x) div_select<SLOTS>(d, par, q, far != 0, sm.div);
            if (!grid_sync(d, bar)) return;
            div_apply(d, par, fuse != 0, sm.s2.xs, sm.s2.gs, sm.s2.smax);
            if (!grid_sync(d, bar, [&] {
                    if (com) centres();
                    else next();
                }))
                return;
        }
        if (com) {
            // a cell's shift and kick are its own CTA's
            com_shift(d);
            if (!end) {
                __syncthreads();
                const int W = n_work(d);
                for (int w = blockIdx.x; w < W; w += gridDim.x) integrate_cell(d, cell_of(d, w), sm.s2.smax);
            }
            if (!grid_sync(d, bar, next)) return;
        }
    }
}

}  // namespace cs3d
