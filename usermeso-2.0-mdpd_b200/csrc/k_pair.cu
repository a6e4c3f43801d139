// mDPD pair passes with each pair evaluated once.
//
// k_density_rows: one lane per particle row of the list (32 consecutive particles per warp, the
//   locally transposed table makes each entry index a coalesced warp load; two to eight lanes per
//   row where the chip is not full, density_lanes), G = 4, 6 or 8
//   neighbour positions in flight per lane (the batch's autotuner picks G).  rho_i
//   (fix_aboundary_rho_meso.cu:119-165) is summed in FP32 with the hardware rsqrt, as the
//   reference forms each term; the reference adds the terms in FP64, which changes rho by about
//   1e-7 of its mean and costs ~13 % of this pass.  The pass also writes, into the particle's
//   row of the compact table, the entries within the force cutoff that the row owns (bit 31 of
//   the list entry, set by the list build: a local j when j > i, a ghost j when j is an image
//   shifted in the positive direction).  The mirrored pair, seen from the other end, has the
//   opposite shift, so every pair is owned by exactly one row.  It also writes (x, y, z, rho) of
//   the particle and its ghost images for the force pass's gathers.
// k_force_pairs: the compact rows of a warp (32 of them; 4, 8 or 16 where that fills the chip
//   better, force_rows) are concatenated and split into 32 equal contiguous shares, one per lane (a prefix scan of the row lengths and one binary search), so
//   every lane evaluates the same number of pairs whatever the row lengths.  The concatenated
//   rows are first staged in shared memory by coalesced loads (consecutive lanes, consecutive
//   entries), so the pair loop's entry reads (each lane in a different row) do not touch 32
//   table lines each.  Each entry carries j's type; j's (x, y, z, rho) and velocity/signature are
//   two float4 gathers, loaded for the next pair while the current one is evaluated.  The mDPD pair force (pair_mdpd_meso.cu:139-225)
//   is summed for the row in 64-bit fixed point (2^-32 units) in registers and flushed when the
//   lane's share moves to the next row; -F goes to j's source particle in the same fixed point,
//   through shared memory when the source is one of the block's rows and global 64-bit
//   atomics otherwise.  Integer addition is associative, so no sum depends on the order of the
//   atomics: results are bitwise reproducible and the pairwise forces cancel exactly (total
//   momentum).  Every pair term is checked against the box's fix_pair_max, which keeps each
//   particle's whole sum inside the fixed-point range; a larger or non-finite term sets the
//   non-finite status.
// k_finalize: fixed-point sums -> FP32 pair force, final half-kick (body force added in FP64),
//   sums cleared: at the end of a run and of a step with energy and virial.  Between two steps of
//   a run k_integrate does the same for the step before it, ahead of its own half-kick.
#include "kernels.h"
#include "pair.cuh"
#include "pair_rows.cuh"

namespace mdpd {

// the density pass keeps G neighbour positions in flight per lane (G = 4, 6 or 8, chosen per
// batch by the autotuner); blocks per SM: 8 at up to 64 registers (G = 4, 6), 7 at up to 72 (G = 8)
template <int G> constexpr int density_blocks() { return G <= 6 ? 8 : 7; }

// ---------------------------------------------------------------------------------------------
// density pass, global indices
// ---------------------------------------------------------------------------------------------
// One lane per row; the geometry of entries goes two at a time through the two-lane FP32
// instructions.  A term is (h - r)^2 with r = rsq * rsqrt(rsq), formed as t = rsq * rsqrt(rsq) - h
// (one rounding; t is -(h - r) exactly) and min(t, 0)^2: pairs beyond the cutoff add 0, and so
// do the particle's own entry and coincident particles (rsq = 0 gives 0 * inf = NaN, which min()
// drops; a denormal rsq gives inf).  The reference skips rsq < 1e-20; here a normal rsq below 1e-20 (two particles
// closer than 1e-10, whose FP32 coordinates are then both below ~1e-3 in magnitude) would add
// h^2.  Rows are padded to the warp's longest with the particle itself.  Owned entries (bit 31,
// set by the list build) within the force cutoff go to the compact row.
template <int kGather, bool UNI> __device__ __forceinline__ void density_rows(const BoxDesc &B, const Unit &U)
{
    static_assert(kGather % 2 == 0, "entries are taken two at a time");
    const int i = U.begin + threadIdx.x;
    const bool live = i < U.end;
    const int c = B.st->cur;
    const bool in_group = live && (B.mask[c][i] & B.rho_bit);
    const int n = live ? MDPD_IDX(B.count[i], B.n_col + 1) : 0;
    int nmax = n;
    for (int o = 16; o > 0; o >>= 1) nmax = max(nmax, __shfl_xor_sync(0xffffffffu, nmax, o));
    // the warp's rows are one contiguous block of the table (entry k of its 32 rows at 32 k): it
    // is asked into L2 at once, so the entry loads after the first group wait on L2, not on DRAM
    if ((threadIdx.x & 31) == 0 && nmax > 0)
        prefetch_l2_bulk(B.table + (unsigned)(i & ~31) * (unsigned)B.n_col, 128u * (unsigned)nmax);
    const int self = live ? i : U.begin;
    const float4 pi = B.pos[self];
    const float h = B.cut_rho, rcf2 = B.rc2_force;
    const unsigned long long pix = pk2(pi.x, pi.x), piy = pk2(pi.y, pi.y), piz = pk2(pi.z, pi.z);
    const unsigned long long nh = pk2(-h, -h);
    const int ncol = B.n_col, ncol2 = B.n_col2;
    // unsigned 32-bit offsets: tables of up to 2^32 entries
    const int *row = B.table + ((unsigned)(i & ~31) * (unsigned)ncol + (unsigned)(i & 31));  // entry k at 32 k
    int *row2 = B.table2 + (size_t)self * ncol2;
    // one FP32 sum in row order: the terms of entries beyond the cutoff are exact zeros, so a row
    // and its filtered copy (full and reduced lists) give the same rho bit for bit
    float acc = 0.f;
    int n2 = 0;
    for (int k0 = 0; k0 < nmax; k0 += kGather) {
        int e[kGather];
        float4 pj[kGather];
#pragma unroll
        for (int q = 0; q < kGather; ++q) e[q] = k0 + q < n ? __ldcs(row + 32 * (k0 + q)) : self;
#pragma unroll
        for (int q = 0; q < kGather; ++q) pj[q] = __ldg(&B.pos[MDPD_IDX(e[q] & kEntryIndexMask, n_all(B))]);
#pragma unroll
        for (int q = 0; q < kGather; q += 2) {
            const unsigned long long dx = sub2(pix, pk2(pj[q].x, pj[q + 1].x));
            const unsigned long long dy = sub2(piy, pk2(pj[q].y, pj[q + 1].y));
            const unsigned long long dz = sub2(piz, pk2(pj[q].z, pj[q + 1].z));
            const unsigned long long rsq = dist2x2(dx, dy, dz);
            float ra, rb;
            upk2(rsq, ra, rb);
            float ta, tb;
            upk2(fma2(rsq, pk2(rsqrt_ftz(ra), rsqrt_ftz(rb)), nh), ta, tb);
            ta = fminf(ta, 0.f);
            tb = fminf(tb, 0.f);
            acc = __fmaf_rn(ta, ta, acc);
            acc = __fmaf_rn(tb, tb, acc);
#pragma unroll
            for (int h2 = 0; h2 < 2; ++h2) {
                const int eq = e[q + h2];
                if (eq < 0 && (h2 ? rb : ra) < rcf2) {
                    const int j = eq & kEntryIndexMask;
                    row2[min(n2, ncol2 - 1)] = UNI ? j : j | (ptype(pj[q + h2]) << kEntryTypeShift);
                    ++n2;
                }
            }
        }
    }
    if (live) {
        B.count2[i] = min(n2, ncol2);
        if (n2 > ncol2) atomicOr(&B.st->status, kErrList2Overflow);
        // a particle outside the density group keeps its rho (not written, as in the reference),
        // but its packed position is refreshed like every other
        const float r = in_group ? (float)(B.mass[ptype(pi)] * B.rho_factor) * acc : B.rho[i];
        if (in_group) B.rho[i] = r;
        B.posrho[i] = make_float4(pi.x, pi.y, pi.z, r);
        if (i >= B.st->n_bulk) {
            const int g1 = min(B.gfirst[i + 1], B.ghost_cap);
            for (int g = B.gfirst[i]; g < g1; ++g) {
                if (in_group) B.rho[B.nlocal + g] = r;
                const float4 pg = B.pos[B.nlocal + g];
                B.posrho[B.nlocal + g] = make_float4(pg.x, pg.y, pg.z, r);
            }
        }
    }
}

template <int kGather, bool UNI, int LPR>
__global__ void __launch_bounds__(128, density_blocks<kGather>()) k_density_rows(const BoxDesc *__restrict__ boxes,
                                                      const Unit *__restrict__ units, int nunits)
{
    const int u = blockIdx.x / LPR;
    if (u >= nunits) return;
    const Unit U = units[u];
    if (LPR == 1) {
        density_rows<kGather, UNI>(boxes[U.box], U);
    } else {
        const int first = U.begin + (blockIdx.x % LPR) * (128 / LPR);
        const BoxDesc &B = boxes[U.box];
        const int i0 = first + (threadIdx.x >> 5) * (32 / LPR);
        if (i0 < U.end)
            density_rows_split<kGather, UNI, LPR == 1 ? 2 : LPR, false>(B, i0, U.end, B.st->cur, B.st->n_bulk);
    }
}

// ---------------------------------------------------------------------------------------------
// force pass
// ---------------------------------------------------------------------------------------------
// shared memory of the force pass, RW rows per warp
template <int RW> struct RowsSmem {
    PairCoeff coeff[kMaxTypes * kMaxTypes];
    float4 pi[4 * RW], vi[4 * RW];
    float rho[4 * RW];
    int pre[4][33];
    unsigned lo[3][4 * RW], hi[3][4 * RW];
    double red[4][7];
    int ent[4][RW * kRowEntries];  // each warp's concatenated compact rows (when they fit)
};

template <bool EV>
__device__ __forceinline__ void ev_to_partial(const BoxDesc &B, const Unit &U, const EvAcc &ev, double (*red)[7])
{
    // every pair once, full weight (the reference halves each side's share)
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    double vals[8] = {ev.vxx, ev.vyy, ev.vzz, ev.vxy, ev.vxz, ev.vyz, ev.pe, 0.0};
    const double tot = warp_sum_spread(vals);  // the warp's total of value lane / 4
    if ((lane & 3) == 0 && (lane >> 2) < 7) red[w][lane >> 2] = tot;
    __syncthreads();
    if (t < 7) {
        double a = 0.0;
        for (int ww = 0; ww < 4; ++ww) a += red[ww][t];
        B.partial[(size_t)(U.begin / kUnit) * kPartialStride + 1 + t] = a;
    }
}

// rows [U.begin, U.end) of one block: 4 RW of them at most
template <bool EXACT, bool EV, bool UNI, int RW>
__device__ __forceinline__ void force_pairs(const BoxDesc &B, const Unit &U, RowsSmem<RW> &S, int stage_cap)
{
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, wb = w * RW;
    for (int q = t; q < (UNI ? 1 : B.ntype * B.ntype); q += blockDim.x) S.coeff[q] = B.coeff[q];
    // lanes below RW hold the warp's rows
    const int row = wb + lane, i = U.begin + row;
    const bool live = lane < RW && i < U.end;
    int len = 0;
    if (live) {
        prefetch_l2(B.table2 + (size_t)i * B.n_col2);  // the row's first 32 entries: one line
        S.pi[row] = B.pos[i];
        S.vi[row] = B.vel[i];
        S.rho[row] = B.rho[i];
        len = MDPD_IDX(B.count2[i], B.n_col2 + 1);
    }
    warp_prefix(len, lane, S.pre[w]);
    if (lane < RW)
        for (int c = 0; c < 3; ++c) S.lo[c][row] = S.hi[c][row] = 0u;
    __syncthreads();
    const int *P = S.pre[w];
    const int T = P[32];
    const int i0 = U.begin + wb, nlocal = B.nlocal, ntype = B.ntype, ncol2 = B.n_col2;
    const int m0 = (lane * T) >> 5, m1 = ((lane + 1) * T) >> 5;
    const float dtis = B.dt_inv_sqrt, fix_max = B.fix_pair_max;
    unsigned long long *fax = B.facc, *fay = B.facc + nlocal, *faz = B.facc + 2 * nlocal;
    EvAcc ev = {0, 0, 0, 0, 0, 0, 0};
    bool bad = false;
    // the warp's rows, concatenated, into shared memory: consecutive lanes load consecutive
    // entries (a row's entries are contiguous in the table), so the pair loop's entry reads,
    // one per lane in 32 different rows, come from shared memory instead of 32 table lines
    const bool staged = T <= stage_cap;  // warp-uniform; stage_cap is kWarpEntries, or 0 to read the table
    int *const ent = S.ent[w];
    if (staged) {
        for (int m = lane; m < T; m += 32) {
            const int r = row_of<RW>(P, m);
            ent[m] = __ldcs(B.table2 + (size_t)(i0 + r) * ncol2 + (m - P[r]));
        }
        __syncwarp();
    }
    if (m0 < m1) {
        int r = row_of<RW>(P, m0);
        int rbeg = P[r], rend = P[r + 1];
        float4 pi = S.pi[wb + r], vi = S.vi[wb + r];
        float rho_i = S.rho[wb + r];
        long long ax = 0, ay = 0, az = 0;
        // j's state for the next entry is loaded while the current pair is evaluated
        const int en = staged ? ent[m0] : __ldcs(B.table2 + (size_t)(i0 + r) * ncol2 + (m0 - rbeg));
        int jn = MDPD_IDX(en & kEntryIndex, n_all(B)), tn = en >> kEntryTypeShift;
        float4 pjn = __ldg(&B.posrho[jn]), vjn = __ldg(&B.vel[jn]);
        int srcn = jn < nlocal ? jn : MDPD_IDX(__ldg(&B.gsrc[jn - nlocal]), nlocal);
        for (int m = m0; m < m1; ++m) {
            if (m >= rend) {  // the share moves on to the next non-empty row
                sadd64(&S.lo[0][wb + r], &S.hi[0][wb + r], ax);
                sadd64(&S.lo[1][wb + r], &S.hi[1][wb + r], ay);
                sadd64(&S.lo[2][wb + r], &S.hi[2][wb + r], az);
                ax = ay = az = 0;
                do {
                    ++r;
                    rbeg = rend;
                    rend = P[r + 1];
                } while (m >= rend);
                pi = S.pi[wb + r], vi = S.vi[wb + r];
                rho_i = S.rho[wb + r];
            }
            const int src = srcn, tj = tn;
            const float4 pj = pjn, vj = vjn;  // pj.w: rho of j
            if (m + 1 < m1) {
                int e;
                if (staged) {
                    e = ent[m + 1];
                } else {
                    int rr = r, rb = rbeg, re = rend;  // entry m + 1: row r or a later non-empty row
                    while (m + 1 >= re) {
                        ++rr;
                        rb = re;
                        re = P[rr + 1];
                    }
                    e = __ldcs(B.table2 + (size_t)(i0 + rr) * ncol2 + (m + 1 - rb));
                }
                const int jj = MDPD_IDX(e & kEntryIndex, n_all(B));
                tn = e >> kEntryTypeShift;
                pjn = __ldg(&B.posrho[jj]);
                vjn = __ldg(&B.vel[jj]);
                srcn = jj < nlocal ? jj : MDPD_IDX(__ldg(&B.gsrc[jj - nlocal]), nlocal);
            }
            const PairCoeff &cf = S.coeff[UNI ? 0 : ptype(pi) * ntype + tj];
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float rsq = dist2(dx, dy, dz);
            float px = 0.f, py = 0.f, pz = 0.f;
            if (rsq < cf.cutsq && rsq >= 1e-20f)
                pair_core<0, EXACT, EV, false>(cf, dx, dy, dz, rsq, vi, vj, __float_as_uint(vi.w), rho_i, pj.w,
                                               false, 1.f, 1.f, dtis, px, py, pz, ev);
            bad |= !(fabsf(px) < fix_max && fabsf(py) < fix_max && fabsf(pz) < fix_max);
            const long long qx = to_fix(px), qy = to_fix(py), qz = to_fix(pz);
            ax += qx, ay += qy, az += qz;
            const int d = src - U.begin;
            if ((unsigned)d < (unsigned)(4 * RW)) {  // one of this block's rows (src < nlocal)
                sadd64(&S.lo[0][d], &S.hi[0][d], -qx);
                sadd64(&S.lo[1][d], &S.hi[1][d], -qy);
                sadd64(&S.lo[2][d], &S.hi[2][d], -qz);
            } else {
                atomicAdd(fax + src, (unsigned long long)(-qx));
                atomicAdd(fay + src, (unsigned long long)(-qy));
                atomicAdd(faz + src, (unsigned long long)(-qz));
            }
        }
        sadd64(&S.lo[0][wb + r], &S.hi[0][wb + r], ax);
        sadd64(&S.lo[1][wb + r], &S.hi[1][wb + r], ay);
        sadd64(&S.lo[2][wb + r], &S.hi[2][wb + r], az);
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&B.st->status, kErrNonFinite);
    __syncthreads();
    if (live) {
        atomicAdd(fax + i, join64(S.lo[0][row], S.hi[0][row]));
        atomicAdd(fay + i, join64(S.lo[1][row], S.hi[1][row]));
        atomicAdd(faz + i, join64(S.lo[2][row], S.hi[2][row]));
    }
    if (EV) ev_to_partial<EV>(B, U, ev, S.red);
}

// 7 blocks per SM (up to 72 registers, no spill) measured fastest against 6 and 8
template <bool EXACT, bool EV, bool UNI, int RW>
__global__ void __launch_bounds__(128, 7) k_force_pairs(const BoxDesc *__restrict__ boxes,
                                                        const Unit *__restrict__ units, int nunits, int staged)
{
    static_assert(!EV || RW == 32, "the energy and virial partials are per unit");
    __shared__ RowsSmem<RW> S;
    constexpr int kParts = 32 / RW;  // blocks per unit
    const int u = blockIdx.x / kParts;
    if (u >= nunits) return;
    Unit U = units[u];
    U.begin += (blockIdx.x % kParts) * (4 * RW);
    if (U.begin >= U.end) return;
    force_pairs<EXACT, EV, UNI, RW>(boxes[U.box], U, S, staged ? RW * kRowEntries : 0);
}

__global__ void __launch_bounds__(kUnit) k_finalize(const BoxDesc *__restrict__ boxes,
                                                    const Unit *__restrict__ units, int nunits, int kick)
{
    const int u = blockIdx.x;  // one unit per block: every load of the pass in flight at once
    if (u >= nunits) return;
    {
        const Unit U = units[u];
        const BoxDesc &B = boxes[U.box];
        const int i = U.begin + threadIdx.x;
        if (i >= U.end) return;
        if (i == 0) B.st->pending = 0;
        const int c = B.st->cur, n = B.nlocal;
        unsigned long long *fa = B.facc;
        // every load of the particle is issued before the first store (the compiler may not move
        // a load above a store to a possibly aliased array): one memory round trip, not four
        const long long ax = (long long)fa[i], ay = (long long)fa[n + i], az = (long long)fa[2 * n + i];
        const int m = B.mask[c][i], t = B.type[c][i];
        const double vx = B.v[c][0][i], vy = B.v[c][1][i], vz = B.v[c][2][i];
        const double dtfm = B.dtfm[t - 1];
        const float fx = (float)((double)ax * kFixInv);
        const float fy = (float)((double)ay * kFixInv);
        const float fz = (float)((double)az * kFixInv);
        fa[i] = 0ull, fa[n + i] = 0ull, fa[2 * n + i] = 0ull;
        B.f[i] = make_float4(fx, fy, fz, 0.f);  // the pair force; the body force is in the kicks
        if (kick && (m & B.nve_bit)) {
            const bool body = m & B.body_bit;
            B.v[c][0][i] = __fma_rn(dtfm, (double)fx + (body ? B.body[0] : 0.0), vx);
            B.v[c][1][i] = __fma_rn(dtfm, (double)fy + (body ? B.body[1] : 0.0), vy);
            B.v[c][2][i] = __fma_rn(dtfm, (double)fz + (body ? B.body[2] : 0.0), vz);
        }
    }
}

template <int G, bool UNI> static void density_launch(cudaStream_t s, BoxDesc *boxes, const UnitList &u, int lanes)
{
    switch (lanes) {
    case 8: k_density_rows<G, UNI, 8><<<u.n * 8, 128, 0, s>>>(boxes, u.d, u.n); break;
    case 4: k_density_rows<G, UNI, 4><<<u.n * 4, 128, 0, s>>>(boxes, u.d, u.n); break;
    case 2: k_density_rows<G, UNI, 2><<<u.n * 2, 128, 0, s>>>(boxes, u.d, u.n); break;
    default: k_density_rows<G, UNI, 1><<<u.n, 128, 0, s>>>(boxes, u.d, u.n); break;
    }
}

template <bool UNI>
static void density_gather(cudaStream_t s, BoxDesc *boxes, const UnitList &u, int gather, int lanes)
{
    switch (gather) {
    case 4: density_launch<4, UNI>(s, boxes, u, lanes); break;
    case 8: density_launch<8, UNI>(s, boxes, u, lanes); break;
    default: density_launch<6, UNI>(s, boxes, u, lanes); break;
    }
}

// Lanes per row of the density pass.  A row of ~42 entries takes 7 rounds of 6 gathers, each
// waiting for its entries and then their positions; while the chip is not full more lanes per row
// take fewer rounds: the most with which every block is still resident at once (8 per SM), 8
// lanes only at half of that (most rows are then one round).  With a full chip the shuffles that
// keep the sum in row order cost more than the rounds saved.  Density pass, us at 1 / 2 / 4 / 8
// lanes: 2,000 particles 11.7 / 10.3 / 7.9 / 6.4; 8,000 12.0 / 10.2 / 7.8 / 7.8; 20,000 11.9 /
// 11.5 / 9.9 / 11.5; 42,000 13.8 / 13.0 / 13.0 / 16.4; 100,000 19.6 / 23.1 / 24.4 / 30.4;
// 200,000 35.9 / 36.7 / 41.5 / 55.0.
static int density_lanes(int nunits, int sms)
{
    const int resident = 8 * sms;
    if (nunits * 16LL <= resident) return 8;
    if (nunits * 4LL <= resident) return 4;
    return nunits * 2LL <= resident ? 2 : 1;
}

void launch_density_half(cudaStream_t s, BoxDesc *boxes, const BatchUnits &u, const StepConfig &c)
{
    if (u.local.n <= 0) return;
    const int lanes = c.full_chip ? 1 : density_lanes(u.local.n, c.sms);
    if (c.uniform_types) density_gather<true>(s, boxes, u.local, c.gather, lanes);
    else density_gather<false>(s, boxes, u.local, c.gather, lanes);
}

template <bool EXACT, bool EV, bool UNI, int RW>
static void force_half(cudaStream_t s, BoxDesc *boxes, const BatchUnits &u, int staged)
{
    k_force_pairs<EXACT, EV, UNI, RW><<<u.local.n * (32 / RW), 128, 0, s>>>(boxes, u.local.d, u.local.n, staged);
}

// Rows per warp of the force pass.  A lane walks its share of the warp's pairs one after another
// (12.6 pairs at 32 rows and rho 6.05, ~2 us each with the loads they wait for), so while the
// chip is not full fewer rows per warp shorten the pass: the fewest with which every block is
// still resident at once (7 per SM).  Past that, up to a few resident waves, 16 rows lose less in
// the last wave; beyond, 32 rows are best: shares are evener, rows change less often and more
// partners are rows of the block, so fewer sums go through global atomics.  Force pass with
// finalize, us at 32 / 16 / 8 / 4 rows:
//       2,000 particles   32 /  21 /  15 /  13        8,000   32 /  21 /  17 /  14
//      20,000             32 /  22 /  17 /  20       42,000   33 /  25 /  26 /  27
//     200,000             72 /  64 /  70 /  87      500,000  137 / 134 / 160 / 207
//   1,000,000            252 / 255 / 320 / 421    4,000,000  888 / 955 / 1242 / 1645
// (a 109,000-particle slab, 0.8 waves at 32 rows: 1 us a step slower at 16).
// The sums are fixed point, so every shape gives the same bits.
static int force_rows(int nunits, int sms)
{
    const int resident = 7 * sms;
    if (nunits * 8LL <= resident) return 4;
    if (nunits * 4LL <= resident) return 8;
    if (nunits * 2LL <= resident) return 16;
    return nunits > resident && nunits <= 4LL * resident ? 16 : 32;
}

template <bool EXACT, bool UNI>
static void force_half_rows(cudaStream_t s, BoxDesc *boxes, const BatchUnits &u, int rows, int staged)
{
    switch (rows) {
    case 4: force_half<EXACT, false, UNI, 4>(s, boxes, u, staged); break;
    case 8: force_half<EXACT, false, UNI, 8>(s, boxes, u, staged); break;
    case 16: force_half<EXACT, false, UNI, 16>(s, boxes, u, staged); break;
    default: force_half<EXACT, false, UNI, 32>(s, boxes, u, staged); break;
    }
}

void launch_force_half(cudaStream_t s, BoxDesc *boxes, const BatchUnits &u, const StepConfig &c, int ev, int kick,
                       bool finish)
{
    const int g = u.local.n;
    if (g <= 0) return;
    const int staged = c.stage_rows;
    const int rows = c.full_chip ? 32 : force_rows(u.local.n, c.sms);
    if (ev) {
        if (c.exact_rng) force_half<true, true, false, 32>(s, boxes, u, staged);
        else force_half<false, true, false, 32>(s, boxes, u, staged);
    } else if (c.exact_rng) {
        if (c.uniform_types) force_half_rows<true, true>(s, boxes, u, rows, staged);
        else force_half_rows<true, false>(s, boxes, u, rows, staged);
    } else {
        if (c.uniform_types) force_half_rows<false, true>(s, boxes, u, rows, staged);
        else force_half_rows<false, false>(s, boxes, u, rows, staged);
    }
    if (finish) launch_finalize(s, boxes, u, kick);
}

void launch_finalize(cudaStream_t s, BoxDesc *boxes, const BatchUnits &u, int kick)
{
    if (u.local.n > 0) k_finalize<<<u.local.n, kUnit, 0, s>>>(boxes, u.local.d, u.local.n, kick);
}

}  // namespace mdpd
