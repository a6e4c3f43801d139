// Row-wise parts of the pair passes, shared by their kernels (k_pair.cu, k_step.cu) and the
// whole-run kernel of small boxes (k_small.cu).
#pragma once

#include "pair.cuh"

namespace mdpd {

constexpr float kFixF = 4294967296.0f;           // 2^32
constexpr int kEntryTypeShift = 27;              // compact entry: j | (type of j - 1) << 27
constexpr int kEntryIndex = (1 << kEntryTypeShift) - 1;

// a gather of data that no thread of this kernel writes (read-only path), or, COH, that it does
template <bool COH, class T> __device__ __forceinline__ T gather(const T *p)
{
    if (COH) return *p;
    return __ldg(p);
}

// approximate 1/sqrt(x), denormal inputs taken as 0 (which gives +inf)
__device__ __forceinline__ float rsqrt_ftz(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The same rows with LPR lanes each (32 / LPR rows per warp): lane s of a row takes entries
// s, s + LPR, ..., so a row waits for LPR times fewer rounds of loads, and the terms are added in
// row order through shuffles (every lane of the row forms the whole sum): the same bits as one
// lane per row.  i0: the warp's first row, in buffer c;
// COH: positions written by this kernel (plain loads).
template <int kGather, bool UNI, int LPR, bool COH>
__device__ __forceinline__ void density_rows_split(const BoxDesc &B, int i0, int end, int c, int n_bulk)
{
    constexpr int R = 32 / LPR;  // rows per warp: lane = s * R + r
    static_assert(kGather % 2 == 0 && kGather * LPR <= 64, "two entries at a time; a round within two list lines");
    const int lane = threadIdx.x & 31, s = lane / R, r = lane % R;
    const int i = i0 + r;
    const bool live = i < end;
    const int self = live ? i : i0;
    const int ncol = B.n_col, ncol2 = B.n_col2, nlocal = B.nlocal;
    const int *row = B.table + ((unsigned)(self & ~31) * (unsigned)ncol + (unsigned)(self & 31));  // entry k at 32 k
    // the first round's entries are read beside the row length (a row holds at least 32 entries;
    // those past its length are dropped below)
    int e[kGather];
#pragma unroll
    for (int q = 0; q < kGather; ++q) e[q] = q * LPR + s < ncol ? __ldcs(row + 32 * (q * LPR + s)) : 0;
    const bool in_group = live && (B.mask[c][self] & B.rho_bit);
    const int n = live ? MDPD_IDX(B.count[self], ncol + 1) : 0;
    const float4 pi = B.pos[self];
    const bool edge = live && self >= n_bulk;
    const int g0 = edge ? B.gfirst[self] : 0, g1 = edge ? min(B.gfirst[self + 1], B.ghost_cap) : 0;
    const int nmax = __reduce_max_sync(0xffffffffu, n);
    const float h = B.cut_rho, rcf2 = B.rc2_force;
    const unsigned long long pix = pk2(pi.x, pi.x), piy = pk2(pi.y, pi.y), piz = pk2(pi.z, pi.z);
    const unsigned long long nh = pk2(-h, -h);
    int *row2 = B.table2 + (size_t)self * ncol2;
    unsigned mine = 0;  // the lanes of this row
#pragma unroll
    for (int q = 0; q < LPR; ++q) mine |= 1u << (q * R);
    mine <<= r;
    const unsigned before = mine & ((1u << lane) - 1u);
    float acc = 0.f;
    int n2 = 0;
    for (int k0 = 0; k0 < nmax; k0 += kGather * LPR) {
        float4 pj[kGather];
#pragma unroll
        for (int q = 0; q < kGather; ++q) {
            const int k = k0 + q * LPR + s;
            if (k0 != 0) e[q] = k < n ? __ldcs(row + 32 * k) : self;
            else if (k >= n) e[q] = self;
        }
#pragma unroll
        for (int q = 0; q < kGather; ++q) pj[q] = gather<COH>(&B.pos[MDPD_IDX(e[q] & kEntryIndexMask, n_all(B))]);
#pragma unroll
        for (int q = 0; q < kGather; q += 2) {
            const unsigned long long dx = sub2(pix, pk2(pj[q].x, pj[q + 1].x));
            const unsigned long long dy = sub2(piy, pk2(pj[q].y, pj[q + 1].y));
            const unsigned long long dz = sub2(piz, pk2(pj[q].z, pj[q + 1].z));
            const unsigned long long rsq = dist2x2(dx, dy, dz);
            float rr[2], t[2];
            upk2(rsq, rr[0], rr[1]);
            upk2(fma2(rsq, pk2(rsqrt_ftz(rr[0]), rsqrt_ftz(rr[1])), nh), t[0], t[1]);
#pragma unroll
            for (int h2 = 0; h2 < 2; ++h2) {
                const float tm = fminf(t[h2], 0.f);
#pragma unroll
                for (int q2 = 0; q2 < LPR; ++q2) {
                    const float tq = __shfl_sync(0xffffffffu, tm, q2 * R + r);
                    acc = __fmaf_rn(tq, tq, acc);
                }
                const int eq = e[q + h2];
                const bool hit = eq < 0 && rr[h2] < rcf2;
                const unsigned b = __ballot_sync(0xffffffffu, hit);
                if (hit) {
                    const int j = eq & kEntryIndexMask;
                    row2[min(n2 + __popc(b & before), ncol2 - 1)] = UNI ? j : j | (ptype(pj[q + h2]) << kEntryTypeShift);
                }
                n2 += __popc(b & mine);
            }
        }
    }
    if (live) {
        const float rho = in_group ? (float)(B.mass[ptype(pi)] * B.rho_factor) * acc : B.rho[i];
        if (s == 0) {
            B.count2[i] = min(n2, ncol2);
            if (n2 > ncol2) atomicOr(&B.st->status, kErrList2Overflow);
            if (in_group) B.rho[i] = rho;
            B.posrho[i] = make_float4(pi.x, pi.y, pi.z, rho);
        }
        for (int g = g0 + s; g < g1; g += LPR) {
            if (in_group) B.rho[nlocal + g] = rho;
            const float4 pg = B.pos[nlocal + g];
            B.posrho[nlocal + g] = make_float4(pg.x, pg.y, pg.z, rho);
        }
    }
}

__device__ __forceinline__ long long to_fix(float v) { return __float2ll_rn(v * kFixF); }

// 64-bit fixed-point add into a shared (lo, hi) pair of 32-bit words with native 32-bit
// atomics: the low word's wrap-arounds carry into the high word, so the pair ends as the exact
// 64-bit sum (mod 2^64) whatever the order of the adds
__device__ __forceinline__ void sadd64(unsigned *lo, unsigned *hi, long long q)
{
    const unsigned ql = (unsigned)q, qh = (unsigned)((unsigned long long)q >> 32);
    const unsigned old = atomicAdd(lo, ql);
    atomicAdd(hi, qh + (old + ql < old ? 1u : 0u));
}

__device__ __forceinline__ unsigned long long join64(unsigned lo, unsigned hi)
{
    return ((unsigned long long)hi << 32) | lo;
}

// the warp's rows as one list of T entries split into 32 equal shares; P: prefix of the row
// lengths (P[r] entries before row r, P[32] = T; len is 0 in lanes that hold no row)
__device__ __forceinline__ void warp_prefix(int len, int lane, int *P)
{
    int pre = len;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += v;
    }
    P[lane + 1] = pre;
    if (lane == 0) P[0] = 0;
}

// the row (of RW) holding entry m of the concatenated rows: the last r with P[r] <= m
template <int RW> __device__ __forceinline__ int row_of(const int *P, int m)
{
    int r = 0;
#pragma unroll
    for (int st = RW / 2; st > 0; st >>= 1)
        if (P[r + st] <= m) r += st;
    return r;
}

// compact entries a warp stages in shared memory per row: rows hold 12.6 owned force-range pairs
// at rho 6.05; a warp with more than RW times this reads them from the table
constexpr int kRowEntries = 20;

// ---------------------------------------------------------------------------------------------
// Classic DPD pair forces of up to R = 32 / LPR rows by one warp, for boxes too small to give every
// row a thread of its own and still fill the chip:
//   test   LPR lanes per row find the entries in range and queue them in list order,
//   pairs  lane l takes pairs l, l + 32, ... of the queued rows, concatenated, and leaves each
//          pair's vector and force in shared memory,
//   sum    a lane per row adds its pairs in list order: the sums, and their bits, of k_force's one
//          thread per row.
// s_pos, s_vel: position and velocity of the block's rows (base onwards); r0: the warp's first row.
// f: the force on row r0 + lane (lanes below R).
// ---------------------------------------------------------------------------------------------
constexpr int kRowQueue = 32;    // queued pairs per row
constexpr int kPairChunk = 128;  // pairs summed at a time

struct FullRowsSmem {
    float4 res[kPairChunk];
    int pre[36];
    int q[16 * (kRowQueue + 1)];
};

template <bool EXACT, bool UNI, int LPR, bool COH>
__device__ __forceinline__ void full_rows(const BoxDesc &B, const float4 *s_pos, const float4 *s_vel, int base, int r0,
                                          int nrows, FullRowsSmem &S, float f[3])
{
    constexpr int R = 32 / LPR, G = LPR >= 16 ? 32 / LPR : 4;  // G: gathers in flight per lane
    static_assert(R <= 16 && G * LPR <= kRowQueue, "a round fits the empty queue");
    const int lane = threadIdx.x & 31, r = lane % R, s = lane / R;
    const bool live = r0 + r < nrows;
    const int self = base + (live ? r0 + r : r0);
    const float4 pi = s_pos[live ? r0 + r : r0];
    const int ti = ptype(pi), ntype = B.ntype;
    const int n = live ? MDPD_IDX(B.count[self], B.n_col + 1) : 0;
    const int ncol = B.n_col;
    const int *row = B.table + ((unsigned)(self & ~31) * (unsigned)ncol + (unsigned)(self & 31));
    const int nmax = __reduce_max_sync(0xffffffffu, n);
    const float dtis = B.dt_inv_sqrt;
    unsigned mine = 0;  // the lanes of this row
#pragma unroll
    for (int q = 0; q < LPR; ++q) mine |= 1u << (q * R);
    mine <<= r;
    const unsigned before = mine & ((1u << lane) - 1u);
    int *const queue = S.q + r * (kRowQueue + 1);
    float fx = 0.f, fy = 0.f, fz = 0.f;
    for (int k0 = 0; k0 < nmax;) {
        int cnt = 0;  // queued pairs of the row
        for (; k0 < nmax; k0 += G * LPR) {
            if (__any_sync(0xffffffffu, cnt + G * LPR > kRowQueue)) break;
            int j[G];
            float4 pj[G];
#pragma unroll
            for (int q = 0; q < G; ++q) {
                const int k = k0 + q * LPR + s;
                j[q] = k < n ? MDPD_IDX(__ldcs(row + 32 * k) & kEntryIndexMask, n_all(B)) : -1;
            }
#pragma unroll
            for (int q = 0; q < G; ++q) pj[q] = j[q] >= 0 ? gather<COH>(&B.pos[j[q]]) : make_float4(1e30f, 0, 0, 0);
#pragma unroll
            for (int q = 0; q < G; ++q) {
                const float dx = pi.x - pj[q].x, dy = pi.y - pj[q].y, dz = pi.z - pj[q].z;
                const float rsq = dist2(dx, dy, dz);
                const bool hit = j[q] >= 0 && rsq < B.coeff[UNI ? 0 : ti * ntype + ptype(pj[q])].cutsq && rsq >= 1e-20f;
                const unsigned b = __ballot_sync(0xffffffffu, hit);
                if (hit) queue[cnt + __popc(b & before)] = j[q];
                cnt += __popc(b & mine);
            }
        }
        // the queued rows as one list of T pairs: pre[r] of them before row r
        int pre = lane < R ? cnt : 0;
#pragma unroll
        for (int o = 1; o < R; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += v;
        }
        if (lane < R) S.pre[r + 1] = pre;
        if (lane == 0) S.pre[0] = 0;
        __syncwarp();
        const int T = S.pre[R];
        int rr = 0, beg = 0, end = S.pre[1];  // the row of this lane's pair
        for (int c0 = 0; c0 < T; c0 += kPairChunk) {
            const int c1 = min(T, c0 + kPairChunk);
            for (int m = c0 + lane; m < c1; m += 32) {
                while (m >= end) {
                    ++rr;
                    beg = end;
                    end = S.pre[rr + 1];
                }
                const int j = S.q[rr * (kRowQueue + 1) + m - beg];
                const float4 pj = gather<COH>(&B.pos[j]), vj = gather<COH>(&B.vel[j]);
                const float4 p = s_pos[r0 + rr], v = s_vel[r0 + rr];
                const float dx = p.x - pj.x, dy = p.y - pj.y, dz = p.z - pj.z;
                EvAcc ev;
                const float fp = pair_scalar<1, EXACT, false, false>(
                    B.coeff[UNI ? 0 : ptype(p) * ntype + ptype(pj)], dx, dy, dz, dist2(dx, dy, dz), v, vj,
                    __float_as_uint(v.w), 0.f, 0.f, false, 1.f, 1.f, dtis, ev);
                S.res[m - c0] = make_float4(dx, dy, dz, fp);
            }
            __syncwarp();
            if (lane < R)
                for (int m = max(S.pre[r], c0), m1 = min(S.pre[r + 1], c1); m < m1; ++m) {
                    const float4 t = S.res[m - c0];
                    fx = __fmaf_rn(t.x, t.w, fx);
                    fy = __fmaf_rn(t.y, t.w, fy);
                    fz = __fmaf_rn(t.z, t.w, fz);
                }
            __syncwarp();
        }
    }
    f[0] = fx, f[1] = fy, f[2] = fz;
}

}  // namespace mdpd
