// Whole runs of one small box: many steps in one cooperative launch.
//
// A small box's step is a chain of passes that each wait on memory a few times and do little work:
// launched one by one (3 kernels, 9 more at a rebuild) a 2,000-particle box took 46 us a step.  Here one
// block per SM owns a contiguous range of rows for the whole run and the passes follow one another
// behind grid barriers (~1 us):
//   integrate   (the last step's final half-kick,) half-kick, drift, pack, ghosts   | barrier
//   decide      every block reads the displacement flag and decides alike
//   rebuild     the passes of k_rebuild.cu on the same device code                   | 9 barriers
//   density     2 to 32 lanes per row (mDPD)                                         | barrier
//   force       mDPD: the block's pairs shared out over each warp, own rows summed in shared
//               memory, partners in other blocks by global atomics; DPD: rows summed in list
//               order                                                                | barrier
// The arithmetic and every order that matters are those of the per-pass kernels, so a box has the
// same bits on either path.  Rows of the block (position, velocity, density, force sums) stay in
// shared memory between its passes.
//
// Every barrier wait is bounded: a block that waits too long raises the run's abort flag, and every
// block that finds it leaves the kernel and sets the box's kErrTimeout status.  The box may then be
// between two passes (bucket counts of half a rebuild): later runs return at once, and the other passes
// do not rebuild such a box (its lists of the last build stay in bounds).
#include "kernels.h"
#include "pair_rows.cuh"
#include "rebuild.cuh"

#include <algorithm>

namespace mdpd {

constexpr int kSmallWarps = 24, kSmallThreads = 32 * kSmallWarps;

struct SmallBar {
    unsigned arrived;
    int abort;
    int moved[3];  // displacement flags of steps k, k + 1, k + 2 (mod 3)
    int next;      // the list build's next item
};

struct SmallArgs {
    BoxDesc B;
    SmallBar *bar;
    int *done;
    int nsteps, rows, parts, nblocks;
    unsigned polls;     // of a barrier wait, at most
    unsigned withhold;  // the barrier target from which on one arrival more is waited for (tests)
};

// all blocks of the grid; false when the wait ran out or another block's did.  s_flag[1]: the word at
// `also` after the barrier (read by the thread that waits)
__device__ __forceinline__ bool grid_barrier(const SmallArgs &A, unsigned &target, int *s_flag, const int *also)
{
    SmallBar *const bar = A.bar;
    target += (unsigned)A.nblocks;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&bar->arrived) : "memory");
        const unsigned want = target + (target >= A.withhold ? 1u : 0u);
        unsigned seen, polls = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&bar->arrived) : "memory");
            if ((int)(seen - want) >= 0) break;
            if ((++polls & 1023u) == 0 && (polls >= A.polls || *(volatile int *)&bar->abort)) {
                *(volatile int *)&bar->abort = 1;
                ok = 0;
                break;
            }
        }
        s_flag[0] = ok;
        if (also) s_flag[1] = *(const volatile int *)also;
    }
    __syncthreads();
    return s_flag[0] != 0;
}

__device__ __forceinline__ int block_sum(int a, int *s_w)
{
    a = __reduce_add_sync(0xffffffffu, a);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x / 32] = a;
    __syncthreads();
    int t = 0;
    for (int w = 0; w < kSmallWarps; ++w) t += s_w[w];
    __syncthreads();
    return t;
}

// Exclusive scan of in[first, n), one chunk per block, in out[first, n + extra): a block adds up what
// comes before its chunk itself.  f(k, sum) stores; returns the total in the block with the last chunk
// (else -1).
template <class F>
__device__ __forceinline__ int scan_chunk(const int *in, int first, int n, int extra, int nblocks, int *s_w, F &&f)
{
    const int len = n + extra - first, chunk = (len + nblocks - 1) / nblocks;
    const int beg = first + blockIdx.x * chunk, end = min(n + extra, beg + chunk);
    if (beg >= end) return -1;
    int before = 0;
#pragma unroll 8
    for (int k = first + threadIdx.x; k < beg; k += kSmallThreads) before += in[k];
    int carry = block_sum(before, s_w);
    if (threadIdx.x < 32) {
        for (int k0 = beg; k0 < end; k0 += 32) {
            const int k = k0 + threadIdx.x, v = k < n ? in[k] : 0;
            int x = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if ((int)threadIdx.x >= o) x += y;
            }
            if (k < end) f(k, carry + x - v);
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    return end == n + extra ? carry : -1;  // valid in warp 0
}

// shared memory of a block: the rows it owns, then scratch of the passes
struct SmallSmem {
    float4 *pos, *vel;
    float *rho;
    unsigned *acc[6];  // mDPD: lo and hi words of the force sums' components; DPD: three floats each
    char *scratch;
};

__host__ __device__ __forceinline__ int small_row_bytes(int rows) { return ((rows * 60 + 127) & ~127); }
constexpr int kPreBytes = 36 * 4;  // prefix of up to 32 row lengths
// one warp's scratch: the list build's, a bucket's keys, or a force pass's staged rows
constexpr int kSmallScratch = sizeof(ListSmem) > kClassMax * 8 ? sizeof(ListSmem) : kClassMax * 8;
static_assert(kSmallScratch % 16 == 0 && sizeof(FullRowsSmem) <= kSmallScratch, "float4 members; the passes' scratch");

__device__ __forceinline__ SmallSmem small_smem(char *p, int rows)
{
    SmallSmem S;
    S.pos = reinterpret_cast<float4 *>(p);
    S.vel = S.pos + rows;
    S.rho = reinterpret_cast<float *>(S.vel + rows);
    for (int c = 0; c < 6; ++c) S.acc[c] = reinterpret_cast<unsigned *>(S.rho + rows * (c + 1));
    S.scratch = p + small_row_bytes(rows);
    return S;
}

// one step's force on the block's row r as FP64 of the FP32 pair force
template <int STYLE>
__device__ __forceinline__ void row_force(const BoxDesc &B, const SmallSmem &S, int r, int i, double f[3])
{
    for (int d = 0; d < 3; ++d) {
        if (STYLE == 0) {
            const long long q = (long long)(B.facc[(size_t)d * B.nlocal + i] + join64(S.acc[d][r], S.acc[3 + d][r]));
            f[d] = (double)(float)((double)q * kFixInv);
        } else {
            f[d] = (double)__uint_as_float(S.acc[d][r]);
        }
    }
}

template <int STYLE>
__device__ __forceinline__ void clear_force(const BoxDesc &B, const SmallSmem &S, int r, int i)
{
    for (int d = 0; d < 3; ++d) {
        if (STYLE == 0) B.facc[(size_t)d * B.nlocal + i] = 0ull;
        S.acc[d][r] = S.acc[3 + d][r] = 0u;
    }
}

// integrate's particle i (row r of the block); returns whether it moved more than skin / 2.
// pending: the last step's forces are to be applied first (its final half-kick)
template <int STYLE>
__device__ __forceinline__ bool small_integrate(const BoxDesc &B, const SmallSmem &S, int r, int i, int c, int n_bulk,
                                                bool pending, uint32_t sn)
{
    const int t = B.type[c][i], m = B.mask[c][i], tag = B.tag[c][i];
    double x[3], v[3], f[3], h[3];
    for (int d = 0; d < 3; ++d) x[d] = B.x[c][d][i], v[d] = B.v[c][d][i], h[d] = B.xh[d][i];
    if (pending) {
        row_force<STYLE>(B, S, r, i, f);
    } else {
        const float4 f4 = B.f[i];
        f[0] = f4.x, f[1] = f4.y, f[2] = f4.z;
    }
    const bool edge = i >= n_bulk;
    const int g0 = edge ? B.gfirst[i] : 0, g1 = edge ? min(B.gfirst[i + 1], B.ghost_cap) : 0;
    int code[7];  // image codes: 7 ghosts at most (a box side is at least three cutoffs)
#pragma unroll
    for (int q = 0; q < 7; ++q) code[q] = g0 + q < g1 ? B.gimg[g0 + q] : 13;
    const uint32_t sg0 = STYLE == 0 ? sig_mdpd(tag, sn) : 0u;
    if (pending) clear_force<STYLE>(B, S, r, i);
    if (m & B.nve_bit) {
        const double dtfm = B.dtfm[t - 1];
        const bool body = m & B.body_bit;
        for (int d = 0; d < 3; ++d) {
            const double ft = f[d] + (body ? B.body[d] : 0.0);
            if (pending) v[d] = __fma_rn(dtfm, ft, v[d]);
            v[d] = __fma_rn(dtfm, ft, v[d]);
            x[d] = __fma_rn(B.dtv, v[d], x[d]);
        }
    }
    for (int d = 0; d < 3; ++d) B.v[c][d][i] = v[d], B.x[c][d][i] = x[d];
    const double ddx = x[0] - h[0], ddy = x[1] - h[1], ddz = x[2] - h[2];
    const float w = pack_w(B, t, m);
    const float4 p = make_float4((float)(x[0] - B.cen[0]), (float)(x[1] - B.cen[1]), (float)(x[2] - B.cen[2]), w);
    const float fvx = (float)v[0], fvy = (float)v[1], fvz = (float)v[2];
    const uint32_t sg = STYLE == 0 ? sg0 : sig_dpd(tag, fvx, fvy, fvz, sn);
    const float4 vv = make_float4(fvx, fvy, fvz, __uint_as_float(sg));
    B.pos[i] = S.pos[r] = p;
    B.vel[i] = S.vel[r] = vv;
#pragma unroll
    for (int q = 0; q < 7; ++q)
        if (g0 + q < g1) put_ghost(B, g0 + q, code[q], x[0], x[1], x[2], w, vv);
    return ddx * ddx + ddy * ddy + ddz * ddz > B.triggersq;
}

// mDPD pairs of the block's rows (the per-pass kernel's scheme, with the rows of the whole block in
// shared memory): each warp's compact rows split into 32 equal shares; own partners by shared-memory
// atomics, the others' sums by global ones
template <bool EXACT, bool UNI>
__device__ __forceinline__ void small_force(const BoxDesc &B, const SmallSmem &S, int base, int nrows, int rows_warp)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wb = w * rows_warp;
    const int mine = min(rows_warp, nrows - wb);  // this warp's rows
    if (mine <= 0) return;
    int *const P = reinterpret_cast<int *>(S.scratch + w * kSmallScratch);
    int *const ent = P + 36;
    const int cap = (kSmallScratch - kPreBytes) / 4;
    warp_prefix(lane < mine ? MDPD_IDX(B.count2[base + wb + lane], B.n_col2 + 1) : 0, lane, P);
    __syncwarp();
    const int T = P[32], i0 = base + wb, nlocal = B.nlocal, ntype = B.ntype, ncol2 = B.n_col2;
    const bool staged = T <= cap;
    if (staged) {
        for (int m = lane; m < T; m += 32) {
            const int r = row_of<32>(P, m);
            ent[m] = __ldcs(B.table2 + (size_t)(i0 + r) * ncol2 + (m - P[r]));
        }
        __syncwarp();
    }
    const int m0 = (lane * T) >> 5, m1 = ((lane + 1) * T) >> 5;
    const float dtis = B.dt_inv_sqrt, fix_max = B.fix_pair_max;
    unsigned long long *fax = B.facc, *fay = B.facc + nlocal, *faz = B.facc + 2 * nlocal;
    EvAcc ev;
    bool bad = false;
    if (m0 < m1) {
        int r = row_of<32>(P, m0), rend = P[r + 1];
        float4 pi = S.pos[wb + r], vi = S.vel[wb + r];
        float rho_i = S.rho[wb + r];
        long long ax = 0, ay = 0, az = 0;
        auto load = [&](int m, int rr, int &tj, float4 &pj, float4 &vj, int &src) {
            const int e = staged ? ent[m] : __ldcs(B.table2 + (size_t)(i0 + rr) * ncol2 + (m - P[rr]));
            const int j = MDPD_IDX(e & kEntryIndex, n_all(B));
            tj = e >> kEntryTypeShift;
            pj = B.posrho[j], vj = B.vel[j];
            src = j < nlocal ? j : MDPD_IDX(B.gsrc[j - nlocal], nlocal);
        };
        int tn, srcn;
        float4 pjn, vjn;
        load(m0, r, tn, pjn, vjn, srcn);
        for (int m = m0; m < m1; ++m) {
            if (m >= rend) {
                sadd64(&S.acc[0][wb + r], &S.acc[3][wb + r], ax);
                sadd64(&S.acc[1][wb + r], &S.acc[4][wb + r], ay);
                sadd64(&S.acc[2][wb + r], &S.acc[5][wb + r], az);
                ax = ay = az = 0;
                do {
                    ++r;
                    rend = P[r + 1];
                } while (m >= rend);
                pi = S.pos[wb + r], vi = S.vel[wb + r];
                rho_i = S.rho[wb + r];
            }
            const int src = srcn, tj = tn;
            const float4 pj = pjn, vj = vjn;  // pj.w: rho of j
            if (m + 1 < m1) {
                int rr = r;
                if (!staged)
                    while (m + 1 >= P[rr + 1]) ++rr;
                load(m + 1, rr, tn, pjn, vjn, srcn);
            }
            const PairCoeff &cf = B.coeff[UNI ? 0 : ptype(pi) * ntype + tj];
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float rsq = dist2(dx, dy, dz);
            float px = 0.f, py = 0.f, pz = 0.f;
            if (rsq < cf.cutsq && rsq >= 1e-20f)
                pair_core<0, EXACT, false, false>(cf, dx, dy, dz, rsq, vi, vj, __float_as_uint(vi.w), rho_i, pj.w, false,
                                                  1.f, 1.f, dtis, px, py, pz, ev);
            bad |= !(fabsf(px) < fix_max && fabsf(py) < fix_max && fabsf(pz) < fix_max);
            const long long qx = to_fix(px), qy = to_fix(py), qz = to_fix(pz);
            ax += qx, ay += qy, az += qz;
            const int d = src - base;
            if ((unsigned)d < (unsigned)nrows) {
                sadd64(&S.acc[0][d], &S.acc[3][d], -qx);
                sadd64(&S.acc[1][d], &S.acc[4][d], -qy);
                sadd64(&S.acc[2][d], &S.acc[5][d], -qz);
            } else {
                atomicAdd(fax + src, (unsigned long long)(-qx));
                atomicAdd(fay + src, (unsigned long long)(-qy));
                atomicAdd(faz + src, (unsigned long long)(-qz));
            }
        }
        sadd64(&S.acc[0][wb + r], &S.acc[3][wb + r], ax);
        sadd64(&S.acc[1][wb + r], &S.acc[4][wb + r], ay);
        sadd64(&S.acc[2][wb + r], &S.acc[5][wb + r], az);
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&B.st->status, kErrNonFinite);
}

// STYLE 0: mDPD (pair-once), 1: classic DPD; LPR: lanes per row of the density pass and of the DPD
// pass's distance tests
template <int STYLE, bool EXACT, bool UNI, int LPR>
__global__ void __launch_bounds__(kSmallThreads, 1) k_run_box(const __grid_constant__ SmallArgs A)
{
    extern __shared__ __align__(128) char s_dyn[];
    __shared__ uint32_t s_seed[kSmallRunSteps + 2];
    __shared__ int s_w[kSmallWarps];
    __shared__ int s_flag[2];
    const BoxDesc &B = A.B;
    const SmallSmem S = small_smem(s_dyn, A.rows);
    constexpr int R = 32 / LPR;                   // rows per warp and round
    constexpr int G = LPR >= 32 ? 2 : LPR >= 8 ? 8 : 6;  // positions in flight per lane, at most 64 entries
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int n = B.nlocal, base = blockIdx.x * A.rows, nrows = max(0, min(A.rows, n - base));
    const int warps = A.nblocks * kSmallWarps, gw = w * A.nblocks + blockIdx.x;  // spread over the SMs
    const int rows_warp = (A.rows + kSmallWarps - 1) / kSmallWarps;
    unsigned target = 0;
    const BoxState S0 = *B.st;  // block-uniform; block 0 writes it back at the end
    int cur = S0.cur, n_bulk = S0.n_bulk, ago = S0.ago, builds = 0, rb = 0;
    for (int k = tid; k < A.nsteps + 2; k += kSmallThreads) s_seed[k] = seed_now(B.seed, S0.step + k);
    for (int r = tid; r < nrows; r += kSmallThreads)
        for (int d = 0; d < 6; ++d) S.acc[d][r] = 0u;
    if (tid == 0) s_flag[0] = !(S0.status & kErrTimeout);  // an earlier run gave up: nothing is done
    __syncthreads();
    auto barrier = [&](const int *also = nullptr) { return grid_barrier(A, target, s_flag, also); };
    bool ok = s_flag[0] != 0;
    for (int k = 0; k < A.nsteps && ok; ++k) {
        const uint32_t sn = s_seed[k + 1];
        bool moved = false;
        for (int r = tid; r < nrows; r += kSmallThreads)
            moved |= small_integrate<STYLE>(B, S, r, base + r, cur, n_bulk, k > 0, sn);
        if (__any_sync(0xffffffffu, moved) && lane == 0) atomicOr(&A.bar->moved[k % 3], 1);
        // the flag after next's slot: last read before this step's first barrier of the step before
        if (blockIdx.x == 0 && tid == 0) A.bar->moved[(k + 1) % 3] = 0;
        if (!(ok = barrier(&A.bar->moved[k % 3]))) break;
        const int any = s_flag[1];
        ++ago;
        rb = 0;
        if (ago >= B.delay && ago % B.every == 0) rb = B.check ? any : 1;
        if (rb) {
            ago = 0;
            ++builds;
            if (blockIdx.x == 0 && tid == 0) A.bar->next = 0;
            for (int r = tid; r < nrows; r += kSmallThreads) key_particle(B, base + r, cur);
            if (!(ok = barrier())) break;
            {
                const int tot = scan_chunk(B.cls_count, 0, 2 * B.nbin, 0, A.nblocks, s_w, [&](int q, int ex) {
                    B.cls_start[q] = ex;
                    B.cls_cursor[q] = ex;
                });
                if (tid == 0 && tot >= 0) B.cls_start[2 * B.nbin] = tot;
            }
            if (!(ok = barrier())) break;
            for (int r = tid; r < nrows; r += kSmallThreads) {
                const int p = warp_add1(B.cls_cursor, MDPD_IDX(B.cls_of[base + r], 2 * B.nbin));
                B.perm[MDPD_IDX(p, n)] = base + r;
            }
            if (!(ok = barrier())) break;
            for (int b0 = 4 * gw; b0 < 2 * B.nbin; b0 += 4 * warps)
                bucket_four<0>(B, b0, 2 * B.nbin, reinterpret_cast<unsigned long long *>(S.scratch + w * kSmallScratch));
            if (!(ok = barrier())) break;
            n_bulk = B.cls_start[B.nbin];
            for (int r = tid; r < nrows; r += kSmallThreads) {
                permute_particle<STYLE>(B, base + r, cur, sn);
                S.pos[r] = B.pos[base + r];
                S.vel[r] = B.vel[base + r];
            }
            cur = 1 - cur;
            if (!(ok = barrier())) break;
            {
                const int cap = n + B.ghost_cap;
                int tot = scan_chunk(B.cls_of, n_bulk, n, 1, A.nblocks, s_w, [&](int q, int ex) { B.gfirst[q] = ex; });
                if (tid == 0 && tot >= 0) B.st->nghost = tot;
                __syncthreads();
                tot = scan_chunk(B.bin_count, 0, B.nbin, 0, A.nblocks, s_w, [&](int q, int ex) {
                    B.bin_start[q] = min(ex, cap);
                    B.bin_cursor[q] = min(ex, cap);
                });
                if (tid == 0 && tot >= 0) B.bin_start[B.nbin] = min(tot, cap);
            }
            if (!(ok = barrier())) break;
            for (int r = tid; r < nrows; r += kSmallThreads) bins_particle(B, base + r, cur, n_bulk);
            if (!(ok = barrier())) break;
            for (int b0 = 4 * gw; b0 < B.nbin; b0 += 4 * warps)
                bucket_four<1>(B, b0, B.nbin, reinterpret_cast<unsigned long long *>(S.scratch + w * kSmallScratch));
            if (!(ok = barrier())) break;
            // items from a counter: bins of the shell have no rows and take no time, full ones ~15 us each
            for (;;) {
                int q = 0;
                if (lane == 0) q = atomicAdd(&A.bar->next, 1);
                q = __shfl_sync(0xffffffffu, q, 0);
                if (q >= B.nbin * A.parts) break;
                list_bin(B, q / A.parts, q % A.parts, A.parts, *reinterpret_cast<ListSmem *>(S.scratch + w * kSmallScratch));
                __syncwarp();
            }
            if (!(ok = barrier())) break;
        }
        if (STYLE == 0) {
            for (int r0 = w * R; r0 < nrows; r0 += kSmallWarps * R)
                density_rows_split<G, UNI, LPR, true>(B, base + r0, base + nrows, cur, n_bulk);
            __syncthreads();
            for (int r = tid; r < nrows; r += kSmallThreads) S.rho[r] = B.rho[base + r];
            if (!(ok = barrier())) break;
            small_force<EXACT, UNI>(B, S, base, nrows, rows_warp);
        } else {
            for (int r0 = w * R; r0 < nrows; r0 += kSmallWarps * R) {
                float f[3];
                full_rows<EXACT, UNI, LPR, true>(B, S.pos, S.vel, base, r0, nrows,
                                                 *reinterpret_cast<FullRowsSmem *>(S.scratch + w * kSmallScratch), f);
                const int r = r0 + lane;
                if (lane < R && r < nrows) {
                    if (!(isfinite(f[0]) && isfinite(f[1]) && isfinite(f[2]))) atomicOr(&B.st->status, kErrNonFinite);
                    for (int d = 0; d < 3; ++d) S.acc[d][r] = __float_as_uint(f[d]);
                }
            }
        }
        ok = barrier();
    }
    if (!ok) {
        if (tid == 0) atomicOr(&B.st->status, kErrTimeout);
        return;
    }
    // the last step's final half-kick
    for (int r = tid; r < nrows; r += kSmallThreads) {
        const int i = base + r, m = B.mask[cur][i], t = B.type[cur][i];
        double f[3];
        row_force<STYLE>(B, S, r, i, f);
        if (STYLE == 0)
            for (int d = 0; d < 3; ++d) B.facc[(size_t)d * n + i] = 0ull;
        B.f[i] = make_float4((float)f[0], (float)f[1], (float)f[2], 0.f);
        if (m & B.nve_bit) {
            const bool body = m & B.body_bit;
            for (int d = 0; d < 3; ++d)
                B.v[cur][d][i] = __fma_rn(B.dtfm[t - 1], f[d] + (body ? B.body[d] : 0.0), B.v[cur][d][i]);
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        BoxState &st = *B.st;
        st.step = S0.step + A.nsteps;
        st.ago = ago;
        st.moved = 0;
        st.rebuild = rb;
        st.n_bulk = n_bulk;
        st.cur = cur;
        st.nbuild = S0.nbuild + builds;
        st.pending = 0;
        st.sn_prev = s_seed[A.nsteps];
        st.sn = s_seed[A.nsteps + 1];
        st.sn_step = st.step + 1;
        st.sn_seed = B.seed;
        st.sn_ok = 1;
        A.done[3] += builds;  // steps that ran the rebuild
    }
}

template <int STYLE, bool EXACT, bool UNI>
static const void *small_kernel(int lpr)
{
    switch (lpr) {
    case 32: return (const void *)k_run_box<STYLE, EXACT, UNI, 32>;
    case 8: return (const void *)k_run_box<STYLE, EXACT, UNI, 8>;
    default: return (const void *)k_run_box<STYLE, EXACT, UNI, 2>;
    }
}

template <int STYLE> static const void *small_kernel(bool exact, bool uni, int lpr)
{
    if (exact) return uni ? small_kernel<STYLE, true, true>(lpr) : small_kernel<STYLE, true, false>(lpr);
    return uni ? small_kernel<STYLE, false, true>(lpr) : small_kernel<STYLE, false, false>(lpr);
}

// mDPD up to 768 rows per block (113,664 particles on 148 SMs; the force pass gives a warp at most 32
// rows), DPD up to 1,400 (what shared memory holds): there the whole run beats a launch per pass, us per
// step with / without:
//   mDPD  2,000  23 / 46     8,000  27 / 50    20,000  36 / 57    42,000  48 / 70   100,000  83 / 107
//   DPD   3,000  19 / 50    20,000  27 / 53    56,000  37 / 61   113,000  61 / 83   200,000 103 / 120
// Boxes with walls, and the threads-per-particle shapes of the full-list passes other than one, take
// the launches.  Mostly empty bins cost either way; up to a bin per particle the run is still ahead (slabs:
// 109,000 particles, 30,000 bins 107 / 132; 24,200 particles, 9,200 bins 53 / 82).
bool small_run_plan(const BoxDesc &B, const StepConfig &c, SmallPlan &p)
{
    if (c.full_chip || c.wall || c.wall_coupling || c.aboundary) return false;
    if (c.style == 0 ? !c.half : c.tpp_force != 1) return false;
    if (B.nbin > B.nlocal + 4096) return false;  // uniform fluids: a bin per 6 to 13 particles
    const int blocks = c.sms, warps = blocks * kSmallWarps;
    p.blocks = blocks;
    p.rows = (B.nlocal + blocks - 1) / blocks;
    p.lpr = p.rows <= kSmallWarps ? 32 : p.rows <= 4 * kSmallWarps ? 8 : 2;
    if (p.rows > (c.style == 0 ? 32 * kSmallWarps : 1400)) return false;
    const long long inner = (long long)(B.mbin[0] - 2) * (B.mbin[1] - 2) * (B.mbin[2] - 2);
    p.parts = 8;
    while (p.parts > 1 && inner * p.parts > warps) p.parts /= 2;
    p.smem = small_row_bytes(p.rows) + kSmallWarps * kSmallScratch;
    p.kernel = c.style == 0 ? small_kernel<0>(c.exact_rng, c.uniform_types, p.lpr)
                            : small_kernel<1>(c.exact_rng, c.uniform_types, p.lpr);
    // One block per SM has to be resident at once: the barriers count on it.  The kernel's limit of dynamic
    // shared memory belongs to the kernel, which boxes of other sizes share: it is set to what the device
    // offers, the same value for every box, so that no box's plan lowers another's.
    int per_sm = 0, dev = 0, coop = 0, optin = 0;
    cudaFuncAttributes fa;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, p.kernel) != cudaSuccess || p.smem > optin - (int)fa.sharedSizeBytes ||
        cudaFuncSetAttribute(p.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin - (int)fa.sharedSizeBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.kernel, kSmallThreads, p.smem) != cudaSuccess ||
        per_sm < 1) {
        (void)cudaGetLastError();
        return false;
    }
    return true;
}

size_t small_bar_bytes() { return sizeof(SmallBar); }

cudaError_t launch_small_run(cudaStream_t s, const BoxDesc &B, const SmallPlan &p, const SmallWait &w, void *bar,
                             int *done, int nsteps)
{
    SmallArgs a;
    a.B = B;
    a.nsteps = nsteps;
    a.bar = static_cast<SmallBar *>(bar);
    a.done = done;
    a.rows = p.rows;
    a.parts = p.parts;
    a.nblocks = p.blocks;
    a.polls = w.polls;
    a.withhold = w.barrier ? w.barrier * (unsigned)p.blocks : 0xffffffffu;
    const cudaError_t e = cudaMemsetAsync(bar, 0, sizeof(SmallBar), s);
    if (e != cudaSuccess) return e;
    void *args[] = {&a};
    return cudaLaunchCooperativeKernel(p.kernel, dim3(p.blocks), dim3(kSmallThreads), args, p.smem, s);
}

}  // namespace mdpd
