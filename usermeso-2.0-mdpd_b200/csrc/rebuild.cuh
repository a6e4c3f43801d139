// Device side of the neighbour rebuild (k_rebuild.cu lists its passes), shared by the rebuild kernels
// and the whole-run kernel of small boxes (k_small.cu).
#pragma once

#include "mdpd_dev.cuh"

namespace mdpd {

// counter[idx] += 1 for each calling lane, one atomic per distinct idx among the converged lanes
// (particles of one bin or class mostly sit next to each other, so a warp's lanes share few
// counters); returns what a per-lane atomicAdd would have returned, in lane order within each idx
__device__ __forceinline__ int warp_add1(int *counter, int idx)
{
    const unsigned active = __activemask();
    const unsigned peers = __match_any_sync(active, idx);
    const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter + idx, __popc(peers));
    base = __shfl_sync(peers, base, leader);
    return base + __popc(peers & ((1u << lane) - 1u));
}

// wraps particle i into the box (x of buffer c) and puts it into its reorder class
__device__ __forceinline__ void key_particle(const BoxDesc &B, int i, int c)
{
    uint32_t bid[3], sub[3];
    bool border = false;
    double xs[3];  // all three loads before the first store (no round trip per axis)
    for (int d = 0; d < 3; ++d) xs[d] = B.x[c][d][i];
    for (int d = 0; d < 3; ++d) {
        double x = xs[d];
        if (x < B.lo[d]) x += B.prd[d];
        if (x >= B.hi[d]) {
            x -= B.prd[d];
            x = fmax(x, B.lo[d]);
        }
        if (!(x >= B.lo[d] && x < B.hi[d])) atomicOr(&B.st->status, kErrLost);
        B.x[c][d][i] = x;
        bid[d] = (uint32_t)clamp_bin(bin_coord(x, B.lo[d], B.bininv[d]), B.mbin[d]);
        const double off = __fma_rn(-(double)(uint32_t)(bid[d] - 1u), B.binsize[d], x);
        sub[d] = (uint32_t)clamp_bin((int)__dmul_rn(off, B.coord_inv[d]), 16);
        border |= (x <= B.lo[d] + B.cutghost) || (x >= B.hi[d] - B.cutghost);
    }
    const int bin = (int)(bid[0] + B.mbin[0] * (bid[1] + bid[2] * B.mbin[1]));
    const int cls = MDPD_IDX((border ? B.nbin : 0) + B.bin_rank[MDPD_IDX(bin, B.nbin)], 2 * B.nbin);
    B.cls_of[i] = cls;
    B.sub_of[i] = (int)morton3(sub[0], sub[1], sub[2]);
    warp_add1(B.cls_count, cls);
}

// Position of particle i as the list build reads it from bpos: x, y, z and, in .w, its list word:
// i for a local or an upper ghost image, ~i for a lower ghost image.  As a signed integer the word
// orders a candidate against a centre (a local) as pair-once ownership does: a candidate whose
// word is above the centre's index is owned by the centre (a local above it, or an upper image;
// a lower image is negative, below every centre), and only the centre itself has an equal word.
__device__ __forceinline__ float4 list_pos(const float4 &p, int i, int nlocal)
{
    const int wd = i < nlocal || (pflags(p) & kUpperImage) ? i : ~i;
    return make_float4(p.x, p.y, p.z, __int_as_float(wd));
}

// One bucket's members in (key, index) order by the whole warp: the ranks from a shared-memory
// copy of the keys (buckets of up to kClassMax members).
template <int MODE>
__device__ __forceinline__ void bucket_warp(const BoxDesc &B, int *arr, int s, int n, int lane,
                                            unsigned long long *key)
{
    const int lim = MODE == 0 ? B.nlocal : n_all(B);
    for (int e = lane; e < n; e += 32) {
        const int idx = MDPD_IDX(arr[s + e], lim);
        key[e] = MODE == 0 ? (((unsigned long long)(uint32_t)B.sub_of[idx] << 32) | (uint32_t)idx)
                           : (unsigned long long)(uint32_t)idx;
    }
    __syncwarp();
    for (int e = lane; e < n; e += 32) {
        const unsigned long long k = key[e];
        int rank = 0;
        for (int q = 0; q < n; ++q) rank += key[q] < k;
        const int idx = (int)(uint32_t)k;
        arr[s + rank] = idx;
        if (MODE == 1) B.bpos[s + rank] = list_pos(B.pos[idx], idx, B.nlocal);
    }
    __syncwarp();
}

// Buckets are taken four at a time per warp, one per group of 8 lanes holding up to 4 members
// each: a bucket of up to 32 members (the usual case: a reorder class is one bin's interior or
// border locals, ~14 at rho 6.05) is ordered with shuffles inside its group, so the warp waits
// once for the loads of four buckets; a larger one is ordered by the whole warp afterwards.
// Work items are 32 buckets (one group of four per warp), so that a small box's few units of 256
// spread over the chip: with a unit per block each warp took eight groups one after another (the
// bin pass of a 2,000-particle box: 17.8 us).
constexpr int kGroupSlots = 4;  // members per lane of an 8-lane group
// buckets b0 .. b0 + 3 (below end) by one warp; `key`: kClassMax words of the warp's own
template <int MODE>  // 0: reorder classes -> perm, 1: bins -> bin_order + bpos
__device__ __forceinline__ void bucket_four(const BoxDesc &B, int b0, int end, unsigned long long *key)
{
    const int lane = threadIdx.x & 31, grp = lane >> 3, l8 = lane & 7;
    int *cnt = MODE == 0 ? B.cls_count : B.bin_count;
    const int *start = MODE == 0 ? B.cls_start : B.bin_start;
    int *arr = MODE == 0 ? B.perm : B.bin_order;
    const int lim = MODE == 0 ? B.nlocal : n_all(B);
    const int b = b0 + grp;
    int n = 0, s = 0, counted = 0;
    if (b < end) {
        n = cnt[b];
        s = start[b];
        // a ghost overflow: the bins' members end with the arrays
        if (MODE == 1) n = min(n, B.nlocal + B.ghost_cap - s);
        counted = cnt[b];
    }
    if (n != 0 && !(MDPD_IN(s, s + n) && MDPD_IN(s + n - 1, lim))) {
        if (l8 == 0) cnt[b] = 0;  // check build: a bucket outside its array
        n = 0;
    }
    if (MODE == 1) {
        // a bin whose last member is a local holds no ghost image (locals come first): it
        // is already in index order, its bpos written by the scatter
        int last = 0;
        if (n > 0 && l8 == 0) last = arr[s + n - 1];
        last = __shfl_sync(0xffffffffu, last, grp << 3);
        if (n == 0 && counted != 0 && l8 == 0) cnt[b] = 0;
        if (n > 0 && last < B.nlocal) {
            if (l8 == 0) cnt[b] = 0;
            n = 0;
        }
    }
    const bool group = n > 0 && n <= 8 * kGroupSlots;
    const int slots = __reduce_max_sync(0xffffffffu, group ? (n + 7) >> 3 : 0);  // warp-uniform
    int idx[kGroupSlots];
    unsigned long long k[kGroupSlots];
#pragma unroll
    for (int m = 0; m < kGroupSlots; ++m) {
        idx[m] = 0;
        if (group && l8 + 8 * m < n) idx[m] = MDPD_IDX(arr[s + l8 + 8 * m], lim);
    }
#pragma unroll
    for (int m = 0; m < kGroupSlots; ++m) {
        k[m] = ~0ull;  // no member: above every key, counted by no rank
        if (group && l8 + 8 * m < n)
            k[m] = MODE == 0 ? (((unsigned long long)(uint32_t)B.sub_of[idx[m]] << 32) | (uint32_t)idx[m])
                             : (unsigned long long)(uint32_t)idx[m];
    }
    // rank of each member: the group's keys below it (every member's key is loaded before
    // any lane gets past these shuffles, so the stores below cannot overwrite an unread one)
    int rank[kGroupSlots] = {};
#pragma unroll
    for (int mm = 0; mm < kGroupSlots; ++mm) {
        if (mm >= slots) break;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const unsigned long long kq = __shfl_sync(0xffffffffu, k[mm], (grp << 3) | q);
#pragma unroll
            for (int m = 0; m < kGroupSlots; ++m) rank[m] += kq < k[m] ? 1 : 0;
        }
    }
#pragma unroll
    for (int m = 0; m < kGroupSlots; ++m) {
        if (group && l8 + 8 * m < n) {
            arr[s + rank[m]] = idx[m];
            if (MODE == 1) B.bpos[s + rank[m]] = list_pos(B.pos[idx[m]], idx[m], B.nlocal);
        }
    }
    if (group && l8 == 0) cnt[b] = 0;
    // buckets of more than 32 members: the whole warp, one after another
    unsigned big = __ballot_sync(0xffffffffu, l8 == 0 && n > 8 * kGroupSlots);
    while (big) {
        const int leader = __ffs(big) - 1;
        big &= big - 1;
        const int bb = b0 + (leader >> 3);
        const int nb = __shfl_sync(0xffffffffu, n, leader), sb = __shfl_sync(0xffffffffu, s, leader);
        __syncwarp();
        if (nb > kClassMax) {
            if (lane == 0) atomicOr(&B.st->status, kErrBucketOverflow);
        } else
            bucket_warp<MODE>(B, arr, sb, nb, lane, key);
        if (lane == 0) cnt[bb] = 0;
    }
}

__device__ __forceinline__ int image_mask(const BoxDesc &B, double x, int d)
{
    // bit 0: image at +prd (x within cutghost of lo), bit 1: image at -prd
    int m = 0;
    if (x <= B.lo[d] + B.cutghost) m |= 1;
    if (x >= B.hi[d] - B.cutghost) m |= 2;
    return m;
}

__device__ __forceinline__ int bits_count(int m) { return 1 + (m & 1) + ((m >> 1) & 1); }

// f(q, sx, sy, sz) for the periodic images of a particle with image masks m, in the order of the ghost
// indices (z slowest), q counting them.  A box side is at least three cutoffs, so a coordinate has
// one image at most and a particle seven; the eight combinations are unrolled, so that f's loads for
// all images can be in flight together.
template <class F> __device__ __forceinline__ void for_images(const int m[3], F &&f)
{
    int q = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        // along each axis the unshifted place comes after a shift by -1 and before one by +1
        int sh[3];
        bool ok = true, any = false;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int up = (c >> d) & 1;
            const int s = (m[d] & 2) ? (up ? 0 : -1) : up;
            ok &= m[d] != 0 || !up;
            any |= s != 0;
            sh[d] = s;
        }
        if (ok && any) f(q++, sh[0], sh[1], sh[2]);
    }
}

// bin of the image of x shifted by (sx, sy, sz) periods (gpu_assign_bin_id's rule)
__device__ __forceinline__ int image_bin(const BoxDesc &B, const double x[3], int sx, int sy, int sz)
{
    const double gc[3] = {x[0] + sx * B.prd[0], x[1] + sy * B.prd[1], x[2] + sz * B.prd[2]};
    int bid[3];
    for (int d = 0; d < 3; ++d) {
        const double v = gc[d];
        const int b = clamp_bin(bin_coord(v, B.lo[d], B.bininv[d]), B.mbin[d]);
        bid[d] = v >= B.lo[d] ? (v <= B.hi[d] ? b : B.mbin[d] - 1) : 0;
    }
    return bid[0] + B.mbin[0] * (bid[1] + bid[2] * B.mbin[1]);
}

// particle k of the new order: every array from buffer c to the other, packed with the step's seed
// sn, its images counted, its bin and its images' bins
template <int STYLE>
__device__ __forceinline__ void permute_particle(const BoxDesc &B, int k, int c, uint32_t sn)
{
    const int o = 1 - c;
    const int old = MDPD_IDX(B.perm[k], B.nlocal);
    // every load of the particle is issued before the first store (the compiler may not move
    // a load above a store to a possibly aliased array): one memory round trip
    double x[3], v[3];
    for (int d = 0; d < 3; ++d) {
        x[d] = B.x[c][d][old];
        v[d] = B.v[c][d][old];
    }
    const int tag = B.tag[c][old], type = B.type[c][old], mask = B.mask[c][old];
    const float phi = B.wall_fix ? B.phi[c][old] : 0.f;
    for (int d = 0; d < 3; ++d) {
        B.x[o][d][k] = x[d];
        B.v[o][d][k] = v[d];
        B.xh[d][k] = x[d];
    }
    B.tag[o][k] = tag;
    B.type[o][k] = type;
    B.mask[o][k] = mask;
    if (B.wall_fix) {
        B.phi[o][k] = phi;              // zero in both buffers otherwise
        if (B.arb_bc) B.count2[k] = -1;  // until the density pass has listed the row's wall particles
    }
    const float fvx = (float)v[0], fvy = (float)v[1], fvz = (float)v[2];
    B.pos[k] = make_float4((float)(x[0] - B.cen[0]), (float)(x[1] - B.cen[1]),
                           (float)(x[2] - B.cen[2]), pack_w(B, type, mask));
    const uint32_t sg = STYLE == 0 ? sig_mdpd(tag, sn) : sig_dpd(tag, fvx, fvy, fvz, sn);
    B.vel[k] = make_float4(fvx, fvy, fvz, __uint_as_float(sg));
    // ghost images of this particle: their number (for the scan) and their bins' counts
    int m[3], nimg = 1;
    for (int d = 0; d < 3; ++d) {
        m[d] = image_mask(B, x[d], d);
        nimg *= bits_count(m[d]);
    }
    B.cls_of[k] = nimg - 1;
    // bin of the local
    int bid[3];
    for (int d = 0; d < 3; ++d) bid[d] = clamp_bin(bin_coord(x[d], B.lo[d], B.bininv[d]), B.mbin[d]);
    const int bin = bid[0] + B.mbin[0] * (bid[1] + bid[2] * B.mbin[1]);
    B.bin_of[k] = bin;
    warp_add1(B.bin_count, MDPD_IDX(bin, B.nbin));
    if (nimg > 1)
        for_images(m, [&](int, int sx, int sy, int sz) {
            atomicAdd(&B.bin_count[MDPD_IDX(image_bin(B, x, sx, sy, sz), B.nbin)], 1);
        });
}

// the locals of a bin: its bulk run and its border run
__device__ __forceinline__ int bin_locals(const BoxDesc &B, int bin)
{
    const int rk = B.bin_rank[bin];
    return B.cls_start[rk + 1] - B.cls_start[rk] + B.cls_start[B.nbin + rk + 1] - B.cls_start[B.nbin + rk];
}

// local k and its images into their bins
__device__ __forceinline__ void bins_particle(const BoxDesc &B, int k, int c, int n_bulk)
{
    const int nl = B.nlocal, na = nl + B.ghost_cap;  // na: places in the bin-ordered arrays
    const int bin = MDPD_IDX(B.bin_of[k], B.nbin);
    const float4 pk = B.pos[k];
    const bool edge = k >= n_bulk;
    const int g0 = edge ? B.gfirst[k] : 0, g1 = edge ? B.gfirst[k + 1] : 0;
    const int rk = B.bin_rank[bin];
    const int b0 = B.cls_start[rk], b1 = B.cls_start[rk + 1];  // the bin's bulk run
    const int e0 = B.cls_start[B.nbin + rk];                     // its border run
    const int p = MDPD_IDX(B.bin_start[bin] + (edge ? (b1 - b0) + (k - e0) : k - b0), na);
    if (p < na) {
        B.bpos[p] = list_pos(pk, k, nl);
        B.bin_order[p] = k;
    }
    if (g1 == g0) return;
    double x[3];
    int m[3];
    for (int d = 0; d < 3; ++d) {
        x[d] = B.x[c][d][k];
        m[d] = image_mask(B, x[d], d);
    }
    const float4 vk = B.vel[k];
    // the images' bins and the number of locals in them first: their loads are in flight together
    int gb[7], nloc[7];
#pragma unroll
    for (int q = 0; q < 7; ++q) gb[q] = -1, nloc[q] = 0;
    for_images(m, [&](int q, int sx, int sy, int sz) {
        const int bn = MDPD_IDX(image_bin(B, x, sx, sy, sz), B.nbin);
#pragma unroll
        for (int e = 0; e < 7; ++e)
            if (e == q) gb[e] = bn;
    });
#pragma unroll
    for (int q = 0; q < 7; ++q)
        if (gb[q] >= 0) nloc[q] = bin_locals(B, gb[q]);
#pragma unroll
    for (int q = 0; q < 7; ++q)
        if (gb[q] >= 0 && g0 + q < B.ghost_cap) nloc[q] += atomicAdd(&B.bin_cursor[gb[q]], 1);
    for_images(m, [&](int q, int sx, int sy, int sz) {
        const int g = g0 + q;
        if (g >= B.ghost_cap) {
            atomicOr(&B.st->status, kErrGhostOverflow);
            return;
        }
        const int gi = nl + g;
        B.gsrc[g] = k;
        const int code = (sx + 1) + 3 * (sy + 1) + 9 * (sz + 1);
        B.gimg[g] = code;
        B.pos[gi] = make_float4((float)(x[0] + sx * B.prd[0] - B.cen[0]), (float)(x[1] + sy * B.prd[1] - B.cen[1]),
                                (float)(x[2] + sz * B.prd[2] - B.cen[2]), ghost_w(pk.w, code));
        B.vel[gi] = vk;
#pragma unroll
        for (int e = 0; e < 7; ++e)
            if (e == q) {
                const int at = MDPD_IDX(nloc[e], na);
                if (at < na) B.bin_order[at] = gi;
            }
    });
}

constexpr int kListChunk = 224;                 // kept candidates per chunk (3.5 rounds)

__device__ __forceinline__ float warp_min(float v)
{
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ float warp_max(float v)
{
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// one warp's shared memory of the list build
struct ListSmem {
    float4 ca[32], cb[32];      // centres: x, x, y, y | z, z, index, row offset
    int n[32];                  // entries of each centre so far
    float4 q[kListChunk];       // kept candidates: x, y, z, list word
    int j[kListChunk];          // their particle indices
    float4 lo, hi;              // the centres' bounding box; cmin
    int d[32], ex[32];          // non-empty stencil bins: start - stream offset; offset
};

// rows of bin b by one warp; with parts > 1 the bin's members are shared out to `parts` warps
__device__ __forceinline__ void list_bin(const BoxDesc &B, int b, int part, int parts, ListSmem &L)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int s = B.bin_start[b], e = B.bin_start[b + 1];
    if (e == s) return;
    if (!(MDPD_IN(s, e) && MDPD_IN(e - 1, n_all(B)))) return;  // check build: a bin outside the arrays
    const int per = parts == 1 ? 32 : min(32, (e - s + parts - 1) / parts);  // centres at a time
    if (B.bin_order[s] >= B.nlocal) return;  // no locals in this bin
    const float rc2 = B.rc2_tail;
    const float rn2 = B.list_reduce ? B.rn2_list : rc2;  // with rc2: every pair (full list)
    // a row marks the entries its centre owns with bit 31 (kOwnedEntry), which the pair-once
    // density pass reads instead of re-deriving ownership per step; other readers mask it off
    const int own = (int)kOwnedEntry;
    const int ncol = B.n_col, nlocal = B.nlocal;
    int *const table = B.table;
    const int bx = b % B.mbin[0], by = (b / B.mbin[0]) % B.mbin[1], bz = b / (B.mbin[0] * B.mbin[1]);
    // stencil bins: lane l < 27 takes offset (l%3-1, l/3%3-1, l/9-1)
    int st = 0, sz = 0;
    if (lane < 27) {
        const int x = bx + lane % 3 - 1, y = by + (lane / 3) % 3 - 1, z = bz + lane / 9 - 1;
        if (x >= 0 && x < B.mbin[0] && y >= 0 && y < B.mbin[1] && z >= 0 && z < B.mbin[2]) {
            const int nb = x + B.mbin[0] * (y + z * B.mbin[1]);
            st = B.bin_start[nb];
            sz = B.bin_start[nb + 1] - st;
            if (sz != 0 && !(MDPD_IN(st, st + sz) && MDPD_IN(st + sz - 1, n_all(B)))) sz = 0;
        }
    }
    int cum = sz;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, cum, o);
        if (lane >= o) cum += v;
    }
    const int total = __shfl_sync(0xffffffffu, cum, 31);
    // the candidate stream is the non-empty stencil bins in slot order; bin k of them starts
    // at stream offset ex_k, so stream position q is particle d_k + q of the bin order with
    // d_k = start_k - ex_k, k the last non-empty bin with ex_k <= q
    const unsigned ne = __ballot_sync(0xffffffffu, sz != 0);
    if (sz != 0) {
        const int k = __popc(ne & lt);
        L.d[k] = st - (cum - sz);
        L.ex[k] = cum - sz;
    }
    __syncwarp();
    // lane k holds ex_k of non-empty bin k (no bin: past every position)
    const int exk = lane < __popc(ne) ? L.ex[lane] : 0x7fffffff;
    const unsigned le = lt | (1u << lane);
    int local_max = 0;
    for (int cb = s + part * per; cb < e; cb += parts * per) {
        // centre batch: members with index < nlocal (they come first in a bin)
        const int pc = cb + lane;
        const int ci = pc < e && lane < per ? MDPD_IDX(B.bin_order[pc], n_all(B)) : nlocal;
        const bool is_c = ci < nlocal;
        const unsigned cm = __ballot_sync(0xffffffffu, is_c);
        if (cm == 0) break;
        const int nc = __popc(cm);
        const float4 pc4 = is_c ? B.bpos[pc] : make_float4(0.f, 0.f, 0.f, 0.f);
        L.ca[lane] = make_float4(pc4.x, pc4.x, pc4.y, pc4.y);
        // entry p of centre i at (i & ~31) * ncol + 32 p + (i & 31): entries p of 32
        // consecutive centres are contiguous
        L.cb[lane] = make_float4(pc4.z, pc4.z, __int_as_float(ci),
                                    __uint_as_float((unsigned)(ci & ~31) * (unsigned)ncol + (unsigned)(ci & 31)));
        L.n[lane] = 0;
        {
            const float inf = __int_as_float(0x7f800000);
            const float lox = warp_min(is_c ? pc4.x : inf), hix = warp_max(is_c ? pc4.x : -inf);
            const float loy = warp_min(is_c ? pc4.y : inf), hiy = warp_max(is_c ? pc4.y : -inf);
            const float loz = warp_min(is_c ? pc4.z : inf), hiz = warp_max(is_c ? pc4.z : -inf);
            // smallest centre index of the batch: a candidate below it (a local with a smaller
            // index, or a lower ghost image) is owned by none of the centres, so on a reduced
            // list it is a hit only within rn2, and the filter keeps it only within rn2 of the box
            int cmin = is_c ? ci : 0x7fffffff;
            for (int o = 16; o > 0; o >>= 1) cmin = min(cmin, __shfl_xor_sync(0xffffffffu, cmin, o));
            if (lane == 0) {
                L.lo = make_float4(lox, loy, loz, __int_as_float(cmin));
                L.hi = make_float4(hix, hiy, hiz, 0.f);
            }
        }
        __syncwarp();
        for (int qs = 0; qs < total;) {
            // filter: fill up to kListChunk kept candidates
            int nk = 0;
            const float4 lo = L.lo, hi = L.hi;
            for (; qs < total && nk <= kListChunk - 32; qs += 32) {
                const int q = qs + lane;
                // bin of position q: the bins that start before qs, plus those that start
                // in [qs, q] (bit ex_k - qs of the round's start mask)
                const unsigned starts = __reduce_or_sync(
                    0xffffffffu, exk >= qs && exk - qs < 32 ? 1u << (exk - qs) : 0u);
                const int kq = __popc(__ballot_sync(0xffffffffu, exk < qs)) + __popc(starts & le) - 1;
                bool keep = false;
                float4 pj = make_float4(0.f, 0.f, 0.f, 0.f);
                if (q < total) {
                    pj = B.bpos[L.d[kq] + q];
                    const float gx = fmaxf(fmaxf(lo.x - pj.x, pj.x - hi.x), 0.f);
                    const float gy = fmaxf(fmaxf(lo.y - pj.y, pj.y - hi.y), 0.f);
                    const float gz = fmaxf(fmaxf(lo.z - pj.z, pj.z - hi.z), 0.f);
                    keep = dist2(gx, gy, gz) <= (__float_as_int(pj.w) < __float_as_int(lo.w) ? rn2 : rc2);
                }
                const unsigned kb = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const int k = nk + __popc(kb & lt);
                    const int wd = __float_as_int(pj.w);
                    L.q[k] = pj;
                    L.j[k] = MDPD_IDX(wd ^ (wd >> 31), n_all(B));
                }
                nk += __popc(kb);
            }
            __syncwarp();
            for (int r0 = 0; r0 < nk; r0 += 64) {
                const int ka = r0 + lane, kb2 = ka + 32;
                const float4 pa = ka < nk ? L.q[ka] : make_float4(1e30f, 1e30f, 1e30f, 0.f);
                const float4 pb = kb2 < nk ? L.q[kb2] : make_float4(1e30f, 1e30f, 1e30f, 0.f);
                const int ja = ka < nk ? L.j[ka] : 0, jb = kb2 < nk ? L.j[kb2] : 0;
                const int wa = __float_as_int(pa.w), wb = __float_as_int(pb.w);
                const unsigned long long px = pk2(pa.x, pb.x), py = pk2(pa.y, pb.y), pz = pk2(pa.z, pb.z);
#pragma unroll 1
                for (int c = 0; c < nc; ++c) {
                    const float4 A = L.ca[c], C = L.cb[c];
                    const int cic = __float_as_int(C.z);
                    float r2a, r2b;
                    upk2(dist2x2(sub2(pk2(A.x, A.y), px), sub2(pk2(A.z, A.w), py), sub2(pk2(C.x, C.y), pz)),
                         r2a, r2b);
                    // owned candidates are hits within rc2, the others within rn2 (<= rc2)
                    const bool oa = wa > cic, ob = wb > cic;
                    const bool ha = r2a <= (oa ? rc2 : rn2) && wa != cic;
                    const bool hb = r2b <= (ob ? rc2 : rn2) && wb != cic;
                    const unsigned bala = __ballot_sync(0xffffffffu, ha);
                    const unsigned balb = __ballot_sync(0xffffffffu, hb);
                    const int n0 = L.n[c];
                    const int na = n0 + __popc(bala);
                    // a row that would overflow keeps writing its last entry (the count
                    // reports the overflow); the table holds ncol entries per row
                    const unsigned row = __float_as_uint(C.w);
                    if (ha)
                        table[row + 32u * (unsigned)min(n0 + __popc(bala & lt), ncol - 1)] = ja | (oa ? own : 0);
                    if (hb)
                        table[row + 32u * (unsigned)min(na + __popc(balb & lt), ncol - 1)] = jb | (ob ? own : 0);
                    L.n[c] = na + __popc(balb);  // every lane stores the same count
                }
            }
            __syncwarp();
        }
        if (is_c) {
            const int my_n = L.n[lane];
            B.count[ci] = my_n < ncol ? my_n : ncol;
            if (my_n > ncol) atomicOr(&B.st->status, kErrListOverflow);
            local_max = max(local_max, my_n);
        }
        __syncwarp();
    }
    for (int o = 16; o > 0; o >>= 1) local_max = max(local_max, __shfl_xor_sync(0xffffffffu, local_max, o));
    if (lane == 0 && local_max > 0) atomicMax(&B.st->max_count, local_max);
}

}  // namespace mdpd
