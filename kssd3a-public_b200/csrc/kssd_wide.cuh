// Wide context groups (contexts that many genomes of an index hold, one object per
// genome) joined on the tensor cores.  Included by kssdgpu.cu inside its namespace.
//
// Every pair of genomes (q, r) of a group adds to its cell num_ctx 1, diff_obj d >= 1,
// num_mut2_ctx d >= 2 and diff_obj_section d, d = min(dna_popcount(o_q ^ o_r),
// NUM_CODENS + 1) (src/command_ani.h:694-716).  Take the group's most frequent object M
// and let e = min(dna_popcount(o ^ M), NUM_CODENS + 1) be a genome's distance to it: most
// genomes have e = 0.  When one of the pair is at M, d is the other's e; when neither is
// and their differences from M lie at different bases, d = e_q + e_r >= 2.  These values
// are sums of products of per-genome terms, so over all groups they are Gram matrices:
//     P = present, Z = (e == 0), L = (e <= 1), U = (e == 1), S = e + present, E = e
//     num_ctx          = P'P
//     diff_obj         = P'P - Z'Z
//     num_mut2_ctx     = P'P - L'L + U'U
//     diff_obj_section = S'S - E'E - P'P
// six symmetric int8 products of depth = groups, whatever the number of alleles.  The
// pairs that this misjudges -- both away from M, with a base in common among their
// differences, or past the cap -- are corrected one by one (wide_correction).
//
// Why: the same counters by one operand row per allele need 4 n^2 per allele, and in a
// species of 1,024 genomes a context has some 40 alleles, nearly all of one or two genomes
// (643,817 rows against 17,000 groups of six).  Which is cheaper depends on the data: where
// minor alleles are common their pairs to correct are many and the alleles few, and the
// join with a row per allele takes over (dense_chosen compares the two).
//
// Measured (B200, whole calls): the self join of 1,024 genomes of one species 1,748 (rows
// per allele) -> 175 us, of 3,000 genomes of ten species 16.4 -> 2.9 ms; a block of 200
// queries against 1,024 genomes of their species 6.82 ms (postings walked per query, 1.9 G
// atomics) -> 0.24 ms, of one query 2.23 -> 0.17 ms, of 30 read sets against 500 genomes
// 975 -> 277 us.
#pragma once

// Groups of at least this many postings are wide.  A group costs six rows of the products
// (12 n^2 operations, about n^2 / 170 ps, and 6 n bytes written), its k (k - 1) / 2 pairs
// by atomics 7.4 ps each: equal near k = n / 24.
inline uint32_t wide_min_postings(int nref)
{
    return (uint32_t)std::min(128, std::max(2, nref / 24));
}

// Contexts per pass: bounds the operand rows, and with at most 2 * (NUM_CODENS + 1) per
// pair and context a pass's corrections fit the fields of one 64-bit word.
constexpr uint64_t kWidePass = 131072;
constexpr int kWideRows = 6;
constexpr uint32_t kWideMaxRefs = 4096;               // a warp's map and list stay in shared memory
constexpr uint64_t kWideBlockBytes = 8ull << 30;      // scratch of a block join, at most
constexpr uint32_t kWideLoads = 4;  // postings of a lane in flight
constexpr uint32_t kWidePairs = 4;  // genomes compared with a lane's at a time
constexpr size_t kWideSmem = 220 * 1024;  // dynamic shared memory of a CTA, at most
// correction word: num_mut2_ctx in bits 0-20, diff_obj in 21-41, diff_obj_section in 42-63
static_assert(kWidePass < (1ull << 21) && kWidePass * 2 * kMinInit < (1ull << 22), "correction fields");

__device__ __forceinline__ uint32_t wide_e(uint32_t o, uint32_t major)
{
    return (uint32_t)min(kMinInit, dna_pop(o ^ major));
}

// the bases at which an object xor the major one differs, as bits 0, 2, 4, ...
__device__ __forceinline__ uint32_t wide_bases(uint32_t x) { return (x | (x >> 1)) & 0x55555555u; }

// What the products overcount on a pair of genomes with objects a and b, both different
// from major: their sum of distances for the difference, and one of each threshold.
__device__ __forceinline__ unsigned long long wide_correction(uint32_t a, uint32_t b, uint32_t ea, uint32_t eb)
{
    const uint32_t d = (uint32_t)min(kMinInit, dna_pop(a ^ b)), est = ea + eb;
    if (d == est)
        return 0;  // then d >= 2
    return (unsigned long long)(d < 2) | ((unsigned long long)(d == 0) << 21) |
           ((unsigned long long)(est - d) << 42);
}
__device__ __forceinline__ unsigned long long wide_correction(uint32_t a, uint32_t b, uint32_t major)
{
    return wide_correction(a, b, wide_e(a, major), wide_e(b, major));
}

// The most frequent object among 32 postings spread over group [b, b + k) (all of them
// when k <= 32); o receives this lane's (lanes at or past k: 0).  Any object would do:
// the choice only decides how many pairs need a correction.
__device__ __forceinline__ uint32_t wide_major(const uint64_t *__restrict__ post, uint32_t b, uint32_t k,
                                               uint32_t lane, uint32_t &o)
{
    const uint32_t at = k > 32 ? (uint32_t)(((uint64_t)lane * k) >> 5) : lane;
    const bool in = at < k;
    o = in ? (uint32_t)__ldg(post + b + at) : 0u;
    const unsigned act = __ballot_sync(0xffffffffu, in);
    uint32_t votes = 0;
    if (in)
        votes = ((uint32_t)__popc(__match_any_sync(act, o)) << 5) | (31u - lane);
    const uint32_t best = __reduce_max_sync(0xffffffffu, votes);
    return __shfl_sync(0xffffffffu, o, (int)(31u - (best & 31u)));
}

// The six operand bytes of four genomes from their distances (0xFF: absent).
struct WideWords {
    uint32_t w[kWideRows];  // P, Z, L, U, S, E
};
__device__ __forceinline__ WideWords wide_words(uint32_t e)
{
    WideWords x;
    const uint32_t present = __vcmpne4(e, 0xFFFFFFFFu);
    x.w[0] = present & 0x01010101u;
    x.w[1] = __vcmpeq4(e, 0u) & 0x01010101u;
    x.w[3] = __vcmpeq4(e, 0x01010101u) & 0x01010101u;
    x.w[2] = x.w[1] | x.w[3];
    x.w[5] = e & present;
    x.w[4] = x.w[5] + x.w[0];
    return x;
}

// Shared memory of one warp of k_wide_rows: the genomes' distances (later the list of those
// that differ at a base), then the genomes away from the major object as (gid | e << 20) <<
// 32 | object ^ major.
__host__ __device__ __forceinline__ size_t wide_warp_smem(uint32_t npad, uint32_t nref)
{
    return (size_t)npad + ((size_t)nref * 8 + 15) / 16 * 16;
}

// Operand rows of the groups 0 .. n_list of list (row c of matrix m at X + m * xs + c *
// npad), and the corrections of their pairs into corr[cell of (q, r)].  A warp takes a
// group: one pass over its postings fills a byte map of the genomes' distances in shared
// memory, from which the rows are written in 16-byte pieces, and lists the genomes away
// from the major object (a tenth of them at 1 % divergence); their pairs are compared
// with kWidePairs of them broadcast and lanes on consecutive others.  Bound by issue (the
// pairs) and the corrections' atomics (L2); the rows are 6 n bytes.
//
// BLOCK: the pairs are those of a query with the group's genomes instead.  qobj[c * nqpad
// + q] is the object of query q at group c (kWideNone: it does not hold it; kWideRun: it
// holds several, from that entry on), written by the counting kernel; the queries' operand
// rows go to Y, the corrections to corr[q * nref + r].  A query of several objects takes the
// place of the one nearest to the major object: its difference to a genome there is that
// one's, and to every other genome the least over the run, so all of them are compared.
struct WideBlock {
    const uint32_t *qobj;
    uint32_t nq, nqpad;
    int8_t *Y;
    size_t ys;
    const uint64_t *qkeys, *qoffs;
    int obj_bits;
};

template <bool BLOCK>
__global__ void __launch_bounds__(256) k_wide_rows(const SharedGroup *__restrict__ list,
                                                   const unsigned long long *__restrict__ items, uint32_t n_list,
                                                   const uint64_t *__restrict__ post, uint32_t nref, uint32_t npad,
                                                   int8_t *__restrict__ X, size_t xs,
                                                   unsigned long long *__restrict__ corr, int bases_only,
                                                   const WideBlock Q)
{
    extern __shared__ __align__(16) unsigned char wsm[];
    const uint32_t lane = threadIdx.x & 31u, warps = blockDim.x >> 5;
    unsigned char *emap = wsm + (threadIdx.x >> 5) * wide_warp_smem(npad, nref);
    unsigned long long *minor = reinterpret_cast<unsigned long long *>(emap + npad);
    const uint4 absent = make_uint4(~0u, ~0u, ~0u, ~0u);
    for (uint32_t s = blockIdx.x * warps + (threadIdx.x >> 5); s < n_list; s += gridDim.x * warps) {
        // a group of the index's list, or (BLOCK) a numbered (begin | k << 32)
        const unsigned long long item = BLOCK ? items[s] : *reinterpret_cast<const unsigned long long *>(list + s);
        const uint32_t b = (uint32_t)item, k = (uint32_t)(item >> 32);
        for (uint32_t i = lane; i < npad / 16; i += 32)
            reinterpret_cast<uint4 *>(emap)[i] = absent;
        uint32_t o;
        const uint32_t major = wide_major(post, b, k, lane, o);
        __syncwarp();
        uint32_t nm = 0;
        for (uint32_t j0 = 0; j0 < k; j0 += 32 * kWideLoads) {
            uint64_t p[kWideLoads];  // in flight together: a group's postings come from HBM
#pragma unroll
            for (uint32_t x = 0; x < kWideLoads; ++x) {
                const uint32_t j = j0 + 32 * x + lane;
                p[x] = j < k ? __ldg(post + b + j) : 0;
            }
#pragma unroll
            for (uint32_t x = 0; x < kWideLoads; ++x) {
                const bool in = j0 + 32 * x + lane < k;
                const uint32_t gid = (uint32_t)(p[x] >> 32), e = in ? wide_e((uint32_t)p[x], major) : 0u;
                if (in)
                    emap[gid] = (unsigned char)e;
                const unsigned away = __ballot_sync(0xffffffffu, e != 0);
                if (e)
                    minor[nm + __popc(away & ((1u << lane) - 1u))] =
                        ((unsigned long long)(gid | (e << kGidBits)) << 32) | ((uint32_t)p[x] ^ major);
                nm += __popc(away);
            }
        }
        __syncwarp();
        for (uint32_t i = lane; i < npad / 16; i += 32) {
            const uint4 e = reinterpret_cast<const uint4 *>(emap)[i];
            const WideWords a = wide_words(e.x), c = wide_words(e.y), d = wide_words(e.z), f = wide_words(e.w);
#pragma unroll
            for (int m = 0; m < kWideRows; ++m)
                reinterpret_cast<uint4 *>(X + m * xs + (size_t)s * npad)[i] = make_uint4(a.w[m], c.w[m], d.w[m], f.w[m]);
        }
        if (BLOCK) {
            for (uint32_t q0 = 0; q0 < Q.nqpad; q0 += 128) {
                const uint32_t q = q0 + 4 * lane;
                uint4 oq = make_uint4(kWideNone, kWideNone, kWideNone, kWideNone);
                if (q < Q.nqpad)
                    oq = __ldcs(reinterpret_cast<const uint4 *>(Q.qobj + (size_t)s * Q.nqpad + q));
                uint32_t ob[4] = {oq.x, oq.y, oq.z, oq.w}, runs[4] = {0, 0, 0, 0};
                uint32_t e4 = 0;
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    uint32_t ex = 0xFFu;
                    if (ob[x] != kWideNone && (ob[x] & kWideRun)) {
                        const uint64_t from = ob[x] & ~kWideRun, end = Q.qoffs[q + x + 1] - Q.qoffs[0];
                        const uint64_t mask = (1ull << Q.obj_bits) - 1, ctx = __ldg(Q.qkeys + from) >> Q.obj_bits;
                        for (uint64_t i = from; i < end; ++i, ++runs[x]) {
                            const uint64_t key = __ldg(Q.qkeys + i);
                            if (key >> Q.obj_bits != ctx)
                                break;
                            ex = min(ex, wide_e((uint32_t)(key & mask), major));
                        }
                    } else if (ob[x] != kWideNone) {
                        ex = wide_e(ob[x], major);
                    }
                    e4 |= ex << (8 * x);
                }
                if (q < Q.nqpad) {
                    const WideWords w = wide_words(e4);
#pragma unroll
                    for (int m = 0; m < kWideRows; ++m)
                        *reinterpret_cast<uint32_t *>(Q.Y + m * Q.ys + (size_t)s * Q.nqpad + q) = w.w[m];
                }
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const uint32_t ex = (e4 >> (8 * x)) & 0xFFu;
                    for (unsigned several = __ballot_sync(0xffffffffu, runs[x] != 0); several; several &= several - 1) {
                        const int src = __ffs(several) - 1;
                        const uint64_t from = __shfl_sync(0xffffffffu, ob[x], src) & ~kWideRun;
                        const uint32_t run = __shfl_sync(0xffffffffu, runs[x], src);
                        const uint32_t ea = __shfl_sync(0xffffffffu, ex, src);
                        const uint32_t mask = (1u << Q.obj_bits) - 1u;
                        unsigned long long *row = corr + (size_t)(q0 + 4 * src + x) * nref;
                        for (uint32_t j = lane; j < nm; j += 32) {
                            const unsigned long long c = minor[j];
                            const uint32_t rc = (uint32_t)(c >> 32), er = rc >> kGidBits;
                            uint32_t d = (uint32_t)kMinInit;
                            for (uint32_t i = 0; i < run; ++i)
                                d = min(d, (uint32_t)dna_pop(((uint32_t)__ldg(Q.qkeys + from + i) & mask) ^ major ^ (uint32_t)c));
                            // the products count a difference, two where the run has no object
                            // at the major one or the genome's is two away, and ea + er of it
                            const uint32_t two = ea ? 1u : er >= 2 ? 1u : 0u;
                            const unsigned long long w = (unsigned long long)(two - (d >= 2 ? 1u : 0u)) |
                                                         ((unsigned long long)(d == 0) << 21) |
                                                         ((unsigned long long)(ea + er - d) << 42);
                            if (w)
                                atomicAdd(row + (rc & ((1u << kGidBits) - 1)), w);
                        }
                    }
                    for (unsigned away = __ballot_sync(0xffffffffu, ex != 0 && ex != 0xFFu && runs[x] == 0); away;
                         away &= away - 1) {
                        const int src = __ffs(away) - 1;
                        const uint32_t oa = __shfl_sync(0xffffffffu, ob[x], src) ^ major;
                        const uint32_t ea = __shfl_sync(0xffffffffu, ex, src);
                        unsigned long long *row = corr + (size_t)(q0 + 4 * src + x) * nref;
                        for (uint32_t j = lane; j < nm; j += 32) {
                            const unsigned long long c = minor[j];
                            const uint32_t rc = (uint32_t)(c >> 32);
                            const unsigned long long w = wide_correction(oa, (uint32_t)c, ea, rc >> kGidBits);
                            if (w)
                                atomicAdd(row + (rc & ((1u << kGidBits) - 1)), w);
                        }
                    }
                }
            }
            __syncwarp();  // the warp's shared memory is reused by its next group
            continue;
        }
        // Only pairs with a base in common among their differences from the major object are
        // corrected (bases_only: objects too short to pass the cap without one), so for every
        // base the genomes that differ there are listed and their pairs compared, a pair at its
        // first common base.  In one species a list holds a tenth of the genomes away, so all
        // ten lists a tenth of their pairs (1,024 genomes: 139 -> 101 us).
        uint32_t bases = 0;
        const bool by_base = bases_only && nm <= npad / 2;  // a list fits
        if (by_base) {
            for (uint32_t i = lane; i < nm; i += 32)
                bases |= wide_bases((uint32_t)minor[i]);
            bases = __reduce_or_sync(0xffffffffu, bases);
        }
        unsigned short *list16 = reinterpret_cast<unsigned short *>(emap);  // the rows are written
        for (uint32_t left = bases; left; left &= left - 1) {
            const uint32_t bit = left & (0u - left);
            uint32_t nb = 0;
            __syncwarp();
            for (uint32_t i0 = 0; i0 < nm; i0 += 32) {
                const uint32_t i = i0 + lane;
                const bool here = i < nm && (wide_bases((uint32_t)minor[i]) & bit);
                const unsigned m = __ballot_sync(0xffffffffu, here);
                if (here)
                    list16[nb + __popc(m & ((1u << lane) - 1u))] = (unsigned short)i;
                nb += __popc(m);
            }
            __syncwarp();
            const uint32_t np = nb * (nb - 1) / 2;
            for (uint32_t t = lane; t < np; t += 32) {
                uint32_t i, j;
                pair_of_rank(t, i, j);
                const unsigned long long a = minor[list16[j]], c = minor[list16[i]];  // j's genome is the higher
                if (wide_bases((uint32_t)a) & wide_bases((uint32_t)c) & (bit - 1))
                    continue;
                const uint32_t qa = (uint32_t)(a >> 32), rc = (uint32_t)(c >> 32);
                const uint32_t g = qa & ((1u << kGidBits) - 1);
                const unsigned long long w = wide_correction((uint32_t)a, (uint32_t)c, qa >> kGidBits, rc >> kGidBits);
                atomicAdd(corr + g * (g - 1) / 2 + (rc & ((1u << kGidBits) - 1)), w);  // g < 2^12
            }
        }
        // else all pairs (i, j), j < i: kWidePairs genomes i against lanes on consecutive j
        // (postings ascend by gid, so i is the pair's higher genome)
        for (uint32_t i0 = 1; i0 < nm && !by_base; i0 += kWidePairs) {
            uint32_t oq[kWidePairs], eq[kWidePairs];
            unsigned long long *row[kWidePairs];
#pragma unroll
            for (uint32_t x = 0; x < kWidePairs; ++x) {
                const unsigned long long a = minor[min(i0 + x, nm - 1)];
                const uint32_t g = (uint32_t)(a >> 32) & ((1u << kGidBits) - 1);
                oq[x] = (uint32_t)a;
                eq[x] = (uint32_t)(a >> 32) >> kGidBits;
                row[x] = corr + g * (g - 1) / 2;  // g < 2^12
            }
            const uint32_t i1 = min(i0 + kWidePairs, nm);
            for (uint32_t j = lane; j + 1 < i1; j += 32) {
                const unsigned long long c = minor[j];
                const uint32_t rc = (uint32_t)(c >> 32), er = rc >> kGidBits, gr = rc & ((1u << kGidBits) - 1);
#pragma unroll
                for (uint32_t x = 0; x < kWidePairs; ++x) {
                    const unsigned long long w = wide_correction(oq[x], (uint32_t)c, eq[x], er);
                    if (w && j < i0 + x && i0 + x < nm)
                        atomicAdd(row[x] + gr, w);
                }
            }
        }
        __syncwarp();  // the warp's shared memory is reused by its next group
    }
}

// The counters of one pair from its six products and its correction word, added to the cell.
__device__ __forceinline__ void wide_credit(const int32_t *g, size_t gs, unsigned long long corr,
                                            unsigned long long *oc, unsigned long long *oo)
{
    const uint32_t p = (uint32_t)g[0], z = (uint32_t)g[gs], l = (uint32_t)g[2 * gs], u = (uint32_t)g[3 * gs],
                   s = (uint32_t)g[4 * gs], e = (uint32_t)g[5 * gs];
    const uint32_t mut2 = p - l + u - ((uint32_t)corr & 0x1FFFFFu);
    const uint32_t diff = p - z - ((uint32_t)(corr >> 21) & 0x1FFFFFu);
    const uint32_t sect = s - e - p - (uint32_t)(corr >> 42);
    if (p) {
        *oc += (unsigned long long)p | ((unsigned long long)mut2 << 32);
        *oo += (unsigned long long)diff | ((unsigned long long)sect << 32);
    }
}

// One pass's products (G[m][q][r] at G + m * gs + q * npad + r, at least the cells q > r)
// and corrections added into the packed triangle; the corrections are left zero.
__global__ void __launch_bounds__(256) k_wide_lower(const int32_t *__restrict__ G, size_t gs, uint32_t npad,
                                                    size_t cells, unsigned long long *__restrict__ corr,
                                                    unsigned long long *__restrict__ oc,
                                                    unsigned long long *__restrict__ oo)
{
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < cells; c += (size_t)gridDim.x * blockDim.x) {
        uint32_t q = (uint32_t)((1.0 + sqrt(1.0 + 8.0 * (double)c)) * 0.5);
        while ((size_t)q * (q - 1) / 2 > c)
            --q;
        while ((size_t)(q + 1) * q / 2 <= c)
            ++q;
        const uint32_t r = (uint32_t)(c - (size_t)q * (q - 1) / 2);
        wide_credit(G + (size_t)q * npad + r, gs, corr[c], oc + c, oo + c);
        corr[c] = 0;
    }
}

// The same for a block of queries: cell (q, r) of rows of nref references.
__global__ void __launch_bounds__(256) k_wide_block(const int32_t *__restrict__ G, size_t gs, uint32_t npad,
                                                    uint32_t nq, uint32_t nref, unsigned long long *__restrict__ corr,
                                                    unsigned long long *__restrict__ oc,
                                                    unsigned long long *__restrict__ oo)
{
    const size_t cells = (size_t)nq * nref;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < cells; c += (size_t)gridDim.x * blockDim.x) {
        const uint32_t q = (uint32_t)(c / nref), r = (uint32_t)(c - (size_t)q * nref);
        wide_credit(G + (size_t)q * npad + r, gs, corr[c], oc + c, oo + c);
        corr[c] = 0;
    }
}
