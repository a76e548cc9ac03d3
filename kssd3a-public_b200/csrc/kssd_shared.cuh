// The shared contexts of a conflict-free index (groups of at least two postings) laid out
// for the self join, and the join over them.  Included by kssdgpu.cu inside its namespace.
//
// Most contexts of an index belong to one genome (2,000 genomes of 200 species: 29.7 of
// 30.7 million), so a join that finds the shared ones among all of them reads 123 MB of
// bounds for 1.0 million groups.  The index therefore keeps a list of its shared groups,
// made once at its build: narrow groups before wide ones (kssd_wide.cuh), in each part the
// small ones (at most kSharedSmall genomes) before the large, and those by lowest genome.
// Groups of one species stand side by side then, and the pairs of a stretch of the list
// fall on the few cells of that species.
//
// The small groups are cut into blocks of about kBlockPairs pairs.  A block's genomes have
// numbers of their own (its table holds them), its postings are copied with those numbers
// in place of the genomes, so that a pair's cell is a triangular index into counts that a
// CTA keeps in shared memory: one atomic per touched cell and counter word leaves the CTA,
// where an atomic per pair made 9.7 million onto 18,000 addresses.
#pragma once

constexpr uint32_t kSharedSmall = 32;   // genomes of a small group, at most
constexpr uint32_t kPairRanks = kSharedSmall * (kSharedSmall - 1) / 2;
constexpr int kBlockLog = 11;
constexpr uint32_t kBlockPairs = 1u << kBlockLog;  // a block: the groups whose first pair lies in a stretch of these
constexpr uint32_t kBlockMost = kBlockPairs - 1 + kPairRanks;                    // its pairs, at most
constexpr uint32_t kBlockPostings = 2 * (kBlockPairs - 1) + kSharedSmall;        // its postings, at most
constexpr uint32_t kBlockGenomes = 64;  // genomes of a block whose postings are numbered
constexpr uint32_t kBlockCells = kBlockGenomes * (kBlockGenomes - 1) / 2;
constexpr uint32_t kBlockSlots = 128;   // hash slots for them
// objects of at most kPackBits bits share a word with the genome's number (the usual case:
// 20 bits); wider ones keep the numbers in an array of bytes
constexpr int kPackBits = 26;
constexpr uint32_t kPackMask = (1u << kPackBits) - 1;
static_assert(kBlockGenomes <= 1u << (32 - kPackBits), "a number fits beside a packed object");
constexpr uint32_t kNoGenome = 0xFFFFFFFFu;

struct SharedGroup {
    uint32_t begin, k;  // first posting in the index, postings
};

struct SharedBlock {
    uint32_t group, groups;      // its groups in the list
    uint32_t posting, postings;  // its postings in the copy
    uint32_t pairs, genomes;     // genomes: 0 for a block of too many
    uint32_t pad[2];
};

// Each shared group's sort key (wide or not, large or small, lowest genome) and its (begin
// | k << 32), in any order: a tile of groups takes its places with one atomic (one per warp
// and 32 groups queued up on the counter: 218 us for 12.2 million groups).
__global__ void __launch_bounds__(kScanThreads) k_shared_collect(const uint32_t *__restrict__ gbeg, uint64_t u,
                                                                 const uint64_t *__restrict__ post, uint32_t wide,
                                                                 int gid_bits, uint32_t *__restrict__ key,
                                                                 unsigned long long *__restrict__ val,
                                                                 unsigned int *__restrict__ count)
{
    using Scan = cub::BlockScan<uint32_t, kScanThreads>;
    __shared__ typename Scan::TempStorage scan_tmp;
    __shared__ uint32_t base;
    const uint64_t ntiles = (u + kScanTile - 1) / kScanTile;
    for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        uint32_t bnd[kScanPerThread + 1];
        scan_load_bounds(gbeg, u, t, bnd);
        uint32_t mine = 0;
#pragma unroll
        for (uint32_t j = 0; j < kScanPerThread; ++j)
            mine += bnd[j + 1] - bnd[j] >= 2;
        uint32_t off, tot;
        Scan(scan_tmp).ExclusiveSum(mine, off, tot);
        if (threadIdx.x == 0)
            base = atomicAdd(count, tot);
        __syncthreads();
        uint32_t at = base + off;
#pragma unroll
        for (uint32_t j = 0; j < kScanPerThread; ++j) {
            const uint32_t b = bnd[j], k = bnd[j + 1] - b;
            if (k >= 2) {
                key[at] = (uint32_t)(__ldg(post + b) >> 32) | (k > kSharedSmall ? 1u << gid_bits : 0u) |
                          (k >= wide ? 2u << gid_bits : 0u);
                val[at++] = (unsigned long long)b | ((unsigned long long)k << 32);
            }
        }
        __syncthreads();  // the base and the scan storage are reused by the next tile
    }
}

// Running sums over the sorted groups: the small groups' pairs and postings.
struct SharedSums {
    unsigned long long pairs, postings;
};
struct SharedSize {
    __host__ __device__ SharedSums operator()(unsigned long long val) const
    {
        const unsigned long long k = val >> 32;
        return k <= kSharedSmall ? SharedSums{k * (k - 1) / 2, k} : SharedSums{0, 0};
    }
};
struct SharedAdd {
    __host__ __device__ SharedSums operator()(const SharedSums &a, const SharedSums &b) const
    {
        return SharedSums{a.pairs + b.pairs, a.postings + b.postings};
    }
};

// A run of small groups in the list: [group, group + groups), holding `pairs` pairs from
// running sum `before` on; its blocks are [block, block + ceil(pairs / kBlockPairs)).
struct SharedRun {
    uint32_t group, groups, block;
    unsigned long long pairs;
};

// mark[run.block + b] = the first group of the run whose first pair is at or past b *
// kBlockPairs (one past the run when there is none), for b = 0 .. its blocks.
__global__ void k_shared_marks(const SharedSums *__restrict__ sums, const SharedRun run, uint32_t *__restrict__ mark)
{
    const unsigned long long before = sums[run.group].pairs;
    const uint32_t blocks = (uint32_t)((run.pairs + kBlockPairs - 1) >> kBlockLog);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < run.groups; i += gridDim.x * blockDim.x) {
        const unsigned long long p = sums[run.group + i].pairs - before;
        // block b starts at this group when b * kBlockPairs is past the group before it
        const unsigned long long lo = i == 0 ? 0 : ((sums[run.group + i - 1].pairs - before) >> kBlockLog) + 1;
        for (unsigned long long b = lo; b << kBlockLog <= p; ++b)
            mark[run.block + b] = run.group + i;
        if (i == run.groups - 1)
            for (unsigned long long b = (p >> kBlockLog) + 1; b <= blocks; ++b)
                mark[run.block + b] = run.group + run.groups;
    }
}

// The list itself.
__global__ void k_shared_list(const unsigned long long *__restrict__ val, uint32_t n, SharedGroup *__restrict__ list)
{
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x)
        list[g] = SharedGroup{(uint32_t)val[g], (uint32_t)(val[g] >> 32)};
}

// One CTA per block of a run: its header, the groups' places in it (first pair | first
// posting << 12), the copied postings (objects and genome numbers, in one word with pack)
// and the genome table.
static_assert(kBlockMost < 1u << 12 && kBlockPostings < 1u << 20, "packed places");
__global__ void __launch_bounds__(256) k_shared_blocks(const SharedGroup *__restrict__ list, int pack,
                                                       const SharedSums *__restrict__ sums, const SharedRun run,
                                                       const uint32_t *__restrict__ mark,
                                                       const uint64_t *__restrict__ post,
                                                       SharedBlock *__restrict__ blocks, uint32_t *__restrict__ place,
                                                       uint32_t *__restrict__ object,
                                                       unsigned char *__restrict__ number, uint32_t *__restrict__ table)
{
    __shared__ uint32_t slot[kBlockSlots];
    __shared__ unsigned char num[kBlockSlots];
    __shared__ uint32_t given;
    const uint32_t b = run.block + blockIdx.x, g0 = mark[b], g1 = mark[b + 1];
    SharedBlock h{g0, g1 - g0, 0, 0, 0, 0, {0, 0}};
    if (g0 == g1) {  // the tail of a group that starts in the block before
        if (threadIdx.x == 0)
            blocks[b] = h;
        return;
    }
    const SharedSums s0 = sums[g0], last = sums[g1 - 1];
    const uint32_t kl = list[g1 - 1].k;
    h.posting = (uint32_t)s0.postings;
    h.postings = (uint32_t)(last.postings - s0.postings) + kl;
    h.pairs = (uint32_t)(last.pairs - s0.pairs) + kl * (kl - 1) / 2;
    if (threadIdx.x < kBlockSlots)
        slot[threadIdx.x] = kNoGenome;
    __syncthreads();
    bool full = false;
    for (uint32_t g = g0 + threadIdx.x; g < g1; g += blockDim.x) {
        const SharedGroup w = list[g];
        const SharedSums s = sums[g];
        place[g] = (uint32_t)(s.pairs - s0.pairs) | ((uint32_t)(s.postings - s0.postings) << 12);
        for (uint32_t i = 0; i < w.k; ++i) {
            const uint64_t p = __ldg(post + w.begin + i);
            const uint32_t gid = (uint32_t)(p >> 32);
            uint32_t at = (gid * 2654435761u) >> 25, probe = 0;
            for (; probe < kBlockSlots; ++probe) {
                uint32_t have = *(volatile uint32_t *)&slot[at];
                if (have == kNoGenome) {
                    have = atomicCAS(&slot[at], kNoGenome, gid);
                    if (have == kNoGenome)
                        have = gid;
                }
                if (have == gid)
                    break;
                at = (at + 1) & (kBlockSlots - 1);
            }
            full |= probe == kBlockSlots;
            object[s.postings + i] = (uint32_t)p;
            number[s.postings + i] = (unsigned char)at;  // the slot, until the numbers are known
        }
    }
    full = __syncthreads_or(full);
    if (threadIdx.x < 32) {  // numbers in slot order
        uint32_t n = 0;
        for (uint32_t i = threadIdx.x; i < kBlockSlots; i += 32) {
            const uint32_t gid = slot[i];
            const unsigned used = __ballot_sync(0xffffffffu, gid != kNoGenome);
            const uint32_t at = n + __popc(used & ((1u << threadIdx.x) - 1u));
            num[i] = (unsigned char)at;
            if (gid != kNoGenome && at < kBlockGenomes)
                table[(size_t)b * kBlockGenomes + at] = gid;
            n += __popc(used);
        }
        if (threadIdx.x == 0)
            given = n;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < h.postings; i += blockDim.x) {  // written by this CTA, behind the barriers
        const uint32_t at = num[number[h.posting + i] & (kBlockSlots - 1)];
        if (pack)
            object[h.posting + i] |= at << kPackBits;
        else
            number[h.posting + i] = (unsigned char)at;
    }
    h.genomes = full || given > kBlockGenomes ? 0 : given;
    if (threadIdx.x == 0)
        blocks[b] = h;
}

// The pair (i < j) of rank t among a group's pairs: j (j - 1) / 2 <= t.
__device__ __forceinline__ void pair_of_rank(uint32_t t, uint32_t &i, uint32_t &j)
{
    j = (uint32_t)((1.0f + sqrtf(1.0f + 8.0f * (float)t)) * 0.5f);
    while (j * (j - 1) / 2 > t)
        --j;
    while ((j + 1) * j / 2 <= t)
        ++j;
    i = t - j * (j - 1) / 2;
}

struct PairSmem {
    uint32_t ctx[kBlockCells];             // num_ctx | num_mut2_ctx << 16
    uint32_t obj[kBlockCells];             // diff_obj | diff_obj_section << 16
    uint32_t object[kBlockPostings];
    uint32_t place[kBlockPairs + 2];
    unsigned short pair[kBlockCells];      // (i, j) of a pair's rank or a cell's number: i | j << 8
    uint32_t gid[kBlockGenomes];
    unsigned char number[kBlockPostings];  // last: not there when objects are packed
};
// counts in halves of a word (32-bit shared-memory atomics are native, 64-bit ones a loop)
static_assert(kBlockMost * (uint32_t)kMinInit < 65536, "packed counts of a block");
static_assert(kPairRanks <= kBlockCells, "one table of pairs for both");

__device__ __forceinline__ void credit_cell(unsigned long long *__restrict__ oc, unsigned long long *__restrict__ oo,
                                            uint32_t qg, uint32_t rg, unsigned long long c, unsigned long long o)
{
    const size_t cell = lower_cell(qg, rg);
    atomicAdd(oc + cell, c);
    if (o)
        atomicAdd(oo + cell, o);
}

// The pairs of blocks [0, nblocks).  A CTA copies a block into shared memory, every thread
// takes a stretch of its pairs (one search for the first one's group, then steps) and adds
// each to its cell's counts, which go to the triangle at the block's end.  A block of more
// than kBlockGenomes genomes credits the triangle pair by pair.
//
// Bound by the shared-memory pipe (73 %: lanes on their own stretches meet in banks, and
// in cells).  Measured (B200, whole calls; before: a scan of all groups' bounds with an
// atomic per pair): 2,000 genomes of 200 species 117 -> 44 us, 6,000 of 600 425 -> 145 us
// (its 288 MB fill 46), 400 in species of 24 330 -> 111 us.  A hash of cells instead of
// block numbers measured 66 us at 2,000 genomes and 604 us at 400 (a probe per pair),
// numbers found by every join 87 and 158 us.
constexpr uint32_t kPairThreads = 256;
template <bool PACK>
__global__ void __launch_bounds__(kPairThreads, PACK ? 5 : 4) k_self_pairs(const SharedBlock *__restrict__ blocks,
                                                                uint32_t nblocks, const SharedGroup *__restrict__ list,
                                                                const uint32_t *__restrict__ place,
                                                                const uint32_t *__restrict__ object,
                                                                const unsigned char *__restrict__ number,
                                                                const uint32_t *__restrict__ table,
                                                                const uint64_t *__restrict__ post,
                                                                unsigned long long *__restrict__ oc,
                                                                unsigned long long *__restrict__ oo)
{
    extern __shared__ __align__(16) unsigned char pair_smem[];
    PairSmem &S = *reinterpret_cast<PairSmem *>(pair_smem);
    for (uint32_t t = threadIdx.x; t < kBlockCells; t += kPairThreads) {
        S.ctx[t] = 0;
        S.obj[t] = 0;
        uint32_t i, j;
        pair_of_rank(t, i, j);
        S.pair[t] = (unsigned short)(i | (j << 8));
    }
    bool waited = false;
    for (uint32_t c = blockIdx.x; c < nblocks; c += gridDim.x) {
        const uint4 h0 = __ldg(reinterpret_cast<const uint4 *>(blocks + c));
        const uint4 h1 = __ldg(reinterpret_cast<const uint4 *>(blocks + c) + 1);
        const uint32_t group = h0.x, groups = h0.y, posting = h0.z, postings = h0.w, pairs = h1.x, genomes = h1.y;
        if (groups == 0)
            continue;
        for (uint32_t i = threadIdx.x; i < groups; i += kPairThreads)
            S.place[i] = __ldg(place + group + i);
        if (threadIdx.x == 0)
            S.place[groups] = pairs;
        if (genomes) {
            for (uint32_t i = threadIdx.x; i < postings; i += kPairThreads) {
                S.object[i] = __ldg(object + posting + i);
                if (!PACK)
                    S.number[i] = __ldg(number + posting + i);
            }
            if (threadIdx.x < genomes)
                S.gid[threadIdx.x] = __ldg(table + (size_t)c * kBlockGenomes + threadIdx.x);
        }
        __syncthreads();
        if (!waited) {
            pdl_wait_primary();  // the counters' zero fill has finished (no-op without a dependency)
            waited = true;
        }
        const uint32_t each = (pairs + kPairThreads - 1) / kPairThreads;
        uint32_t t = threadIdx.x * each;
        if (t < pairs) {
            uint32_t lo = 0, hi = groups - 1;  // the last group whose first pair is at or before t
            while (lo < hi) {
                const uint32_t mid = (lo + hi + 1) >> 1;
                if ((S.place[mid] & 0xFFFu) <= t)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            uint32_t q = lo, at = S.place[q], next = S.place[q + 1] & 0xFFFu;
            const uint32_t ij = S.pair[t - (at & 0xFFFu)];
            uint32_t i = ij & 0xFFu, j = ij >> 8;
            const uint32_t t1 = min(t + each, pairs);
            if (genomes) {
                uint32_t oy = S.object[(at >> 12) + j], ny = PACK ? oy >> kPackBits : S.number[(at >> 12) + j];
                for (;;) {
                    const uint32_t ox = S.object[(at >> 12) + i], nx = PACK ? ox >> kPackBits : S.number[(at >> 12) + i];
                    const uint32_t d = (uint32_t)min(kMinInit, dna_pop((ox ^ oy) & (PACK ? kPackMask : ~0u)));
                    const uint32_t w = max(nx, ny), cell = w * (w - 1) / 2 + min(nx, ny);
                    atomicAdd(&S.ctx[cell], 1u | (d > 1 ? 0x10000u : 0u));
                    if (d)
                        atomicAdd(&S.obj[cell], 1u | (d << 16));
                    if (++t >= t1)
                        break;
                    ++i;
                    if (t == next || i == j) {  // the next genome, or group (every group holds a pair)
                        ++j;
                        i = 0;
                        if (t == next) {
                            ++q;
                            at = S.place[q];
                            next = S.place[q + 1] & 0xFFFu;
                            j = 1;
                        }
                        oy = S.object[(at >> 12) + j];
                        ny = PACK ? oy >> kPackBits : S.number[(at >> 12) + j];
                    }
                }
            } else {
                for (;;) {
                    const uint64_t *p = post + __ldg(&list[group + q].begin);
                    const uint64_t pi = __ldg(p + i), pj = __ldg(p + j);
                    const int d = min(kMinInit, dna_pop((uint32_t)pi ^ (uint32_t)pj));
                    credit_cell(oc, oo, (uint32_t)(pj >> 32), (uint32_t)(pi >> 32), inc_ctx(d), d ? inc_obj(d) : 0);
                    if (++t >= t1)
                        break;
                    ++i;
                    if (t == next) {
                        ++q;
                        next = S.place[q + 1] & 0xFFFu;
                        i = 0;
                        j = 1;
                    } else if (i == j) {
                        ++j;
                        i = 0;
                    }
                }
            }
        }
        __syncthreads();
        for (uint32_t x = threadIdx.x; x < genomes * (genomes - 1) / 2; x += kPairThreads) {
            const uint32_t cc = S.ctx[x], co = S.obj[x];
            if (cc) {
                const uint32_t ab = S.pair[x], a = S.gid[ab & 0xFFu], b = S.gid[ab >> 8];
                credit_cell(oc, oo, max(a, b), min(a, b),
                            (unsigned long long)(cc & 0xFFFFu) | ((unsigned long long)(cc >> 16) << 32),
                            (unsigned long long)(co & 0xFFFFu) | ((unsigned long long)(co >> 16) << 32));
                S.ctx[x] = 0;
                S.obj[x] = 0;
            }
        }
        __syncthreads();  // the block's tables are reused by the next
    }
    // A CTA without a block waits too: the next kernel on the stream is ordered behind this one
    // alone, and must not start while the fill still runs.
    if (!waited)
        pdl_wait_primary();
}

// Large groups, one CTA each: a warp takes every eighth genome j, its lanes consecutive
// genomes below it, so that a warp's credits of one row are neighbours.
__global__ void __launch_bounds__(256) k_self_large(const SharedGroup *__restrict__ list, uint32_t n,
                                                    const uint64_t *__restrict__ post,
                                                    unsigned long long *__restrict__ oc,
                                                    unsigned long long *__restrict__ oo)
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t g = blockIdx.x; g < n; g += gridDim.x) {
        const SharedGroup w = list[g];
        for (uint32_t j = 1 + warp; j < w.k; j += 8) {
            const uint64_t pj = __ldg(post + w.begin + j);
            for (uint32_t i = lane; i < j; i += 32) {
                const uint64_t pi = __ldg(post + w.begin + i);
                const int d = min(kMinInit, dna_pop((uint32_t)pi ^ (uint32_t)pj));
                credit_cell(oc, oo, (uint32_t)(pj >> 32), (uint32_t)(pi >> 32), inc_ctx(d), d ? inc_obj(d) : 0);
            }
        }
    }
}
