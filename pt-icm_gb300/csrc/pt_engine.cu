// pt_engine.cu -- the PT-ICM engine for sm_103a.
//
// One persistent kernel runs `nsteps` parallel-tempering steps for a batch of
// instances.  A step is, as in the reference's solve loop
// (src/solver.cc:67-127):
//   1. Metropolis sweeps of every replica        (src/replica.cc:5-38)
//   2. replica exchange, chains*(nt-1) attempts  (src/replica_exchange.cc:5-100)
//   3. isoenergetic cluster moves on the nc coldest temperatures
//                                                (src/icm.cc:8-215)
//
// Layout: every replica of an instance lives in shared memory of the block
// that owns it (int8 spins, int32 local fields f_i = sum_j J_ij s_j), the
// adjacency is staged into shared memory by bulk (TMA) copies, and exchange
// permutes the slot->replica map instead of moving spins.  A block owns `rpc`
// replicas of one instance; `group` blocks share an instance and meet at a
// bounded grid barrier once per step (cooperative launch).
//
// Production sweeps visit the sites colour class by colour class (no two
// sites of a class are adjacent) with Philox uniforms compared against
// per-temperature integer thresholds ceil(exp(-beta*dE) * 2^32), computed on
// the host in FP64.  The replay variant visits sites in the reference's
// sequential order and consumes a recorded uniform stream with FP64
// exp(-beta*dE) tables, reproducing the reference bit for bit.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdio>

#include "pticm_device.cuh"
#include "pticm_engine.h"

namespace pticm {

template <typename T>
__device__ __forceinline__ T* sm_ptr(uint8_t* base, uint32_t off) {
    return reinterpret_cast<T*>(base + off);
}

// Thread-0 phase timers (clock64), enabled by EngineArgs::prof; the marks and
// counters live in shared memory, so that an unprofiled run keeps nothing of
// them in registers.
struct ProfStore {
    long long mark, sub;
    long long c[PROF_PHASES];
};
struct Prof {
    bool on;
    ProfStore* s;
    __device__ __forceinline__ void init() const {
        if (!on) return;
        s->mark = s->sub = clock64();
        for (int q = 0; q < PROF_PHASES; q++) s->c[q] = 0;
    }
    __device__ __forceinline__ void tick(int slot) const {
        if (on) { const long long t = clock64(); s->c[slot] += t - s->mark; s->mark = t; s->sub = t; }
    }
    __device__ __forceinline__ void subtick(int slot) const {
        if (on) { const long long t = clock64(); s->c[slot] += t - s->sub; s->sub = t; }
    }
};

// ------------------------------------------------------------ union-find
// Concurrent union-find in shared memory: roots are hooked larger-under-
// smaller with CAS (parent indices strictly decrease, so no cycle forms) and
// finds halve paths.  Loops are capped; -1 / false report the cap.
__device__ __forceinline__ int uf_find(volatile int* parent, int x) {
    for (int it = 0; it < (1 << 20); it++) {
        const int p = parent[x];
        if (p == x) return x;
        const int gp = parent[p];
        if (gp == p) return p;
        parent[x] = gp;
        x = gp;
    }
    return -1;
}

__device__ __forceinline__ bool uf_unite(int* parent, int a, int b) {
    volatile int* vp = parent;
    for (int it = 0; it < (1 << 20); it++) {
        a = uf_find(vp, a);
        b = uf_find(vp, b);
        if (a < 0 || b < 0) return false;
        if (a == b) return true;
        if (a < b) { const int t = a; a = b; b = t; }
        if (atomicCAS(parent + a, a, b) == a) return true;
    }
    return false;
}

// ---------------------------------------------------------- team helpers
// An ICM "team" is either one warp (many pairs per block) or the whole block
// (one pair per block).  A warp reduces with redux instructions; the warps of
// a block team meet in shared memory, with one barrier per reduction: keys in
// a slot per warp, sums by one 32-bit atomic per warp (64-bit shared atomic
// minima are compare-and-swap loops: sixteen warps queueing on them took
// 0.5 us per reduction).
__device__ __forceinline__ unsigned long long warp_min(unsigned long long k) {
    const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t)(k >> 32));
    const uint32_t lo = __reduce_min_sync(0xffffffffu, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0xFFFFFFFFu);
    return ((unsigned long long)hi << 32) | lo;
}

// Control words of a team in shared memory (a warp team uses the first two).
enum TeamCtl : int {
    TC_BEST = 0,      // warp team: the giant component's root
    TC_TAIL = 1,      // breadth-first queue tail
    TC_OVERLAP = 2,   // overlap sites listed, zero between pairs
    TC_OTHERS = 3,    // other sites listed, zero between pairs
    TC_S = 4,         // sites listed outside the giant component, zero between pairs
    TC_STALE = 5,     // a published word had not arrived, zero between pairs
    TC_COUNT = 6,     // a sum of counts; zeroed when a pair begins
    TC_EXPIRED = 7,   // the wait for published words ran out
    TC_DE = 8,        // two 64-bit energy changes; zeroed when a pair begins
    TC_DEADLINE = 12, // 64-bit time at which that wait ends (a warp team's lies in its two words)
    TC_WORDS = 16
};

template <bool BLOCK>
struct Team {
    int tr, ts;                  // rank and size
    int* ctl;                    // control words (shared)
    unsigned long long* keys;    // block team: two keys per warp (shared)
    __device__ __forceinline__ void sync() const {
        if (BLOCK) __syncthreads(); else __syncwarp();
    }
    // A pair begins.  The sums' readers of the pair before have passed a
    // barrier since, and one comes before the next use.
    __device__ __forceinline__ void begin() const {
        if (BLOCK && tr == 0) {
            ctl[TC_COUNT] = 0;
            reinterpret_cast<unsigned long long*>(ctl + TC_DE)[0] = 0ull;
            reinterpret_cast<unsigned long long*>(ctl + TC_DE)[1] = 0ull;
        }
    }
    // Sum of a count over the team, once per pair.
    __device__ __forceinline__ int count(int c) const {
        c = __reduce_add_sync(0xffffffffu, c);
        if (!BLOCK) return c;
        if ((threadIdx.x & 31) == 0 && c != 0) atomicAdd(ctl + TC_COUNT, c);
        __syncthreads();
        return *(volatile int*)(ctl + TC_COUNT);
    }
    // Sums of two energy changes, for the thread of rank 0, once per pair.
    // With `small` (all energies within 2^30) both are exact modulo 2^32.
    __device__ __forceinline__ void sum_energies(long long& a, long long& b, bool small) const {
        unsigned long long* const acc = reinterpret_cast<unsigned long long*>(ctl + TC_DE);
        if (small) {
            int x = (int)__reduce_add_sync(0xffffffffu, (unsigned)a), y = (int)__reduce_add_sync(0xffffffffu, (unsigned)b);
            if (BLOCK) {
                if ((threadIdx.x & 31) == 0) {
                    if (x) atomicAdd(reinterpret_cast<int*>(acc), x);
                    if (y) atomicAdd(reinterpret_cast<int*>(acc + 1), y);
                }
                __syncthreads();
                x = *(volatile int*)acc;
                y = *(volatile int*)(acc + 1);
            }
            a = x;
            b = y;
            return;
        }
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (!BLOCK) return;
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(acc, (unsigned long long)a);
            atomicAdd(acc + 1, (unsigned long long)b);
        }
        __syncthreads();
        a = (long long)*(volatile unsigned long long*)acc;
        b = (long long)*(volatile unsigned long long*)(acc + 1);
    }
};

// 64-bit finaliser of splitmix64 (Steele, Lea, Flood, OOPSLA 2014): a
// bijective mixer giving independent-looking keys for consecutive inputs.
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Where a launch's data lives, known at compile time, so that the pointers
// below have a known address space: a shared load or atomic through a
// generic pointer first finds out where it points (on the N=2000 workload
// the sweep, the cluster search and the flips all shorten by a tenth).
enum Space : int {
    SP_ANY = 0,      // found out at run time
    SP_SHARED = 1,   // adjacency staged; replicas, thresholds and cluster scratch in shared memory
    SP_STATE = 2,    // as SP_SHARED, but the adjacency may be in device memory (an instance of a batch)
    SP_LARGE = 3,    // spins and cluster scratch in shared memory; adjacency, thresholds and the overlap list in device memory
    SP_LARGE4 = 4,   // as SP_LARGE with four replicas in the block, their spins interleaved: byte 4 i + j is replica j's site i
};
constexpr bool space_large(int space) { return space == SP_LARGE || space == SP_LARGE4; }
constexpr int space_stride(int space) { return space == SP_LARGE4 ? 4 : 1; }   // bytes between a replica's sites

// One replica's spins in a block.
template <int SPACE>
struct SpinRow {
    int8_t* p;
    __device__ __forceinline__ int8_t& operator[](int i) const { return p[space_stride(SPACE) * i]; }
};

// Per-block view of a job: its descriptor (in shared memory) and pointers,
// which are shared-memory offsets of the launch's plan or device addresses.
struct BlockCtx {
    const InstanceDesc& D;
    int rank, r0;
    const int32_t* row;
    const uint32_t* adj;
    int8_t* spin;
    int32_t* field;     // null: fields are gathered
    const int32_t* h;   // null: no linear terms
    long long* E;
    uint32_t* slot;
    uint32_t* rslot;
    int32_t* tb;        // threshold row base of each local replica
};

template <int SPACE>
__device__ __forceinline__ SpinRow<SPACE> spin_row(const BlockCtx& B, int j) {
    return SpinRow<SPACE>{B.spin + (SPACE == SP_LARGE4 ? j : j * B.D.n_pad)};
}

// ICM team scratch: BFS queue / union-find parents (n ints), overlap flags
// (n bytes), visited bits (icm_team_bytes); a block team's overlap list (n
// ints) follows (icm_block_bytes of the shared-memory plan).
struct IcmScratch {
    int* queue;
    uint8_t* d;
    uint32_t* vis;
    int* list;          // block team only: overlap sites first, the others from the end
};

__device__ __forceinline__ IcmScratch icm_scratch(uint8_t* base, int n_pad) {
    IcmScratch X;
    X.queue = reinterpret_cast<int*>(base);
    X.d = base + (size_t)n_pad * 4;
    X.vis = reinterpret_cast<uint32_t*>(base + (size_t)n_pad * 5);
    X.list = reinterpret_cast<int*>(base + icm_team_bytes(n_pad));
    return X;
}

// Calls f(e) for every packed entry (col << 8 | uint8 J) of site i's
// neighbour list: a scalar head up to a 16-byte boundary, four entries per
// 16-byte load, a scalar tail (plain loads: the list may be staged in shared
// memory; a list that is not 16-byte aligned is walked entry by entry).
// For small bodies only (field gathers and pushes): the body is expanded
// several times, and a large one (union-find) costs more in instruction
// fetch than the wider loads save.
template <class F>
__device__ __forceinline__ void for_each_neighbour(const int32_t* row, const uint32_t* adj, int i, F&& f) {
    int a = row[i];
    const int e1 = row[i + 1];
    if ((reinterpret_cast<uintptr_t>(adj) & 15u) == 0) {
        for (; a < e1 && (a & 3); a++) f(adj[a]);
#pragma unroll 2
        for (; a + 4 <= e1; a += 4) {
            const uint4 q = *reinterpret_cast<const uint4*>(adj + a);
            f(q.x);
            f(q.y);
            f(q.z);
            f(q.w);
        }
    }
    for (; a < e1; a++) f(adj[a]);
}

// ------------------------------------------------------------------ ICM
// One cluster move on the pair (A, B) = (chain 2c, chain 2c+1) at slot k.
// The team computes the overlap (sites where A and B differ), the
// reference's global-flip rule (src/icm.cc:20-28: more than n/2 differing
// sites -> negate A), a seed uniform among differing sites (src/icm.cc:33;
// here the differing site with the smallest per-site random key, which is
// uniform), then finds the seed's cluster C of differing sites -- breadth-
// first, or by labelling the components of the whole overlap (src/icm.cc:
// 37-72 grows it depth-first; the cluster is the same set) -- and flips the
// smaller of C and the rest of the overlap in both replicas.  Fields are
// updated per flipped site (or recomputed when the set is large); energies
// change by -2 s_u h_u per flipped site plus -2 J s_u s_v per edge leaving
// the set (s_v equal in A and B), an exact integer update.  Members held by
// another block are read from the published copy and flipped by their own
// block, which finds the same set -- or, given `result`, the block only writes
// what is to be flipped (apply_pairs).
template <bool BLOCK, bool REPLAY, bool LS, int SPACE, bool GLINK = false>
__device__ __forceinline__ int icm_pair(const EngineArgs& A, const BlockCtx& B, const Team<BLOCK>& team, int q,
                                        int rA, int rB, unsigned long long step, int ls, const IcmScratch& X,
                                        int where_err, const Prof P, unsigned long long* result = nullptr) {
    const InstanceDesc& D = B.D;
    const int n = D.n, npad = D.n_pad;
    const int32_t* const brow = B.row;
    const uint32_t* const badj = B.adj;
    const int32_t* const bh = B.h;
    const bool has_h = bh != nullptr;
    // (share: the result goes to the blocks that hold the replicas, and the
    // published words serve as both states)
    const bool share = space_large(SPACE) && result != nullptr;
    const bool locA = !share && rA >= B.r0 && rA < B.r0 + D.rpc;
    const bool locB = !share && rB >= B.r0 && rB < B.r0 + D.rpc;
    const int parity = (int)(step & 1ull);
    // a member held by another block: its published words of this step
    const unsigned long long* const pub0 = A.spins_pub + parity * A.spins_pub_half + (D.spin_off >> 4);
    const unsigned long long* const pubA = pub0 + (long long)rA * (npad >> 4);
    const unsigned long long* const pubB = pub0 + (long long)rB * (npad >> 4);
    const uint32_t tag = A.pub_base + (uint32_t)ls;
    // (a word that does not carry the tag yet marks the pass stale, and the
    // pass is made again)
    bool stale = false;
    auto pub_bits = [&](unsigned long long w) -> uint32_t {
        stale |= (uint32_t)(w >> 32) != tag;
        return (uint32_t)w;
    };
    // sites 4 w .. 4 w + 3 of a loaded word as +-1 bytes, and one site
    auto quad_bytes = [&](unsigned long long word, int w) -> uint32_t {
        const uint32_t b = (pub_bits(word) >> ((w & 7) * 4)) & 15u;
        return ~(((b * 0x00204081u) & 0x01010101u) * 0xFEu);   // bit set: 0x01, clear: 0xFF
    };
    auto pub_site = [&](const unsigned long long* pub, int i) -> int8_t {
        return ((pub_bits(ld_relaxed_gpu_u64(pub + (i >> 5))) >> (i & 31)) & 1u) ? (int8_t)1 : (int8_t)-1;
    };
    const SpinRow<SPACE> sA = spin_row<SPACE>(B, locA ? rA - B.r0 : 0), sB = spin_row<SPACE>(B, locB ? rB - B.r0 : 0);
    // no stored fields in field_gather mode: field updates are skipped
    int32_t* fA = (locA && B.field) ? B.field + (rA - B.r0) * npad : nullptr;
    int32_t* fB = (locB && B.field) ? B.field + (rB - B.r0) * npad : nullptr;
    uint8_t* d = X.d;
    const int nwords = (n + 31) >> 5;
    P.subtick(PROF_ICM_ENERGY);
    // a caller's seed for this pair (device numbering), or skip the pair
    int forced = -1;
    const bool exact = REPLAY || A.icm_exact != 0;
    if (!REPLAY && A.icm_force != nullptr) {
        const long long f = A.icm_force[q];
        if (f == -2) return 0;
        if (f >= (long long)n || f < -2) {
            if (team.tr == 0) dev_fail(A.status, A.abort_flag, DEV_BAD_INDEX, where_err + 5, q, f);
            return 0;
        }
        if (f >= 0) forced = A.perm[D.perm_off + f];
    }

    // overlap, its size, seed candidates among differing and equal sites
    unsigned long long r64 = 0;
    if (!REPLAY) {
        const uint4 rnd = philox4x32_10(make_uint4((uint32_t)q, (uint32_t)D.inst_id, (uint32_t)step,
                                                   (uint32_t)(step >> 32)), stream_key(A.seed, STREAM_ICM));
        r64 = ((unsigned long long)rnd.y << 32) | rnd.x;
    }
    int cnt = 0;
    unsigned long long kd = ~0ull, ke = ~0ull;
    team.begin();
    const int algo = D.icm_algo;
    auto overlap_site = [&](int i, int8_t a, int8_t b) {
        const bool di = a != b;
        d[i] = di;
        if (algo == ENGINE_ICM_UNION_FIND) X.queue[i] = i;   // union-find parents
        if (!BLOCK) cnt += di;
        if (!REPLAY) {
            const unsigned long long key = (mix64(r64 + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1)) &
                                            0xFFFFFFFF00000000ull) | (unsigned)i;
            if (di) kd = min(kd, key);
            else ke = min(ke, key);
        }
    };
    // a block team lists the overlap sites (from the front) and the others
    // (from the back), so that its later passes visit overlap sites only;
    // the counters are zero between pairs
    int* lst = X.list;
    for (unsigned int tries = 0;; tries++) {
    auto append = [&](bool valid, bool di, int i) {
        const int lane = threadIdx.x & 31;
        const unsigned mf = __ballot_sync(0xffffffffu, valid && di);
        const unsigned mb = __ballot_sync(0xffffffffu, valid && !di);
        int f0 = 0, b0 = 0;
        if (lane == 0) {
            if (mf) f0 = atomicAdd(team.ctl + TC_OVERLAP, __popc(mf));
            if (mb) b0 = atomicAdd(team.ctl + TC_OTHERS, __popc(mb));
        }
        f0 = __shfl_sync(0xffffffffu, f0, 0);
        b0 = __shfl_sync(0xffffffffu, b0, 0);
        const unsigned lt = (1u << lane) - 1u;
        const int pf = f0 + __popc(mf & lt), pb = n - 1 - b0 - __popc(mb & lt);
        if (valid && di && pf < n) lst[pf] = i;
        if (valid && !di && pb >= 0) lst[pb] = i;
    };
    if (BLOCK && LS) {
        // four sites per thread: one 32-bit word of each replica's spins (the
        // partner's expanded from its published bits, which eight threads
        // share one L2 load of), the overlap flags stored as one word, and the sites appended to
        // the list with one warp scan and one atomic per warp and list
        // (rows are n_pad bytes, a multiple of 16: every word is aligned)
        const int lane = threadIdx.x & 31;
        const int nq = (n + 3) >> 2;
        // the next round's words are loaded before this round's are used
        // (a partner's words come from L2)
        auto load_words = [&](int w, unsigned long long& wa, unsigned long long& wb) {
            if (SPACE == SP_LARGE4) {
                // byte j of four words, put together
                const uint4 q = reinterpret_cast<const uint4*>(B.spin)[w];
                auto quad = [&](int j) -> uint32_t {
                    const uint32_t sel = (uint32_t)j | ((uint32_t)(4 + j) << 4);
                    return __byte_perm(__byte_perm(q.x, q.y, sel), __byte_perm(q.z, q.w, sel), 0x5410);
                };
                wa = locA ? quad(rA - B.r0) : ld_relaxed_gpu_u64(pubA + (w >> 3));
                wb = locB ? quad(rB - B.r0) : ld_relaxed_gpu_u64(pubB + (w >> 3));
            } else {
                wa = locA ? reinterpret_cast<const uint32_t*>(sA.p)[w] : ld_relaxed_gpu_u64(pubA + (w >> 3));
                wb = locB ? reinterpret_cast<const uint32_t*>(sB.p)[w] : ld_relaxed_gpu_u64(pubB + (w >> 3));
            }
        };
        unsigned long long na = 0, nb = 0;
        if (team.tr < nq) load_words(team.tr, na, nb);
        for (int w0 = 0; w0 < nq; w0 += team.ts) {
            const int w = w0 + team.tr;
            const bool have = w < nq;
            const unsigned long long ra = na, rb = nb;
            if (w + team.ts < nq) load_words(w + team.ts, na, nb);
            uint32_t dw = 0;
            int fm = 0, bm = 0;
            if (have) {
                const uint32_t wa = locA ? (uint32_t)ra : quad_bytes(ra, w), wb = locB ? (uint32_t)rb : quad_bytes(rb, w);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int i = 4 * w + j;
                    if (i >= n) break;
                    const int8_t a = (int8_t)(wa >> (8 * j)), b = (int8_t)(wb >> (8 * j));
                    const bool di = a != b;
                    dw |= (uint32_t)di << (8 * j);
                    fm |= (int)di << j;
                    bm |= (int)!di << j;
                    const unsigned long long key =
                        (mix64(r64 + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1)) & 0xFFFFFFFF00000000ull) |
                        (unsigned)i;
                    if (di) kd = min(kd, key);
                    else ke = min(ke, key);
                }
                reinterpret_cast<uint32_t*>(d)[w] = dw;
                if (algo == ENGINE_ICM_UNION_FIND)   // union-find parents
                    reinterpret_cast<int4*>(X.queue)[w] = make_int4(4 * w, 4 * w + 1, 4 * w + 2, 4 * w + 3);
            }
            // list positions: both counts packed in one int, one inclusive scan
            const int packed = __popc(fm) | (__popc(bm) << 16);
            int incl = packed;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            int base_f = 0, base_b = 0;
            if (lane == 31) {
                if (incl & 0xffff) base_f = atomicAdd(team.ctl + TC_OVERLAP, incl & 0xffff);
                if (incl >> 16) base_b = atomicAdd(team.ctl + TC_OTHERS, incl >> 16);
            }
            base_f = __shfl_sync(0xffffffffu, base_f, 31);
            base_b = __shfl_sync(0xffffffffu, base_b, 31);
            const int excl = incl - packed;
            int pf = base_f + (excl & 0xffff), pb = n - 1 - (base_b + (excl >> 16));
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if ((fm >> j) & 1) lst[pf++] = 4 * w + j;
                if ((bm >> j) & 1) lst[pb--] = 4 * w + j;
            }
        }
    } else {
        // two sites per round, both loaded first: the partner's spins come
        // from the published copy in L2 (the wide 1024-thread variants keep
        // this shorter code, which needs fewer registers)
        for (int base = 0; base < n; base += 2 * team.ts) {
            const int i = base + team.tr, i2 = i + team.ts;
            int8_t a = 0, b = 0, a2 = 0, b2 = 0;
            if (i < n) {
                a = locA ? sA[i] : pub_site(pubA, i);
                b = locB ? sB[i] : pub_site(pubB, i);
            }
            if (i2 < n) {
                a2 = locA ? sA[i2] : pub_site(pubA, i2);
                b2 = locB ? sB[i2] : pub_site(pubB, i2);
            }
            if (i < n) overlap_site(i, a, b);
            if (i2 < n) overlap_site(i2, a2, b2);
            if (BLOCK) {
                append(i < n, a != b, i);
                append(i2 < n, a2 != b2, i2);
            }
        }
    }
    if (algo == ENGINE_ICM_BFS || share)   // the visited bits of the breadth-first search; the flipped set's
        for (int w = team.tr; w < nwords; w += team.ts) X.vis[w] = 0u;
    // the overlap's size and whether any word was stale; every warp's best
    // seed candidates (a block team takes the one it needs after the barrier)
    bool again;
    if (!REPLAY) {
        kd = warp_min(kd);
        ke = warp_min(ke);
    }
    if (BLOCK) {
        if (!REPLAY && (threadIdx.x & 31) == 0) {
            team.keys[2 * (threadIdx.x >> 5)] = kd;
            team.keys[2 * (threadIdx.x >> 5) + 1] = ke;
        }
        if (stale) *(volatile int*)(team.ctl + TC_STALE) = 1;
        __syncthreads();
        cnt = *(volatile int*)(team.ctl + TC_OVERLAP);
        again = *(volatile int*)(team.ctl + TC_STALE) != 0;
    } else {
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        again = __any_sync(0xffffffffu, stale);
    }
    if (!again) break;
    // a partner's word had not arrived (its block published it before the
    // energy this block waited for, but nothing orders the two): once more,
    // at most as long as any wait on another block, and not when another has
    // ended the run (the deadline lies in shared memory: the passes before it
    // is needed keep no register for it)
    team.sync();
    int expired = 0;
    if (team.tr == 0) {
        volatile unsigned long long* const deadline =
            reinterpret_cast<unsigned long long*>(team.ctl + (BLOCK ? TC_DEADLINE : TC_BEST));
        const unsigned long long t = globaltimer_ns();
        if (tries == 0) *deadline = t + (A.wait_limit_ns ? A.wait_limit_ns : kWaitLimitNs);
        else expired = t > *deadline || *(volatile int*)A.abort_flag != 0;
        if (BLOCK) {
            team.ctl[TC_OVERLAP] = 0;
            team.ctl[TC_OTHERS] = 0;
            team.ctl[TC_STALE] = 0;
            team.ctl[TC_EXPIRED] = expired;
        }
    }
    team.sync();
    expired = BLOCK ? *(volatile int*)(team.ctl + TC_EXPIRED) : __shfl_sync(0xffffffffu, expired, 0);
    if (expired) {
        // (the run ends with this error at the group's next meeting)
        if (team.tr == 0) dev_fail(A.status, A.abort_flag, DEV_BARRIER_TIMEOUT, 4, blockIdx.x, tag);
        return 0;
    }
    stale = false;
    cnt = 0;
    kd = ke = ~0ull;
    }
    const bool gflip = cnt > n / 2;
    if (forced >= 0 && (d[forced] != 0) == gflip) {
        // a caller's seed must be a differing site after the global flip:
        // report it before any state changes (and clear the list counters)
        if (team.tr == 0) dev_fail(A.status, A.abort_flag, DEV_BAD_INDEX, where_err + 6, q, forced);
        team.sync();
        if (BLOCK && team.tr == 0) { team.ctl[TC_OVERLAP] = 0; team.ctl[TC_OTHERS] = 0; team.ctl[TC_S] = 0; }
        team.sync();
        return 0;
    }
    // the overlap list of a block team: [l0, l0 + llen) of lst
    const int l0 = gflip ? cnt : 0, llen = gflip ? n - cnt : cnt;
    auto for_overlap = [&](auto&& f) {
        if (BLOCK) {
            for (int t = team.tr; t < llen; t += team.ts) f(lst[l0 + t]);
        } else {
            for (int u = team.tr; u < n; u += team.ts)
                if (d[u]) f(u);
        }
    };
    long long dEa = 0, dEb = 0;
    if (gflip) {
        for (int i = team.tr; i < n; i += team.ts) {
            if (locA) {
                const int a = sA[i];
                if (has_h) dEa -= 2 * bh[i] * a;   // E(-s) = E(s) - 2 sum h s
                sA[i] = (int8_t)-a;
                if (fA) fA[i] = -fA[i];
            }
            if (share && has_h) dEa -= 2 * bh[i] * pub_site(pubA, i);
            d[i] ^= 1;
        }
        cnt = n - cnt;
        team.sync();
    }
    P.subtick(PROF_ICM_DIFF);
    int seed = -1;
    if (REPLAY) {
        const long long idx = (long long)ls * D.nc + q;
        const long long traced = (idx < (long long)A.replay.n_icm) ? A.replay.icm_seed[idx] : -2;
        if ((traced < 0) != (cnt == 0)) {
            if (team.tr == 0) dev_fail(A.status, A.abort_flag, DEV_REPLAY_MISMATCH, where_err, idx, cnt);
            return 0;
        }
        if (cnt > 0) {
            if (traced >= n) {
                if (team.tr == 0) dev_fail(A.status, A.abort_flag, DEV_BAD_INDEX, where_err + 1, idx, traced);
                return 0;
            }
            seed = A.perm[D.perm_off + traced];
            if (!d[seed]) {
                if (team.tr == 0) dev_fail(A.status, A.abort_flag, DEV_REPLAY_MISMATCH, where_err + 2, idx, seed);
                return 0;
            }
        }
    } else if (cnt > 0) {
        if (BLOCK) {
            const int lane = threadIdx.x & 31;
            kd = warp_min(lane < (team.ts >> 5) ? team.keys[2 * lane + (gflip ? 1 : 0)] : ~0ull);
        } else if (gflip) {
            kd = ke;
        }
        seed = forced >= 0 ? forced : (int)(kd & 0xFFFFFFFFull);
        if (seed < 0 || seed >= n) {
            if (team.tr == 0) dev_fail(A.status, A.abort_flag, DEV_BAD_INDEX, where_err + 4, q, seed);
            return 0;
        }
    }
    P.subtick(PROF_ICM_SEED);
    bool absolute = false;   // energies set from scratch (large flipped sets)
    int swapped = 0;         // the flipped set was D\C (the chains hold each other's result)
    // a block team's union-find lists the sites it found outside the giant
    // component L in the free part of lst (S, at sbase); when the flipped set
    // lies in S it is taken from there: the sites of S whose final root is
    // (fast_eq) or is not (!fast_eq) fast_root
    bool fast = false, fast_eq = false;
    int fast_root = -1, ns = 0;
    int sbase = l0 == 0 ? llen : 0;
    if (cnt > 0) {
        int csize = 0;
        if (algo == ENGINE_ICM_BFS) {
            // breadth-first search from the seed; members of C get d = 2
            // (the visited bits make each site's claim unique)
            volatile int* vctl = team.ctl;
            if (team.tr == 0) {
                X.queue[0] = seed;
                X.vis[seed >> 5] |= 1u << (seed & 31);
                d[seed] = 2;
                vctl[TC_TAIL] = 1;
            }
            team.sync();
            const int lane = threadIdx.x & 31;
            int lo = 0;
            for (int level = 0; level <= n; level++) {
                const int hi = vctl[TC_TAIL];
                team.sync();
                if (lo == hi) break;
                for (int base = lo; base < hi; base += team.ts) {
                    const int idx = base + team.tr;
                    const bool have = idx < hi;
                    const int u = have ? X.queue[idx] : 0;
                    const int e0 = have ? brow[u] : 0;
                    const int deg = have ? brow[u + 1] - e0 : 0;
                    for (int k = 0; __any_sync(0xffffffffu, k < deg); k++) {
                        bool found = false;
                        int v = 0;
                        if (k < deg) {
                            v = (int)(badj[e0 + k] >> 8);
                            if (((volatile uint8_t*)d)[v] == 1) {
                                const uint32_t bit = 1u << (v & 31);
                                found = !(atomicOr(X.vis + (v >> 5), bit) & bit);
                            }
                        }
                        const unsigned m = __ballot_sync(0xffffffffu, found);
                        if (m) {
                            const int leader = __ffs(m) - 1;
                            int slot0 = 0;
                            if (lane == leader) slot0 = atomicAdd(team.ctl + TC_TAIL, __popc(m));
                            slot0 = __shfl_sync(0xffffffffu, slot0, leader);
                            if (found) {
                                X.queue[slot0 + __popc(m & ((1u << lane) - 1u))] = v;
                                d[v] = 2;
                            }
                        }
                    }
                }
                team.sync();
                lo = hi;
            }
            csize = lo;
            P.subtick(PROF_ICM_UNION);
        } else {
            // label the components of the whole overlap subgraph, then mark the
            // sites sharing the seed's label
            int* lab = X.queue;
            volatile int* vl = lab;
            bool ok = true;
            // (union-find parents were set with the overlap)
            if (algo != ENGINE_ICM_UNION_FIND) {
                for (int i = team.tr; i < n; i += team.ts) lab[i] = d[i] ? i : n;
                team.sync();
            }
            // (few neighbours: every edge is a link, nothing to sample)
            const bool direct = algo == ENGINE_ICM_UNION_FIND && D.all_edges != 0;
            if (direct) {
                // every edge from its upper end: each site is hooked under
                // its lowest overlap neighbour below it by a plain store,
                // then united with the others below it
                for_overlap([&](int u) {
                    int lo = u;
                    const int e1 = brow[u + 1];
#pragma unroll 4
                    for (int a = brow[u]; a < e1; a++) {
                        const int v = (int)(badj[a] >> 8);
                        if (v < lo && d[v]) lo = v;
                    }
                    if (lo < u) lab[u] = lo;
                });
                team.sync();
                P.subtick(PROF_UF_LINK0);
                for_overlap([&](int u) {
                    const int e1 = brow[u + 1];
                    int lo = u;
#pragma unroll 4
                    for (int a = brow[u]; a < e1; a++) {
                        const int v = (int)(badj[a] >> 8);
                        if (v < lo && d[v]) lo = v;
                    }
                    for (int a = brow[u]; a < e1; a++) {
                        const int v = (int)(badj[a] >> 8);
                        if (v < u && v != lo && d[v]) ok &= uf_unite(lab, u, v);
                    }
                });
                team.sync();
                P.subtick(PROF_UF_LINK1);
                if (BLOCK) {
                    // the cluster's size, and the flipped set from the list
                    const int rs = uf_find(vl, seed);
                    int c = 0;
                    for (int t = team.tr; t < llen; t += team.ts) c += uf_find(vl, lst[l0 + t]) == rs;
                    csize = team.count(c);
                    if (team.tr == 0) { team.ctl[TC_OVERLAP] = 0; team.ctl[TC_OTHERS] = 0; }
                    fast = true;
                    fast_root = rs;
                    fast_eq = exact || csize * 2 <= cnt;
                    sbase = l0;
                    ns = llen;
                    P.subtick(PROF_UF_SIZE);
                }
            } else if (algo == ENGINE_ICM_UNION_FIND) {
                // Afforest (Sutton, Ben-Nun, Barak, IPDPS 2018): in two
                // rounds, link every overlap site to its first two overlap
                // neighbours and compress the trees in between; take the most frequent
                // root of a sample as the large component L, then process the
                // full adjacency only of sites outside L.  An edge skipped at
                // an end in L is processed from its other end, unless that end
                // is in L too -- then both are already joined.
                // (GLINK: with the neighbour lists in device memory, a
                // thread scans four of its sites side by side, so that
                // their dependent loads overlap)
                const bool glink = GLINK && BLOCK && (space_large(SPACE) || !__isShared(badj)) &&
                                   (reinterpret_cast<uintptr_t>(badj) & 15u) == 0;
                // (a block team's round 0 keeps the link left for round 1, by
                // list position, in the free part of the list: S is listed
                // there only later)
                int* const link1 = (BLOCK && (LS || GLINK)) ? lst + sbase : nullptr;
                // u's first two overlap neighbours (-1: none): the list four
                // entries at a time, four independent loads, then four flags
                auto first_two = [&](int u, int& v0, int& v1) {
                    v0 = v1 = -1;
                    const int e1 = brow[u + 1];
                    for (int a = brow[u]; a < e1 && v1 < 0; a += 4) {
                        int v[4];
                        bool on[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) v[j] = a + j < e1 ? (int)(badj[a + j] >> 8) : u;
#pragma unroll
                        for (int j = 0; j < 4; j++) on[j] = a + j < e1 && d[v[j]];
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            if (on[j]) {
                                if (v0 < 0) v0 = v[j];
                                else if (v1 < 0) v1 = v[j];
                            }
                    }
                };
                // Round 0 hooks u under the lower of the two when that lies
                // below u: a plain store by u's own thread, no find and no
                // compare-and-swap (parents strictly decrease, so no cycle;
                // unions by find walked trees that nothing had compressed
                // yet).  Round 1 unites u with what the hook left, after the
                // compression.  (In round 1 of a team without kept targets
                // the hook's outcome is found again and not stored.)
                int round = 0;
                auto hook = [&](int u, int v0, int v1) {
                    const int lo = v1 >= 0 && v1 < v0 ? v1 : v0;
                    if (lo < 0) return -1;
                    if (lo > u) {
                        // (not hooked: the second neighbour may hang under u;
                        // whichever of two parents is stored, it is a link)
                        if (round == 0 && v1 >= 0) atomicMin(lab + v1, u);
                        return v0;
                    }
                    if (round == 0) lab[u] = lo;
                    return v1 < 0 ? -1 : (lo == v0 ? v1 : v0);
                };
                for (round = 0; round < 2; round++) {
                    if (round == 1 && link1 != nullptr) {
                        for (int t = team.tr; t < llen; t += 4 * team.ts) {
                            int u[4], tg[4];
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const int tk = t + k * team.ts;
                                u[k] = tk < llen ? lst[l0 + tk] : -1;
                                tg[k] = tk < llen ? link1[tk] : -1;
                            }
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                if (u[k] >= 0 && tg[k] >= 0) ok &= uf_unite(lab, u[k], tg[k]);
                        }
                    } else if (glink) {
                        // four list sites at a time, each with the two 16-byte
                        // pieces of its list that hold its first entries (five
                        // to eight of them: usually both targets).  The loads
                        // are scattered, so what they cost is one L1 lookup
                        // per lane and load: two pieces instead of eight
                        // entries
                        const uint4* const adj4 = reinterpret_cast<const uint4*>(badj);
                        for (int t = team.tr; t < llen; t += 4 * team.ts) {
                            int u[4], a[4], e[4];
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const int tk = t + k * team.ts;
                                u[k] = tk < llen ? lst[l0 + tk] : -1;
                            }
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                a[k] = u[k] >= 0 ? brow[u[k]] : 0;
                                e[k] = u[k] >= 0 ? brow[u[k] + 1] : 0;
                            }
                            int v0[4], v1[4];
#pragma unroll
                            for (int k = 0; k < 4; k++) v0[k] = v1[k] = -1;
                            // 16-byte pieces j and j + 1 of the sites whose
                            // links are not both found, all loads before their
                            // use
                            for (int j0 = 0;; j0 += 2) {
                                uint4 p[4][2];
                                bool more = false;
#pragma unroll
                                for (int k = 0; k < 4; k++)
#pragma unroll
                                    for (int j = 0; j < 2; j++)
                                        p[k][j] = v1[k] < 0 && 4 * ((a[k] >> 2) + j0 + j) < e[k] ? adj4[(a[k] >> 2) + j0 + j]
                                                                                                 : make_uint4(0, 0, 0, 0);
#pragma unroll
                                for (int k = 0; k < 4; k++) {
                                    const int b0 = (a[k] & ~3) + 4 * j0;
                                    const uint32_t w8[8] = {p[k][0].x, p[k][0].y, p[k][0].z, p[k][0].w,
                                                            p[k][1].x, p[k][1].y, p[k][1].z, p[k][1].w};
#pragma unroll
                                    for (int x = 0; x < 8; x++) {
                                        const int v = (int)(w8[x] >> 8);
                                        if (v1[k] < 0 && b0 + x >= a[k] && b0 + x < e[k] && d[v]) {
                                            if (v0[k] < 0) v0[k] = v;
                                            else v1[k] = v;
                                        }
                                    }
                                    more |= v1[k] < 0 && b0 + 8 < e[k];
                                }
                                if (!more) break;
                            }
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                if (u[k] < 0) continue;
                                const int rest = hook(u[k], v0[k], v1[k]);
                                if (link1 != nullptr) link1[t + k * team.ts] = rest;
                                else if (round == 1 && rest >= 0) ok &= uf_unite(lab, u[k], rest);
                            }
                        }
                    } else if (link1 != nullptr) {
                        // round 0 of a block team: the list four entries at a
                        // time
                        for (int t = team.tr; t < llen; t += team.ts) {
                            const int u = lst[l0 + t];
                            int v0, v1;
                            first_two(u, v0, v1);
                            link1[t] = hook(u, v0, v1);
                        }
                    } else
                    for_overlap([&](int u) {
                        int v0, v1;
                        first_two(u, v0, v1);
                        const int rest = hook(u, v0, v1);
                        if (round == 1 && rest >= 0) ok &= uf_unite(lab, u, rest);
                    });
                    team.sync();
                    P.subtick(round == 0 ? PROF_UF_LINK0 : PROF_UF_LINK1);
                    if (round == 0) {
                        // (after the last round the vote's and phase 3's
                        // finds halve the paths they walk)
                        if (glink) {
                            // four list entries loaded side by side
                            for (int t = team.tr; t < llen; t += 4 * team.ts) {
                                int u[4];
#pragma unroll
                                for (int k = 0; k < 4; k++) {
                                    const int tk = t + k * team.ts;
                                    u[k] = tk < llen ? lst[l0 + tk] : -1;
                                }
#pragma unroll
                                for (int k = 0; k < 4; k++) {
                                    if (u[k] < 0) continue;
                                    const int r = uf_find(vl, u[k]);
                                    if (r < 0) ok = false;
                                    else vl[u[k]] = r;
                                }
                            }
                        } else
                        for_overlap([&](int u) {
                            const int r = uf_find(vl, u);
                            if (r < 0) ok = false;
                            else vl[u] = r;
                        });
                        team.sync();
                        P.subtick(PROF_UF_COMPRESS);
                    }
                }
                int L = -1;
                if (BLOCK || team.tr < 32) {
                    // vote over 32 sampled overlap sites: a block team samples
                    // its overlap list, every warp the same 32 entries, so
                    // that each warp knows the winner without a barrier (the
                    // roots do not change until the next union); in a warp
                    // team each lane takes the first overlap site in a
                    // 32-byte window of the flags (eight independent word
                    // loads; the flags start on 16 bytes, bytes from n on are
                    // masked)
                    int cand = -1;
                    if (BLOCK) {
                        cand = uf_find(vl, lst[l0 + (int)(((long long)(threadIdx.x & 31) * llen) >> 5)]);
                    } else {
                        const int w0 = (int)(((long long)team.tr * n) >> 7);
                        uint32_t fw[8];
#pragma unroll
                        for (int j = 0; j < 8; j++)
                            fw[j] = 4 * (w0 + j) < n ? reinterpret_cast<const uint32_t*>(d)[w0 + j] : 0u;
                        for (int j = 0; j < 8 && cand < 0; j++)
                            for (int b = 0; b < 4; b++) {
                                const int i = 4 * (w0 + j) + b;
                                if (i < n && ((fw[j] >> (8 * b)) & 0xffu)) { cand = uf_find(vl, i); break; }
                            }
                    }
                    const unsigned grp = __match_any_sync(0xffffffffu, cand);
                    int votes = cand >= 0 ? __popc(grp) : 0, best = cand;
                    for (int o = 16; o > 0; o >>= 1) {
                        const int ov = __shfl_xor_sync(0xffffffffu, votes, o);
                        const int oc = __shfl_xor_sync(0xffffffffu, best, o);
                        if (ov > votes || (ov == votes && oc < best)) { votes = ov; best = oc; }
                    }
                    if (BLOCK) L = best;
                    else if (team.tr == 0) team.ctl[TC_BEST] = best;
                }
                if (!BLOCK) {
                    team.sync();
                    L = *(volatile int*)team.ctl;
                }
                P.subtick(PROF_UF_VOTE);
                for_overlap([&](int u) {
                    if (uf_find(vl, u) == L) return;
                    if (BLOCK) {
                        // S never outgrows the free part of lst: |S| <= llen <= n - llen
                        const int pos = atomicAdd(team.ctl + TC_S, 1);
                        if (pos < llen) lst[sbase + pos] = u;
                        return;
                    }
                    const int e1 = brow[u + 1];
#pragma unroll 4
                    for (int a = brow[u]; a < e1; a++) {
                        const int v = (int)(badj[a] >> 8);
                        if (d[v]) ok &= uf_unite(lab, u, v);
                    }
                });
                team.sync();
                P.subtick(PROF_UF_OUTSIDE);
                if (BLOCK) {
                    // the edges of S: one warp per site and one lane per
                    // neighbour (the unions of a site side by side) when
                    // that takes fewer rounds than one thread per site; a
                    // list far above the mean always by its warp (44 x 44
                    // lattice and eight sites with 64 neighbours: step 46.2
                    // -> 28.5 us)
                    const int ns0 = min(*(volatile int*)(team.ctl + TC_S), llen);
                    const int nw = team.ts >> 5, lane = team.tr & 31;
                    const int mean = (D.nnz + n - 1) / n, long_list = max(16, 3 * mean);
                    const bool by_warp = (ns0 + nw - 1) / nw < mean;
                    const int t0 = by_warp ? team.tr >> 5 : team.tr, dt = by_warp ? nw : team.ts;
                    for (int t = t0; t - (by_warp ? 0 : lane) < ns0; t += dt) {
                        int u = 0, a = 0, e1 = 0;
                        if (t < ns0) {
                            u = lst[sbase + t];
                            a = brow[u];
                            e1 = brow[u + 1];
                        }
                        // a thread's own list, then the warp's long ones
                        unsigned wide = by_warp ? 1u : __ballot_sync(0xffffffffu, e1 - a > long_list);
                        int x = u, b = e1 - a > long_list ? e1 : a, be = e1, db = 1;
                        for (bool own = !by_warp; own || wide; own = false) {
                            if (!own) {
                                const int src = __ffs(wide) - 1;
                                x = __shfl_sync(0xffffffffu, u, src);
                                b = __shfl_sync(0xffffffffu, a, src) + lane;
                                be = __shfl_sync(0xffffffffu, e1, src);
                                db = 32;
                                wide &= wide - 1;
                            }
                            for (; b < be; b += db) {
                                const int v = (int)(badj[b] >> 8);
                                if (d[v]) ok &= uf_unite(lab, x, v);
                            }
                        }
                    }
                    team.sync();
                    P.subtick(PROF_UF_SUNION);
                }
                if (BLOCK) {
                    // sites in L's component at their phase-3 check stay in it:
                    // every site outside the final component of L is in S
                    ns = min(*(volatile int*)(team.ctl + TC_S), llen);
                    const int rL = uf_find(vl, L), rs = uf_find(vl, seed);
                    int c = 0;   // |S \ comp(L)| when the seed is in comp(L), else |C|
                    for (int t = team.tr; t < ns; t += team.ts) {
                        const int r = uf_find(vl, lst[sbase + t]);
                        c += (rs == rL) ? (r != rL) : (r == rs);
                    }
                    c = team.count(c);
                    // every thread has read the list counters: reset them
                    // for the next pair (a barrier of this pair's flip or
                    // energy reduction comes before its next use)
                    if (team.tr == 0) { team.ctl[TC_OVERLAP] = 0; team.ctl[TC_OTHERS] = 0; team.ctl[TC_S] = 0; }
                    csize = (rs == rL) ? cnt - c : c;
                    const bool sw = !exact && csize * 2 > cnt;
                    fast = (rs == rL) ? sw : !sw;   // the flipped set lies in S
                    fast_root = rs == rL ? rL : rs;
                    fast_eq = rs != rL;
                    P.subtick(PROF_UF_SIZE);
                }
            } else {
                // minimum-label propagation with root hooking and pointer jumping
                // (Shiloach-Vishkin style); labels only decrease and always name
                // a site of the same component
                bool conv = false;
                for (int round = 0; round < 512 && !conv; round++) {
                    int changed = 0;
                    for (int u = team.tr; u < n; u += team.ts) {
                        if (!d[u]) continue;
                        const int lu = vl[u];
                        int best = lu;
                        const int e1 = brow[u + 1];
#pragma unroll 4
                        for (int a = brow[u]; a < e1; a++) {
                            const int v = (int)(badj[a] >> 8);
                            const int lv = vl[v];
                            if (d[v]) best = min(best, lv);
                        }
                        if (best < lu) {
                            atomicMin(lab + lu, best);
                            atomicMin(lab + u, best);
                            changed = 1;
                        }
                    }
                    conv = !(BLOCK ? (__syncthreads_or(changed) != 0) : (__any_sync(0xffffffffu, changed) != 0));
                    if (!BLOCK) __syncwarp();
                    for (int u = team.tr; u < n; u += team.ts) {
                        if (!d[u]) continue;
                        int l = vl[u];
                        for (int g = 0; g < n; g++) {
                            const int ll = vl[l];
                            if (ll >= l) break;
                            l = ll;
                        }
                        vl[u] = l;
                    }
                    team.sync();
                }
                ok = conv;
            }
            if (!ok) dev_fail(A.status, A.abort_flag, DEV_UF_LIMIT, where_err + 3, q, algo);
            P.subtick(PROF_ICM_UNION);
            const int root = (algo == ENGINE_ICM_UNION_FIND) ? uf_find(vl, seed) : vl[seed];
            if (BLOCK && algo == ENGINE_ICM_UNION_FIND) {
                // csize is known.  When the flipped set is not in S it is the
                // rest of the overlap: mark the selected part of S (d = 3),
                // and the flipped set is every overlap site not marked
                if (!fast) {
                    for (int t = team.tr; t < ns; t += team.ts) {
                        const int u = lst[sbase + t];
                        if ((uf_find(vl, u) == fast_root) == fast_eq) d[u] = 3;
                    }
                    team.sync();
                }
            } else {
                // mark the cluster C (d = 2) and count it
                for_overlap([&](int u) {
                    const int lu = (algo == ENGINE_ICM_UNION_FIND) ? uf_find(vl, u) : vl[u];
                    if (lu != root) return;
                    d[u] = 2;
                    csize++;
                });
                csize = team.count(csize);
            }
        }
        // (A, B) -> (A flipped on C, B flipped on C) is the same pair of
        // states as (B flipped on D\C, A flipped on D\C): flip the smaller of
        // C and D\C.  With D\C the pair's two chains hold each other's
        // result at this temperature -- the ICM move followed by an exchange
        // of the two chains' configurations at one temperature, which leaves
        // the joint distribution of the (independent, identical) chains
        // invariant.  Replay keeps the reference's flips.
        swapped = (!exact && csize * 2 > cnt) ? 1 : 0;
        const uint8_t fmark = swapped ? 1 : 2;
        const int fsize = swapped ? cnt - csize : csize;
        // membership of an overlap site in the flipped set
        const bool rest = BLOCK && algo == ENGINE_ICM_UNION_FIND && !fast;
        auto in_flip = [&](int u) { return rest ? d[u] != 3 : d[u] == fmark; };
        // one pass over a flipped site: flip it and push its field change to
        // its neighbours; the energy changes by the edges leaving the flipped
        // set F.  F is a union of overlap components, so a neighbour outside
        // F is outside the overlap (equal in A and B) and keeps its spin.
        // (by_warp: the lanes of a warp share the site, read its spins
        // before lane 0 flips them and take every 32nd edge)
        auto flip_push = [&](int u, bool by_warp) {
            const int hu = has_h ? bh[u] : 0;
            const int lane = by_warp ? (threadIdx.x & 31) : 0;
            int sa = 0, sb = 0;   // spins before the flip
            if (locA) sa = sA[u];
            if (locB) sb = sB[u];
            if (share) {
                sb = pub_site(pubB, u);
                sa = -sb;   // (u is in the overlap)
            }
            if (by_warp) __syncwarp();
            if (lane == 0) {
                if (locA) sA[u] = (int8_t)-sa;
                if (locB) sB[u] = (int8_t)-sb;
                if (share) atomicOr(X.vis + (u >> 5), 1u << (u & 31));
                if (locA || share) dEa -= 2 * sa * hu;
                if (locB || share) dEb -= 2 * sb * hu;
            }
            const int e1 = brow[u + 1], da = by_warp ? 32 : 1;
#pragma unroll 4
            for (int a = brow[u] + lane; a < e1; a += da) {
                const uint32_t e = badj[a];
                const int v = (int)(e >> 8);
                const int J = (int)(int8_t)(e & 0xffu);
                if (fA) atomicAdd(fA + v, J * (-2 * sa));
                if (fB) atomicAdd(fB + v, J * (-2 * sb));
                if (!d[v]) {
                    const int sv = share ? pub_site(pubB, v) : (locA ? sA[v] : sB[v]);
                    if (locA || share) dEa -= 2 * J * sa * sv;
                    if (locB || share) dEb -= 2 * J * sb * sv;
                }
            }
        };
        if (fast) {
            // one warp per site when that takes fewer rounds (as for the
            // unions of S); the membership test is the same in every lane
            const int nw = team.ts >> 5;
            const bool by_warp = BLOCK && (ns + nw - 1) / nw < (D.nnz + n - 1) / n;
            const int t0 = by_warp ? team.tr >> 5 : team.tr, dt = by_warp ? nw : team.ts;
            for (int t = t0; t < ns; t += dt) {
                const int u = lst[sbase + t];
                if ((uf_find((volatile int*)X.queue, u) == fast_root) == fast_eq) flip_push(u, by_warp);
            }
        } else if (BLOCK && !share && (long long)fsize * 4 > (long long)n) {
            // a large cluster: flip, then fields and energies from scratch
            // (gathers, no atomics; the cost does not grow with the cluster)
            for_overlap([&](int u) {
                if (!in_flip(u)) return;
                if (locA) sA[u] = (int8_t)-sA[u];
                if (locB) sB[u] = (int8_t)-sB[u];
            });
            team.sync();
            long long eA = 0, eB = 0;
            for (int i = team.tr; i < n; i += team.ts) {
                int fa = 0, fb = 0;
                const int e1 = brow[i + 1];
#pragma unroll 4
                for (int a = brow[i]; a < e1; a++) {
                    const uint32_t e = badj[a];
                    const int v = (int)(e >> 8);
                    const int J = (int)(int8_t)(e & 0xffu);
                    if (locA) fa += J * sA[v];
                    if (locB) fb += J * sB[v];
                }
                const int h2 = has_h ? 2 * bh[i] : 0;
                if (locA) { if (fA) fA[i] = fa; eA += (long long)sA[i] * (h2 + fa); }
                if (locB) { if (fB) fB[i] = fb; eB += (long long)sB[i] * (h2 + fb); }
            }
            team.sum_energies(eA, eB, A.small_energy != 0);
            if (team.tr == 0) {
                if (locA) B.E[rA] = eA / 2;
                if (locB) B.E[rB] = eB / 2;
            }
            absolute = true;
        } else {
            // a small flipped set, flipped and pushed in one pass
            for_overlap([&](int u) {
                if (in_flip(u)) flip_push(u, false);
            });
        }
        if (!BLOCK || absolute) team.sync();   // (a block team's energy sums have the barrier)
    }
    if (!absolute && (gflip || cnt > 0)) {
        team.sum_energies(dEa, dEb, A.small_energy != 0);
        if (team.tr == 0) {
            if (locA) B.E[rA] += dEa;
            if (locB && cnt > 0) B.E[rB] += dEb;
        }
    }
    if (share) {
        // the sites to flip in A and in B and both energies, each word with
        // the step's tag
        for (int w = team.tr; w < nwords; w += team.ts) {
            const uint32_t f = X.vis[w];
            st_relaxed_gpu_u64(result + w, ((unsigned long long)tag << 32) | (gflip ? ~f : f));
            st_relaxed_gpu_u64(result + nwords + w, ((unsigned long long)tag << 32) | f);
        }
        if (team.tr == 0) {
            st_relaxed_gpu_u64(result + 2 * nwords, pub_word(tag, B.E[rA] + dEa));
            st_relaxed_gpu_u64(result + 2 * nwords + 1, pub_word(tag, B.E[rB] + dEb));
        }
        team.sync();   // (the next pair clears the bits)
    }
    if (!(BLOCK && algo == ENGINE_ICM_UNION_FIND && cnt > 0)) {
        // (a block team's union-find reset the list counters after its size
        // reduction and passed a barrier since)
        if (BLOCK && team.tr == 0) {
            team.ctl[TC_OVERLAP] = 0;   // the list counters, for the next pair
            team.ctl[TC_OTHERS] = 0;
            team.ctl[TC_S] = 0;
        }
        team.sync();
    }
    P.subtick(PROF_ICM_FLIP);
    if (P.on && cnt > 0) P.s->c[PROF_ICM_COUNT]++;
    return swapped;
}

// Local field of site i gathered from the neighbours' spins (field_gather
// mode, where fields are not stored): f_i = sum_j J_ij s_j.
template <class Spins>
__device__ __forceinline__ int gather_field(const int32_t* row, const uint32_t* adj, Spins sp, int i) {
    int f = 0;
    for_each_neighbour(row, adj, i, [&](uint32_t e) { f += (int)(int8_t)(e & 0xffu) * sp[e >> 8]; });
    return f;
}

// The part of site i's local field that thread `sub` of G gathers: the 16-byte
// pieces sub, sub + G, ... of its neighbour list, two at a time, entries
// outside the list as zeros.  All loads of a pair of pieces are independent;
// a list walked entry by entry up to alignment and from there takes twice as
// long as its twenty neighbours' loads (N=2000: 0.93 us a colour class).
// (The list starts on 16 bytes and is readable to the end of its last piece.)
__device__ __forceinline__ int gather_pieces(const int32_t* row, const uint32_t* adj, const int8_t* sp, int i, int sub,
                                             int G) {
    const int e0 = row[i], deg = row[i + 1] - e0, p1 = (e0 + deg + 3) >> 2;
    const uint4* const adj4 = reinterpret_cast<const uint4*>(adj);
    int f = 0;
    for (int p = (e0 >> 2) + sub; p < p1; p += 2 * G) {
        const uint4 u = adj4[p];
        uint4 v = make_uint4(0, 0, 0, 0);
        if (p + G < p1) v = adj4[p + G];
        uint32_t e[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
        int s[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int at = 4 * (k < 4 ? p : p + G) + (k & 3);
            if ((unsigned)(at - e0) >= (unsigned)deg) e[k] = 0;
            s[k] = sp[e[k] >> 8];
        }
#pragma unroll
        for (int k = 0; k < 8; k++) f += (int)(int8_t)(e[k] & 0xffu) * s[k];
    }
    return f;
}

// Takes over what the group's blocks worked out for the pairs of this block's
// replicas: tagged words of the sites to flip and the new energies, eight
// sites per thread and replica, four replicas' words loaded together.  (Every
// block has published its results or is working on them: no block waits
// before its own pairs are out.)  False in a warp whose wait ran out: replicas
// may then be flipped in part, and no sweep may follow.
template <int SPACE>
__device__ __forceinline__ bool apply_pairs(const EngineArgs& A, const BlockCtx& B, int chains_even, uint32_t tag,
                                            volatile int* abortf) {
    const InstanceDesc& D = B.D;
    const int tid = threadIdx.x, T = blockDim.x, n = D.n, nt = D.nt, W = (n + 31) >> 5;
    const unsigned long long limit = A.wait_limit_ns ? A.wait_limit_ns : kWaitLimitNs;
    // replica j's result and whether it is the pair's second (null: no pair)
    auto result_of = [&](int j, bool& second) -> const unsigned long long* {
        if (j >= D.rpc) return nullptr;
        const int sl = (int)B.rslot[j], c = sl / nt, kk = nt - 1 - (sl - c * nt);
        second = c & 1;
        return kk < D.nc && c < chains_even ? A.icm_pub + (long long)((c >> 1) * D.nc + kk) * A.icm_pub_stride : nullptr;
    };
    for (int j0 = 0; j0 < D.rpc; j0 += 4) {
        const unsigned long long* from[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
            bool second = false;
            from[x] = result_of(j0 + x, second);
            if (from[x] != nullptr) {
                if (tid < 32) {
                    unsigned long long w = 0;
                    if (!poll_tagged(from[x] + 2 * W + second, tid == 0, tag, w, abortf, A.status, limit, 6)) return false;
                    if (tid == 0) B.E[B.r0 + j0 + x] = (long long)(int32_t)(uint32_t)w;
                }
                if (second) from[x] += W;
            }
        }
        for (int u0 = tid & ~31; u0 < 4 * W; u0 += T) {
            const int u = u0 + (tid & 31);
            unsigned long long w[4] = {0, 0, 0, 0};
#pragma unroll
            for (int x = 0; x < 4; x++)
                if (from[x] != nullptr && u < 4 * W) w[x] = ld_relaxed_gpu_u64(from[x] + (u >> 2));
#pragma unroll
            for (int x = 0; x < 4; x++) {
                if (from[x] == nullptr) continue;
                const bool late = u < 4 * W && (uint32_t)(w[x] >> 32) != tag;
                if (__any_sync(0xffffffffu, late) &&
                    !poll_tagged(from[x] + (late ? u >> 2 : 0), late, tag, w[x], abortf, A.status, limit, 6))
                    return false;
                const SpinRow<SPACE> sp = spin_row<SPACE>(B, j0 + x);
                for (uint32_t m = ((uint32_t)w[x] >> (8 * (u & 3))) & 0xffu; m != 0 && u < 4 * W; m &= m - 1) {
                    const int i = 8 * u + __ffs((int)m) - 1;
                    if (i < n) sp[i] = (int8_t)-sp[i];
                }
            }
        }
    }
    return true;
}

// The local fields of four interleaved replicas at one site per lane (its list
// of my_deg entries from my0; 0 entries: none).  Four neighbouring lanes gather one another's sites in turn, each
// a quarter of the list's 16-byte pieces, so that a group's loads are whole
// sectors of one list; one 32-bit load brings a neighbour's spin in all four
// replicas.  What bounds it is that load's bank conflicts and the lists' way
// from L2: 176 us a sweep of N=20000, degree 40, 4 replicas on each of 128
// SMs.  (One thread per site and a byte load per replica, four times the
// shared wavefronts and an L1 lookup per lane and piece: 413 us; pieces loaded
// two at a time when they are needed: 52 us more; at the start of each 32
// sites only: 13 us more.)
// PACKED (no field beyond +-127): with the four spins as signed digits of a
// 32-bit number, base 256, one multiply-add sums all four fields, modulo 2^32;
// the digits are taken apart at the end.
// The first kAhead pieces of the four sites are in registers already; as each
// site is done, those of the site that the warp visits next take their place,
// across the colour classes (lists don't change): L2 answers behind the sums.
constexpr int kAhead = 3;
// (of the site of the s-th lane in each group of four)
__device__ __forceinline__ void load_ahead(const uint32_t* adj, int s, int my0, int my_deg, uint4 (&ahead)[kAhead]) {
    const int lane = threadIdx.x & 31, src = (lane & ~3) + s;
    const uint4* const adj4 = reinterpret_cast<const uint4*>(adj);
    const int e0 = __shfl_sync(0xffffffffu, my0, src), deg = __shfl_sync(0xffffffffu, my_deg, src);
    const int p0 = (e0 >> 2) + (lane & 3), p1 = (e0 + deg + 3) >> 2;
#pragma unroll
    for (int x = 0; x < kAhead; x++) ahead[x] = p0 + 4 * x < p1 ? adj4[p0 + 4 * x] : make_uint4(0, 0, 0, 0);
}
template <bool PACKED>
__device__ __forceinline__ void gather4(const uint32_t* adj, const uint32_t* s4, int my0, int my_deg, int next0,
                                        int next_deg, uint4 (&ahead)[4][kAhead], int (&f)[4]) {
    const int lane = threadIdx.x & 31, sub = lane & 3;
    const uint4* const adj4 = reinterpret_cast<const uint4*>(adj);
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const int src = (lane & ~3) + s;
        const int e0 = __shfl_sync(0xffffffffu, my0, src), deg = __shfl_sync(0xffffffffu, my_deg, src);
        const int p0 = (e0 >> 2) + sub, p1 = (e0 + deg + 3) >> 2;
        int acc = 0, g[4] = {0, 0, 0, 0};
        auto piece = [&](const uint4& q, int p) {
            uint32_t e[4] = {q.x, q.y, q.z, q.w}, r[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if ((unsigned)(4 * p + k - e0) >= (unsigned)deg) e[k] = 0;
                r[k] = s4[e[k] >> 8];
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int w = (int)(int8_t)(e[k] & 0xffu);
                if (PACKED) {
                    // bytes to digits: a negative digit borrows from the next
                    acc += w * (int)(r[k] - ((r[k] & 0x00808080u) << 1));
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++) g[j] += w * (int)(int8_t)(r[k] >> (8 * j));
                }
            }
        };
#pragma unroll
        for (int x = 0; x < kAhead; x++) piece(ahead[s][x], p0 + 4 * x);
        load_ahead(adj, s, next0, next_deg, ahead[s]);
#pragma unroll 1
        for (int p = p0 + 4 * kAhead; p < p1; p += 4) piece(adj4[p], p);
        if (PACKED) {
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            if (sub == s) f[0] = acc;
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                g[j] += __shfl_xor_sync(0xffffffffu, g[j], 1);
                g[j] += __shfl_xor_sync(0xffffffffu, g[j], 2);
                if (sub == s) f[j] = g[j];
            }
        }
    }
    if (PACKED) {
        int acc = f[0];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            f[j] = (int)(int8_t)(acc & 0xff);
            acc = (acc - f[j]) >> 8;
        }
    }
}

// --------------------------------------------------------------- sweeps
// A warp pushes the field changes of at most this many accepted sites one
// site at a time (a lane per neighbour); with more, each lane pushes its own
// (on C2, 4 to 8 measured best: 26.5 us per PT step against 27.6 with every
// lane pushing its own).
constexpr int kCoopPushSites = 4;
// With fields gathered and several replicas in a block, a thread visits one
// site of each of at most this many replicas per neighbour-list read.
constexpr int kGatherReps = 4;

// Colour-class Metropolis sweep of the block's replicas (production).
// dE_i = -2 s_i (h_i + f_i); accepted with probability min(1, exp(-beta dE))
// (src/replica.cc:31-38); an accepted flip pushes J_ij * (-2 s_i) into each
// neighbour's field (the integer form of src/problem.cc:164-181), or, where no
// fields are stored, every visit gathers its own.  With one replica per block
// (ONE) every thread keeps its energy change and flip count in registers until
// a phase boundary; with several, warps aggregate per replica before touching
// shared memory.  COOP: the narrow block team, whose instances with few
// neighbours gather (InstanceDesc::lanes), and whose others push together.
template <bool ONE, bool COOP, int SPACE>
__device__ void colored_sweep(const EngineArgs& A, const BlockCtx& B, unsigned long long sweep_idx,
                              int32_t* s_col, const uint32_t* s_thr, int* s_dEp, unsigned* s_flp,
                              unsigned long long* s_flips, long long* s_bestE, int* s_improved,
                              int* s_misc, bool best_per_phase) {
    const InstanceDesc& D = B.D;
    const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31;
    const int npad = D.n_pad, rpc = ONE ? 1 : D.rpc;
    const int32_t* row = B.row;
    const uint32_t* adj = B.adj;
    const int kmax = D.kmax;
    ThreadRng12 rng;
    // counter: (rank in the group, thread), sweep, instance id in the high
    // half of the call word (a thread makes far fewer than 2^16 calls)
    const int G = ONE && COOP ? D.lanes : 0, ng = G > 0 ? T / G : T, grp = G > 0 ? tid / G : tid,
              sub = G > 0 ? tid & (G - 1) : 0;
    rng.start(stream_key(A.seed, STREAM_SWEEP), (uint32_t)(B.rank * T + grp + sub * ng), sweep_idx,
              (uint32_t)D.inst_id << 16);
    int acc_de = 0;
    unsigned acc_fl = 0;
    // several replicas in the block, fields gathered
    const bool gm = !ONE && B.field == nullptr && rpc <= kGatherReps;
    int8_t* const sp1 = B.spin;
    int32_t* const fd1 = B.field;
    const int32_t* const h1 = B.h;
    const uint32_t* const thr1 = ONE ? s_thr + B.tb[0] : s_thr;
    const int ncolors = D.ncolors;
    // interleaved replicas: the warp's 32 sites now and next (their class,
    // first site and lists), and list pieces loaded ahead
    struct Sites { int c, base, e0, deg; } at{}, next{};
    uint4 ahead[4][kAhead];
    auto advance = [&](Sites& x) {
        x.base += T;
        while (x.c < ncolors && x.base >= s_col[x.c + 1]) {
            if (++x.c < ncolors) x.base = s_col[x.c] + (tid & ~31);
        }
        const int i = x.base + lane;
        x.e0 = x.deg = 0;
        if (x.c < ncolors && i < s_col[x.c + 1]) {
            x.e0 = row[i];
            x.deg = row[i + 1] - x.e0;
        }
    };
    ThreadRngWindow rng4;
    if (SPACE == SP_LARGE4 || (!ONE && !gm))
        rng4.start(stream_key(A.seed, STREAM_SWEEP), (uint32_t)(B.rank * T + tid), sweep_idx, (uint32_t)D.inst_id << 16);
    if (SPACE == SP_LARGE4) {
        at.base = s_col[0] + (tid & ~31) - T;
        advance(at);
        next = at;
        advance(next);
#pragma unroll
        for (int s = 0; s < 4; s++) load_ahead(adj, s, at.e0, at.deg, ahead[s]);
    }
    for (int c = 0; c < ncolors; c++) {
        const int c0 = s_col[c];
        const int Sc = s_col[c + 1] - c0;
        if (ONE && COOP && fd1 != nullptr) {
            // each thread decides its own site (the same site and random
            // draws as one site per thread).  A warp with few accepted sites
            // (the cold replicas) pushes their field changes one site at a
            // time with a lane per neighbour, so that no lane walks a long
            // neighbour list alone; a warp with many (the hot replicas)
            // lets every lane push its own site's changes, side by side
            int8_t* const sp = sp1;
            int32_t* const fd = fd1;
            const uint32_t* const thr_row = thr1;
            for (int base = c0 + (tid & ~31); base < c0 + Sc; base += T) {
                const int i = base + lane;
                bool acc = false;
                int s = 0, e0 = 0, e1 = 0;
                if (i < c0 + Sc) {
                    s = sp[i];
                    const int f = fd[i] + (h1 != nullptr ? h1[i] : 0);
                    const int de = -2 * s * f;
                    acc = de <= 0;
                    if (!acc) {
                        const uint32_t thr = thr_row[min(de >> 1, kmax)];
                        acc = (rng.next_one() < thr) || (thr == 0xFFFFFFFFu);
                    }
                    if (acc) {
                        sp[i] = (int8_t)-s;
                        acc_de += de;
                        acc_fl++;
                        e0 = row[i];
                        e1 = row[i + 1];
                    }
                }
                unsigned m = __ballot_sync(0xffffffffu, acc);
                if (__popc(m) > kCoopPushSites) {
                    if (acc) {
                        const int dl = -2 * s;
                        for_each_neighbour(row, adj, i,
                                           [&](uint32_t e) { atomicAdd(fd + (e >> 8), (int)(int8_t)(e & 0xffu) * dl); });
                    }
                    m = 0;
                }
                while (m) {
                    const int src = __ffs(m) - 1;
                    m &= m - 1;
                    const int a0 = __shfl_sync(0xffffffffu, e0, src), a1 = __shfl_sync(0xffffffffu, e1, src);
                    const int dl = -2 * __shfl_sync(0xffffffffu, s, src);
                    for (int a = a0 + lane; a < a1; a += 32) {
                        const uint32_t e = adj[a];
                        atomicAdd(fd + (e >> 8), (int)(int8_t)(e & 0xffu) * dl);
                    }
                }
            }
        } else if (ONE && COOP && G > 0) {
            // A site's field is gathered by G neighbouring threads (no stored
            // fields: nothing to push, so hot and cold replicas cost alike).
            // Every thread keeps the random stream of one of the T logical
            // threads that the sites of a class are dealt to: thread g G + s
            // that of logical thread g + s T / G, so that a class of at most
            // T / G sites uses all threads, and a larger one takes its
            // T / G-site portions in turn.
            for (int j0 = 0; j0 < Sc; j0 += T)
                for (int s = 0; s < G; s++) {
                    const int portion = j0 + s * ng;
                    if (portion >= Sc) break;
                    const int j = portion + grp, i = c0 + j;
                    const bool have = j < Sc, mine = have && sub == s;
                    if (mine) rng.fill_one();   // (runs under the gather's loads)
                    int f = 0;
                    if (have) f = gather_pieces(row, adj, sp1, i, sub, G);
                    for (int o = G >> 1; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
                    if (mine) {
                        const int sv = sp1[i];
                        const int de = -2 * sv * (f + (h1 != nullptr ? h1[i] : 0));
                        bool acc = de <= 0;
                        if (!acc) {
                            const uint32_t thr = thr1[min(de >> 1, kmax)];
                            acc = (rng.next_one() < thr) || (thr == 0xFFFFFFFFu);
                        }
                        if (acc) {
                            sp1[i] = (int8_t)-sv;
                            acc_de += de;
                            acc_fl++;
                        }
                    }
                }
        } else if (ONE) {
            int8_t* sp = B.spin;
            int32_t* fd = B.field;   // null in field_gather mode
            const uint32_t* thr_row = s_thr + B.tb[0];
            for (int i = c0 + tid; i < c0 + Sc; i += T) {
                const int s = sp[i];
                const int f = (fd ? fd[i] : gather_field(row, adj, sp, i)) + (B.h ? B.h[i] : 0);
                const int de = -2 * s * f;
                bool acc = de <= 0;
                if (!acc) {
                    const uint32_t thr = thr_row[min(de >> 1, kmax)];
                    acc = (rng.next() < thr) || (thr == 0xFFFFFFFFu);
                }
                if (acc) {
                    sp[i] = (int8_t)-s;
                    acc_de += de;
                    acc_fl++;
                    if (fd) {
                        const int dl = -2 * s;
                        for_each_neighbour(row, adj, i,
                                           [&](uint32_t e) { atomicAdd(fd + (e >> 8), (int)(int8_t)(e & 0xffu) * dl); });
                    }
                }
            }
        } else if (SPACE == SP_LARGE4) {
            // (the four replicas' energy changes and flips: one addition per
            // warp, replica and class)
            int g_de[4] = {0, 0, 0, 0};
            unsigned g_fl[4] = {0, 0, 0, 0};
            uint32_t* const s4 = reinterpret_cast<uint32_t*>(B.spin);
            for (int base = c0 + (tid & ~31); base < c0 + Sc; base += T) {
                const int i = base + lane;
                int f[4];
                const int e0 = at.e0, deg = at.deg;
                at = next;
                advance(next);
                if (kmax <= 127) gather4<true>(adj, s4, e0, deg, at.e0, at.deg, ahead, f);
                else gather4<false>(adj, s4, e0, deg, at.e0, at.deg, ahead, f);
                const bool have = i < c0 + Sc;
                const int hi = have && B.h ? B.h[i] : 0;
                const uint32_t w0 = have ? s4[i] : 0u;
                uint32_t w = w0;
                // the four thresholds side by side, then the decisions in
                // replica order, without a branch (branches and a refill of
                // twelve words wherever a lane ran out: 245 us a sweep)
                int de[4];
                uint32_t thr[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    de[j] = have ? -2 * (int)(int8_t)(w0 >> (8 * j)) * (f[j] + hi) : 0;
                    thr[j] = s_thr[B.tb[j] + min(max(de[j], 0) >> 1, kmax)];
                }
                uint32_t u[4];
                rng4.peek(u);
                uint32_t drawn = 0;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const bool up = de[j] > 0;
                    const bool acc = have && (!up || u[0] < thr[j] || thr[j] == 0xFFFFFFFFu);
                    if (up) {
                        u[0] = u[1];
                        u[1] = u[2];
                        u[2] = u[3];
                        drawn++;
                    }
                    if (acc) {
                        w ^= 0xFEu << (8 * j);   // 0x01 <-> 0xFF
                        g_de[j] += de[j];
                        g_fl[j]++;
                    }
                }
                rng4.take(drawn);
                if (w != w0) s4[i] = w;
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int v = (int)__reduce_add_sync(0xffffffffu, (unsigned)g_de[j]);
                const unsigned f = __reduce_add_sync(0xffffffffu, g_fl[j]);
                if (lane == 0 && f != 0) {
                    atomicAdd(s_dEp + j, v);
                    atomicAdd(s_flp + j, f);
                }
            }
        } else if (gm) {
            // a thread visits site i of each of the block's replicas: the
            // neighbour list is read once for all of them (sites of one
            // colour class share no edge, so the gathered spins are settled)
            int g_de[kGatherReps];
            unsigned g_fl[kGatherReps];
#pragma unroll
            for (int j = 0; j < kGatherReps; j++) {
                g_de[j] = 0;
                g_fl[j] = 0;
            }
            for (int i = c0 + tid; i < c0 + Sc; i += T) {
                int f[kGatherReps];
#pragma unroll
                for (int j = 0; j < kGatherReps; j++) f[j] = 0;
                // the neighbour list 16 bytes at a time, one load in flight
                // (four spin loads per entry keep the thread busy)
                auto scan = [&](auto&& visit) {
                    int a = row[i];
                    const int a1 = row[i + 1];
                    if ((reinterpret_cast<uintptr_t>(adj) & 15u) == 0) {
                        for (; a < a1 && (a & 3); a++) visit(adj[a]);
#pragma unroll 1
                        for (; a + 4 <= a1; a += 4) {
                            const uint4 q = *reinterpret_cast<const uint4*>(adj + a);
                            visit(q.x);
                            visit(q.y);
                            visit(q.z);
                            visit(q.w);
                        }
                    }
                    for (; a < a1; a++) visit(adj[a]);
                };
                scan([&](uint32_t e) {
                    const int w = (int)(int8_t)(e & 0xffu);
                    const int8_t* sn = B.spin + (e >> 8);
#pragma unroll
                    for (int j = 0; j < kGatherReps; j++)
                        if (j < rpc) f[j] += w * sn[j * npad];
                });
                const int hi = B.h ? B.h[i] : 0;
#pragma unroll
                for (int j = 0; j < kGatherReps; j++) {
                    if (j < rpc) {
                        int8_t* sp = B.spin + j * npad;
                        const int s = sp[i];
                        const int de = -2 * s * (f[j] + hi);
                        bool acc = de <= 0;
                        if (!acc) {
                            const uint32_t thr = s_thr[B.tb[j] + min(de >> 1, kmax)];
                            acc = (rng.next() < thr) || (thr == 0xFFFFFFFFu);
                        }
                        if (acc) {
                            sp[i] = (int8_t)-s;
                            g_de[j] += de;
                            g_fl[j]++;
                        }
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < kGatherReps; j++) {
                if (j < rpc) {
                    int v = g_de[j];
                    unsigned f = g_fl[j];
                    for (int o = 16; o > 0; o >>= 1) {
                        v += __shfl_xor_sync(0xffffffffu, v, o);
                        f += __shfl_xor_sync(0xffffffffu, f, o);
                    }
                    if (lane == 0 && (v != 0 || f != 0)) {
                        atomicAdd(s_dEp + j, v);
                        atomicAdd(s_flp + j, f);
                    }
                }
            }
        } else {
            const int items = rpc * Sc;
            const int items_w = (items + 31) & ~31;   // whole warps iterate together
            // (item it: replica jt, site ct of the class; two divisions a
            // class instead of one an item)
            const int Sd = max(Sc, 1), jd = T / Sd, cd = T - jd * Sd;
            int jt = tid / Sd, ct = tid - jt * Sd;
            // four items of a thread at a time (sites of one class share no
            // edge, so none sees another's flip): their loads overlap, and
            // their draws take at most one Philox block
            for (int it = tid; it < items_w; it += 4 * T) {
                int jx[4], ix[4], sx[4], de[4];
                uint32_t thr[4];
#pragma unroll
                for (int x = 0; x < 4; x++) {
                    const bool have = it + x * T < items;
                    jx[x] = have ? jt : 0;
                    ix[x] = c0 + (have ? ct : 0);
                    const int8_t* sp = B.spin + jx[x] * npad;
                    sx[x] = have ? sp[ix[x]] : 0;
                    const int f = (B.field ? B.field[jx[x] * npad + ix[x]] : have ? gather_field(row, adj, sp, ix[x]) : 0) +
                                  (B.h ? B.h[ix[x]] : 0);
                    de[x] = -2 * sx[x] * f;
                    jt += jd;
                    ct += cd;
                    if (ct >= Sd) {
                        ct -= Sd;
                        jt++;
                    }
                }
#pragma unroll
                for (int x = 0; x < 4; x++) thr[x] = s_thr[B.tb[jx[x]] + min(max(de[x], 0) >> 1, kmax)];
                uint32_t u[4], drawn = 0;
                rng4.peek(u);
                bool acc[4];
#pragma unroll
                for (int x = 0; x < 4; x++) {
                    const bool up = de[x] > 0;
                    acc[x] = sx[x] != 0 && (!up || u[0] < thr[x] || thr[x] == 0xFFFFFFFFu);
                    if (up) {
                        u[0] = u[1];
                        u[1] = u[2];
                        u[2] = u[3];
                        drawn++;
                    }
                }
                rng4.take(drawn);
#pragma unroll
                for (int x = 0; x < 4; x++) {
                    if (acc[x]) {
                        B.spin[jx[x] * npad + ix[x]] = (int8_t)-sx[x];
                        if (B.field) {
                            int32_t* const fd = B.field + jx[x] * npad;
                            const int dl = -2 * sx[x];
                            for_each_neighbour(row, adj, ix[x], [&](uint32_t e) {
                                atomicAdd(fd + (e >> 8), (int)(int8_t)(e & 0xffu) * dl);
                            });
                        }
                    }
                    // one shared-memory update per replica per warp instead of
                    // per flip (the items of a warp lie in one replica, or in
                    // a few neighbouring ones: its lanes' sums by replica)
                    unsigned left = __ballot_sync(0xffffffffu, acc[x]);
                    while (left) {
                        const int jj = __shfl_sync(0xffffffffu, jx[x], __ffs(left) - 1);
                        const bool mine = acc[x] && jx[x] == jj;
                        const unsigned grp = __ballot_sync(0xffffffffu, mine);
                        const int sde = (int)__reduce_add_sync(0xffffffffu, mine ? (unsigned)de[x] : 0u);
                        if (lane == 0) {
                            atomicAdd(s_dEp + jj, sde);
                            atomicAdd(s_flp + jj, (unsigned)__popc(grp));
                        }
                        left &= ~grp;
                    }
                }
            }
        }
        const bool track = best_per_phase || c + 1 == D.ncolors;
        if (ONE && track) {
            int v = acc_de;
            unsigned f = acc_fl;
            for (int o = 16; o > 0; o >>= 1) {
                v += __shfl_xor_sync(0xffffffffu, v, o);
                f += __shfl_xor_sync(0xffffffffu, f, o);
            }
            if (lane == 0 && (v != 0 || f != 0)) {
                atomicAdd(s_dEp, v);
                atomicAdd(s_flp, f);
            }
            acc_de = 0;
            acc_fl = 0;
        }
        __syncthreads();
        if (!track) continue;
        // phase boundary: fold the phase's energy change, track the best state
        for (int jj = tid; jj < rpc; jj += T) {
            const int r = B.r0 + jj;
            const long long E = B.E[r] + s_dEp[jj];
            B.E[r] = E;
            s_dEp[jj] = 0;
            s_flips[jj] += s_flp[jj];
            s_flp[jj] = 0;
            const bool imp = E < s_bestE[jj];
            s_improved[jj] = imp;
            if (imp) {
                s_bestE[jj] = E;
                A.best_sweep[D.rep_off + r] = sweep_idx;
                atomicAdd(s_misc + 1, 1);
            }
        }
        __syncthreads();
        if (s_misc[1] > 0) {
            for (int idx = tid; idx < rpc * npad; idx += T) {
                const int j = ONE ? 0 : idx / npad;
                if (s_improved[j])
                    A.best_state[D.spin_off + (long long)B.r0 * npad + idx] = spin_row<SPACE>(B, j)[idx - j * npad];
            }
            __syncthreads();
            if (tid == 0) s_misc[1] = 0;
            __syncthreads();
        }
    }
}

// Sequential sweep in the reference's site order (replay).  One warp per
// replica: lane 0 makes each decision exactly as src/replica.cc:31-38 does
// (dE <= 0, else u < exp(-beta*dE) with a recorded u), the warp applies the
// field update and copies a new best state (src/replica.cc:18-29).
static __device__ void replay_sweep(const EngineArgs& A, const BlockCtx& B, int ls, int sw,
                             unsigned long long sweep_idx, const double* s_ptab,
                             unsigned long long* s_flips, long long* s_bestE) {
    const InstanceDesc& D = B.D;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n = D.n, npad = D.n_pad, kst = D.kmax + 1;
    for (int j = warp; j < D.rpc; j += nw) {
        const int r = B.r0 + j;
        int8_t* sp = B.spin + j * npad;
        int32_t* fd = B.field + j * npad;
        const long long oi = ((long long)ls * A.sweeps + sw) * D.R + r;
        unsigned long long pos = A.replay.sweep_offsets[oi];
        const unsigned long long end = A.replay.sweep_offsets[oi + 1];
        const int pbase = (int)(B.rslot[j] % (uint32_t)D.nt) * kst;
        long long E = B.E[r];
        long long bestE = s_bestE[j];
        unsigned long long flips = 0;
        bool bad = false;
        for (int o = 0; o < n; o++) {
            const int i = A.perm[D.perm_off + o];
            int acc = 0, s = 0, de = 0;
            if (lane == 0) {
                s = sp[i];
                const int f = fd[i] + (B.h ? B.h[i] : 0);
                de = -2 * s * f;
                if (de <= 0) {
                    acc = 1;
                } else {
                    double u = 1.0;
                    if (pos < end && pos < A.replay.n_uniforms) u = A.replay.uniforms[pos];
                    else bad = true;
                    pos++;
                    acc = u < s_ptab[pbase + min(de >> 1, D.kmax)];
                }
            }
            acc = __shfl_sync(0xffffffffu, acc, 0);
            if (!acc) continue;
            s = __shfl_sync(0xffffffffu, s, 0);
            de = __shfl_sync(0xffffffffu, de, 0);
            if (lane == 0) sp[i] = (int8_t)-s;
            const int e0 = B.row[i], e1 = B.row[i + 1];
            for (int a = e0 + lane; a < e1; a += 32) {
                const uint32_t e = B.adj[a];
                atomicAdd(fd + (e >> 8), (int)(int8_t)(e & 0xffu) * (-2 * s));
            }
            E += de;
            flips++;
            __syncwarp();
            if (E < bestE) {
                bestE = E;
                for (int x = lane; x < npad; x += 32) A.best_state[D.spin_off + (long long)r * npad + x] = sp[x];
                if (lane == 0) A.best_sweep[D.rep_off + r] = sweep_idx;
            }
            __syncwarp();
        }
        if (lane == 0) {
            if (bad || pos != end) dev_fail(A.status, A.abort_flag, DEV_REPLAY_MISMATCH, 10, oi, (long long)(end - pos));
            B.E[r] = E;
            s_bestE[j] = bestE;
            s_flips[j] += flips;
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------- exchange
// Accepts a swap with energy difference dE across dbeta: x = dbeta * dE > 0
// or log u < x, in FP64.  The sign of x is the product of the signs, and the
// comparison is decided in FP32 unless log u lies within 1e-5 of x relative
// to |x| (the FP32 product is within 2^-21 of x), so that the FP64 pipe,
// slow on this chip, is left to about one attempt in 10^5.
__device__ __forceinline__ bool swap_accepted(double dbeta, long long dE, float log_u) {
    const float db = (float)dbeta, xf = db * (float)dE;
    if (dE == 0 && fabsf(db) < 1e30f) return log_u < 0.f;
    if (fabsf(xf) > 1e-30f && fabsf(db) > 1e-30f) {
        if (xf > 0.f) return true;
        if (fabsf(log_u - xf) > 1e-5f * fabsf(xf)) return log_u < xf;
    }
    const double x = dbeta * (double)dE;
    return x > 0.0 || (double)log_u < x;
}

// Production exchange with the reference's attempt order
// (src/replica_exchange.cc:5-100): a shuffled order of the nt-1 adjacent
// pairs is walked by one cursor shared by all chains (attempt a goes to chain
// a % chains); the order is reshuffled whenever the cursor wraps.  Attempt
// on pair k accepts iff dBeta*dE > 0 or log u < dBeta*dE, and swaps the
// slot->replica entries.  Within one pass over the order each pair appears
// once, so an attempt waits only for earlier attempts on the neighbouring
// pairs of its chain; all attempts that wait for none are made together,
// with exactly the sequential semantics.
//
// Everything but the energies is known beforehand: the draws (by the whole
// block), and by one warp each pass's chains, waits and the next pass's order,
// one word per (pass, pair), before the wait for the other blocks' energies.
// (Levels by relaxation, attempts in FP64 and the reshuffles after that wait
// took 8.2 us for 20 pairs and two chains.)
constexpr uint32_t kWaitLeft = 1u << 30, kWaitRight = 1u << 31, kPosBits = 24;

static __device__ void exchange_reference_draw(const EngineArgs& A, const InstanceDesc& D, unsigned long long step,
                                        float* s_xlogu, uint32_t* s_xrand) {
    const int total = D.chains * (D.nt - 1), ndraw = 2 * total;
    const uint2 key = stream_key(A.seed, STREAM_EXCHANGE);
    for (int call = threadIdx.x; call * 4 < ndraw; call += blockDim.x) {
        const uint4 r = philox4x32_10(make_uint4((uint32_t)call, (uint32_t)D.inst_id, (uint32_t)step,
                                                 (uint32_t)(step >> 32)), key);
        const uint32_t v[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int dix = call * 4 + q;
            if (dix < total) s_xlogu[dix] = __logf(u01_open0(v[q]));
            else if (dix < ndraw) s_xrand[dix - total] = v[q];
        }
    }
    __syncthreads();
}

// One warp: s_xrand's shuffle keys become, per (pass, pair), the pair's
// position in the pass's order (low 24 bits), its chain (six bits) and whether
// an earlier attempt on the pair below or above goes to the same chain.
// s_pos: each pair's position after all passes' reshuffles, which the exchange
// makes the order.
static __device__ void exchange_reference_plan(const InstanceDesc& D, const uint32_t* s_order, uint32_t* s_xrand,
                                        uint32_t* s_pos, int* s_next) {
    const int lane = threadIdx.x & 31, C = D.chains, m = D.nt - 1;
    for (int i = lane; i < m; i += 32) s_pos[s_order[i]] = (uint32_t)i;
    __syncwarp();
    for (int round = 0; round < C; round++) {
        uint32_t* const keys = s_xrand + round * m;
        for (int kb = lane; kb < m; kb += 32) {
            const int p = (int)s_pos[kb];
            // the pair's next position: the rank of its key (ties by position)
            const uint32_t mine = keys[p];
            int rank = 0;
#pragma unroll 8
            for (int j = 0; j < m; j++) {
                const uint32_t kj = keys[j];
                rank += (kj < mine) || (kj == mine && j < p);
            }
            s_next[kb] = rank;
        }
        __syncwarp();
        for (int kb = lane; kb < m; kb += 32) {
            const int p = (int)s_pos[kb], c = (round * m + p) % C;
            uint32_t w = (uint32_t)p | ((uint32_t)c << kPosBits);
            if (kb > 0) {
                const int q = (int)s_pos[kb - 1];
                if (q < p && (round * m + q) % C == c) w |= kWaitLeft;
            }
            if (kb + 1 < m) {
                const int q = (int)s_pos[kb + 1];
                if (q < p && (round * m + q) % C == c) w |= kWaitRight;
            }
            keys[kb] = w;
        }
        __syncwarp();
        for (int kb = lane; kb < m; kb += 32) s_pos[kb] = (uint32_t)s_next[kb];
        __syncwarp();
    }
}

static __device__ void exchange_reference_order(const BlockCtx& B, const double* s_dbeta, unsigned* s_att, unsigned* s_succ,
                                         const float* s_xlogu, const uint32_t* s_xrand, const uint32_t* s_pos,
                                         uint32_t* s_order, int* s_done, const Prof P) {
    const InstanceDesc& D = B.D;
    const int nt = D.nt, C = D.chains, m = nt - 1;
    if (m > 0 && threadIdx.x < 32) {
        const int lane = threadIdx.x;
        uint32_t* const slot = B.slot;
        const long long* const E = B.E;
        auto attempt = [&](int kb, uint32_t w, int round) {
            const int k = (int)((w >> kPosBits) & 63u) * nt + kb;
            const uint32_t r1 = slot[k], r2 = slot[k + 1];
            s_att[k]++;
            if (swap_accepted(s_dbeta[kb], E[r1] - E[r2], s_xlogu[round * m + (int)(w & ((1u << kPosBits) - 1u))])) {
                s_succ[k]++;
                slot[k] = r2;
                slot[k + 1] = r1;
            }
        };
        if (m <= 64) {
            // two pairs per lane (lane, lane + 32), the attempts made as bits
            // of one word: 20 pairs and two chains take 4.0 -> 2.2 us
            for (int round = 0; round < C; round++) {
                uint32_t w[2];
                unsigned long long needs[2];   // attempts waited for
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int kb = lane + 32 * q;
                    w[q] = kb < m ? s_xrand[round * m + kb] : 0u;
                    needs[q] = (w[q] & kWaitLeft ? 1ull << ((kb - 1) & 63) : 0ull) |
                               (w[q] & kWaitRight ? 1ull << ((kb + 1) & 63) : 0ull);
                }
                unsigned long long todo = m == 64 ? ~0ull : (1ull << m) - 1ull;
                while (todo) {
                    const bool g0 = ((todo >> lane) & 1ull) && !(needs[0] & todo);
                    const bool g1 = ((todo >> (lane + 32)) & 1ull) && !(needs[1] & todo);
                    if (g0) attempt(lane, w[0], round);
                    if (g1) attempt(lane + 32, w[1], round);
                    const unsigned long long made = (unsigned long long)__ballot_sync(0xffffffffu, g0) |
                                                    ((unsigned long long)__ballot_sync(0xffffffffu, g1) << 32);
                    if (made == 0) break;   // (cannot happen: the earliest attempt left waits for none)
                    todo &= ~made;
                    __syncwarp();
                }
            }
        } else {
            volatile int* const done = s_done;
            for (int round = 0; round < C; round++) {
                for (int kb = lane; kb < m; kb += 32) done[kb] = 0;
                __syncwarp();
                for (int left = m; left > 0;) {
                    // the attempts that wait for none (marked 2 until all have looked)
                    int made = 0;
                    for (int kb = lane; kb < m; kb += 32) {
                        const uint32_t w = s_xrand[round * m + kb];
                        if (done[kb] == 0 && !((w & kWaitLeft) && done[kb - 1] != 1) && !((w & kWaitRight) && done[kb + 1] != 1)) {
                            attempt(kb, w, round);
                            done[kb] = 2;
                            made++;
                        }
                    }
                    __syncwarp();
                    for (int kb = lane; kb < m; kb += 32)
                        if (done[kb] == 2) done[kb] = 1;
                    __syncwarp();
                    made = __reduce_add_sync(0xffffffffu, made);
                    if (made == 0) break;   // (as above)
                    left -= made;
                }
            }
        }
        for (int kb = lane; kb < m; kb += 32) s_order[s_pos[kb]] = (uint32_t)kb;
        P.subtick(PROF_X_APPLY);
    }
    __syncthreads();
}

// Log-uniforms of the even/odd exchange: a thread's pair of each pass, drawn
// before the step's energies are known (they do not depend on them).
struct EvenOddDraws {
    float lu0, lu1;
};

__device__ __forceinline__ float even_odd_log_u(unsigned long long seed, uint32_t inst, unsigned long long step, int k,
                                                int par) {
    const uint4 r = philox4x32_10(make_uint4((uint32_t)(k | (par << 30)), inst, (uint32_t)step, (uint32_t)(step >> 32)),
                                  stream_key(seed, STREAM_EXCHANGE));
    return __logf(u01_open0(r.x));
}

// The t-th pair of a pass (pairs kb = par, par + 2, ... of every chain).
__device__ __forceinline__ int even_odd_pair(int t, int par, int per_chain, int nt, int& kb) {
    const int c = t / per_chain;
    kb = par + 2 * (t - c * per_chain);
    return c * nt + kb;
}

__device__ __forceinline__ EvenOddDraws even_odd_draw(const EngineArgs& A, const InstanceDesc& D, unsigned long long step) {
    const int nt = D.nt, C = D.chains, m = nt - 1, per0 = (m + 1) / 2, per1 = m / 2;
    const int tid = threadIdx.x;
    EvenOddDraws u{0.f, 0.f};
    if (C * per0 > (int)blockDim.x) return u;   // (then drawn as the pairs are visited)
    int kb;
    if (tid < C * per0) u.lu0 = even_odd_log_u(A.seed, (uint32_t)D.inst_id, step, even_odd_pair(tid, 0, per0, nt, kb), 0);
    if (tid < C * per1) u.lu1 = even_odd_log_u(A.seed, (uint32_t)D.inst_id, step, even_odd_pair(tid, 1, per1, nt, kb), 1);
    return u;
}

// Deterministic even/odd exchange: per chain, all even pairs, then all odd
// pairs, each set in parallel (nt-1 attempts per chain per step).
static __device__ void exchange_even_odd(const EngineArgs& A, const BlockCtx& B, unsigned long long step,
                                  const double* s_dbeta, unsigned* s_att, unsigned* s_succ, EvenOddDraws u) {
    const InstanceDesc& D = B.D;
    const int tid = threadIdx.x, T = blockDim.x;
    const int nt = D.nt, C = D.chains, m = nt - 1;
    const uint32_t inst = (uint32_t)D.inst_id;
    uint32_t* const slot = B.slot;
    const long long* const E = B.E;
    const int per0 = (m + 1) / 2, per1 = m / 2;
    const bool one = C * per0 <= T;   // at most one pair per thread and pass: drawn ahead
    for (int par = 0; par < 2; par++) {
        const int per_chain = par ? per1 : per0;
        const int total = C * per_chain;
        for (int t = tid; t < total; t += T) {
            int kb;
            const int k = even_odd_pair(t, par, per_chain, nt, kb);
            const float lu = one ? (par ? u.lu1 : u.lu0) : even_odd_log_u(A.seed, inst, step, k, par);
            const uint32_t r1 = slot[k], r2 = slot[k + 1];
            s_att[k]++;
            if (swap_accepted(s_dbeta[kb], E[r1] - E[r2], lu)) {
                s_succ[k]++;
                slot[k] = r2;
                slot[k + 1] = r1;
            }
        }
        __syncthreads();
    }
}

// Replayed exchange: the recorded pair sequence and log-uniforms, applied
// sequentially in FP64 exactly as src/replica_exchange.cc:20-40 computes.
static __device__ void exchange_replay(const EngineArgs& A, const BlockCtx& B, int ls, const double* s_beta,
                                unsigned* s_att, unsigned* s_succ) {
    const InstanceDesc& D = B.D;
    if (threadIdx.x == 0) {
        const int nt = D.nt, per = D.chains * (nt - 1);
        for (int t = 0; t < per; t++) {
            const long long idx = (long long)ls * per + t;
            if (idx >= (long long)A.replay.n_xchg) {
                dev_fail(A.status, A.abort_flag, DEV_REPLAY_MISMATCH, 20, idx, 0);
                break;
            }
            const int k = A.replay.xchg_slot[idx];
            if (k < 0 || k + 1 >= D.R || (k % nt) == nt - 1) {
                dev_fail(A.status, A.abort_flag, DEV_BAD_INDEX, 21, idx, k);
                break;
            }
            const int kb = k % nt;
            const uint32_t r1 = B.slot[k], r2 = B.slot[k + 1];
            const double dB = __dsub_rn(s_beta[kb], s_beta[kb + 1]);
            const double dE = (double)(B.E[r1] - B.E[r2]);
            const double x = __dmul_rn(dB, dE);
            s_att[k]++;
            if (__dmul_rn(dE, dB) > 0.0 || A.replay.xchg_logu[idx] < x) {
                s_succ[k]++;
                B.slot[k] = r2;
                B.slot[k + 1] = r1;
            }
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------- kernel
// Launch bounds: blocks of several replicas, and narrow block teams (NARROW),
// run at most kNarrowThreads threads, which leaves each thread 128 registers
// instead of the 64 of a 1024-thread bound; replay and wide block teams (one
// replica of a large instance per block) keep 1024.
template <bool REPLAY, bool BLOCKTEAM, bool NARROW, int SPACE>
__global__ void __launch_bounds__((REPLAY || (BLOCKTEAM && !NARROW)) ? 1024 : kNarrowThreads, 1)
    pt_engine_kernel(const EngineArgs A) {
    extern __shared__ __align__(128) uint8_t smem[];
    // the job's descriptor and the profiling counters: one copy per block
    // (per-thread copies of uniform values would live in local memory)
    __shared__ InstanceDesc s_D;
    __shared__ int s_rank;
    __shared__ ProfStore s_prof;
    const SmemPlan& S = A.sm;
    const int tid = threadIdx.x, T = blockDim.x;
    volatile int* abortf = A.abort_flag;
    uint64_t* mbar = sm_ptr<uint64_t>(smem, S.mbar);
    if (S.stage_adj) {
        if (tid == 0) mbar_init(mbar, 1);
        __syncthreads();
    }
    uint32_t bulk_parity = 0;
    const int job_end = A.sched_off[blockIdx.x + 1];
    for (int job = A.sched_off[blockIdx.x]; job < job_end; job++) {
    const int inst = A.sched[2 * job];
    if (tid == 0) {
        s_D = A.desc[inst];
        s_rank = A.sched[2 * job + 1];
    }
    __syncthreads();
    const InstanceDesc& D = s_D;
    const int rank = s_rank, rep0 = rank * D.rpc;
    const int n = D.n, npad = D.n_pad, R = D.R, nt = D.nt, rpc = D.rpc, kst = D.kmax + 1;

    int32_t* s_col = sm_ptr<int32_t>(smem, S.col);
    int32_t* s_h = sm_ptr<int32_t>(smem, S.h);
    // acceptance thresholds: shared memory, or read through L1 (field_gather)
    uint32_t* s_thr_w = sm_ptr<uint32_t>(smem, S.thr);
    const bool thr_global = space_large(SPACE) || (SPACE == SP_ANY && S.field_gather);
    const uint32_t* s_thr = thr_global ? A.thr + D.thr_off : s_thr_w;
    double* s_ptab = sm_ptr<double>(smem, S.ptab);
    uint32_t* s_order = sm_ptr<uint32_t>(smem, S.order);
    double* s_beta = sm_ptr<double>(smem, S.beta);
    double* s_dbeta = sm_ptr<double>(smem, S.dbeta);
    int* s_dEp = sm_ptr<int>(smem, S.dEp);
    unsigned* s_flp = sm_ptr<unsigned>(smem, S.flp);
    long long* s_bestE = sm_ptr<long long>(smem, S.bestE);
    unsigned long long* s_flips = sm_ptr<unsigned long long>(smem, S.flips);
    int* s_improved = sm_ptr<int>(smem, S.improved);
    unsigned* s_att = sm_ptr<unsigned>(smem, S.att);
    unsigned* s_succ = sm_ptr<unsigned>(smem, S.succ);
    float* s_xlogu = sm_ptr<float>(smem, S.xlogu);
    uint32_t* s_xrand = sm_ptr<uint32_t>(smem, S.xrand);
    int* s_lvl = sm_ptr<int>(smem, S.xlevel);
    uint32_t* s_tmp = sm_ptr<uint32_t>(smem, S.xpos);
    uint8_t* const g_icm = A.icm_pool + (size_t)blockIdx.x * (size_t)A.icm_pool_stride;
    uint8_t* s_icm = smem + S.icm;
    if (SPACE == SP_ANY && (S.state_global || S.field_gather) && !S.icm_split) s_icm = g_icm;
    int* s_misc = sm_ptr<int>(smem, S.misc);
    long long* s_mag = sm_ptr<long long>(smem, S.mag);
    // a block team's keys (two per warp) and control words; warp teams use
    // the first two control words of a place of their own
    unsigned long long* s_team_keys = sm_ptr<unsigned long long>(smem, S.misc + 64);
    int* s_team_ctl = sm_ptr<int>(smem, S.misc + 64 + 16 * 32);
    int* s_warp_ctl = sm_ptr<int>(smem, S.misc + 64);

    const int32_t* g_row = A.row + D.row_off;
    const uint32_t* g_adj = A.adj + D.adj_off;

    // ---- stage the adjacency (bulk copies) and load the block's state
    bool staged = S.stage_adj && D.stage;
    if (staged && ((reinterpret_cast<uintptr_t>(g_row) | reinterpret_cast<uintptr_t>(g_adj)) & 15u)) {
        // a bulk copy needs 16-byte aligned sources: record and skip it
        if (tid == 0) dev_fail(A.status, A.abort_flag, DEV_BAD_INDEX, 3, blockIdx.x, inst);
        staged = false;
    }
    if (staged) {
        int32_t* s_row = sm_ptr<int32_t>(smem, S.row);
        uint32_t* s_adj = sm_ptr<uint32_t>(smem, S.adj);
        if (tid == 0) {
            // the previous job's generic-proxy reads of this region are done
            // (block barrier at the end of every job); order them before the
            // bulk copy's writes
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            const uint32_t rb = (uint32_t)(((n + 1) * 4 + 15) & ~15);
            const uint32_t ab = (uint32_t)((D.nnz * 4 + 15) & ~15);
            mbar_expect_tx(mbar, rb + ab);
            bulk_g2s(s_row, g_row, rb, mbar);
            if (ab) bulk_g2s(s_adj, g_adj, ab, mbar);
        }
    }
    if (SPACE == SP_SHARED && !staged) {
        // (recorded above; the other blocks of the group see the abort)
        __syncthreads();
        continue;
    }
    BlockCtx B{D, rank, rep0};
    B.spin = sm_ptr<int8_t>(smem, S.spin);
    // (a narrow block team with lanes gathers its fields)
    B.field = (BLOCKTEAM && NARROW && D.lanes > 0) || space_large(SPACE) || (SPACE == SP_ANY && S.field_gather) ? nullptr : sm_ptr<int32_t>(smem, S.field);
    if (SPACE == SP_ANY && S.state_global) {
        // replicas too large for shared memory work on their master copy
        B.spin = A.spins + D.spin_off + (long long)rep0 * D.n_pad;
        if (!(BLOCKTEAM && NARROW && D.lanes > 0)) B.field = A.fields + D.spin_off + (long long)rep0 * D.n_pad;
    }
    B.slot = sm_ptr<uint32_t>(smem, S.slot);
    B.rslot = sm_ptr<uint32_t>(smem, S.rslot);
    B.tb = sm_ptr<int32_t>(smem, S.rslot) + rpc;
    B.E = sm_ptr<long long>(smem, S.E);
    B.h = D.has_h ? s_h : nullptr;
    B.row = sm_ptr<int32_t>(smem, S.row);
    B.adj = sm_ptr<uint32_t>(smem, S.adj);
    if (space_large(SPACE) || (SPACE != SP_SHARED && !staged)) {
        B.row = g_row;
        B.adj = g_adj;
    }
    for (int i = tid; i <= D.ncolors; i += T) s_col[i] = A.col[D.col_off + i];
    if (D.has_h)
        for (int i = tid; i < n; i += T) s_h[i] = A.hpool[D.h_off + i];
    if (!S.state_global) {
        const long long base = D.spin_off + (long long)B.r0 * npad;
        for (int idx = tid; idx < rpc * npad; idx += T) {
            const int j = space_stride(SPACE) == 1 ? 0 : idx / npad;
            spin_row<SPACE>(B, j)[idx - j * npad] = A.spins[base + idx];
            if (B.field) B.field[idx] = A.fields[base + idx];
        }
    }
    for (int r = tid; r < R; r += T) {
        B.slot[r] = A.slot_rep[D.rep_off + r];
        B.E[r] = A.energy[D.rep_off + r];
        s_att[r] = 0;
        s_succ[r] = 0;
    }
    for (int k = tid; k < nt; k += T) {
        s_order[k] = A.xorder[D.rep_off + k];
        s_beta[k] = A.beta[D.beta_off + k];
    }
    for (int k = tid; k < nt * kst; k += T) {
        if (!thr_global) s_thr_w[k] = A.thr[D.thr_off + k];
        if (REPLAY) s_ptab[k] = A.ptab[D.ptab_off + k];
    }
    for (int j = tid; j < rpc; j += T) {
        s_bestE[j] = A.best_E[D.rep_off + B.r0 + j];
        s_flips[j] = 0;
        s_dEp[j] = 0;
        s_flp[j] = 0;
        s_improved[j] = 0;
    }
    if (tid < 8) s_misc[tid] = 0;
    // the group barrier's generation (it cannot move before this block arrives)
    unsigned int bar_gen = 0;
    if (tid == 0 && D.group > 1) bar_gen = *(volatile unsigned int*)(A.bar + 2 * inst + 1);
    if (tid == 0) {
        for (int q = 0; q < TC_WORDS; q++) s_team_ctl[q] = 0;
    }
    __syncthreads();
    for (int k = tid; k + 1 < nt; k += T) s_dbeta[k] = s_beta[k] - s_beta[k + 1];
    for (int s = tid; s < R; s += T) {
        const uint32_t r = B.slot[s];
        if ((int)r >= B.r0 && (int)r < B.r0 + rpc) {
            B.rslot[r - B.r0] = (uint32_t)s;
            B.tb[r - B.r0] = (int)(((uint32_t)s % (uint32_t)nt) * (uint32_t)kst);
        }
    }
    if (staged) {
        if (!mbar_wait_bounded(mbar, bulk_parity, A.wait_limit_ns ? A.wait_limit_ns : kWaitLimitNs) && tid == 0)
            dev_fail(A.status, A.abort_flag, DEV_TMA_TIMEOUT, 2, blockIdx.x, inst);
        bulk_parity ^= 1u;
    }
    __syncthreads();

    const bool icm_on = (A.phase_mask & PHASE_ICM) && D.nc > 0 && D.chains >= 2;
    const Prof P{A.prof != nullptr && tid == 0, &s_prof};
    P.init();
    const long long t_start = P.on ? s_prof.mark : 0;
    const bool best_pp = (A.flags & ENGINE_BEST_PER_PHASE) != 0;
    unsigned long long t_step1 = 0;
    for (int ls = 0; ls < A.nsteps; ls++) {
        if (ls == 1 && tid == 0) t_step1 = globaltimer_ns();
        if (D.group == 1 && (ls & 15) == 0) {
            // (a group of blocks sees an abort in its barrier; a block alone
            // looks every sixteenth step, a read of L2)
            if (tid == 0) s_misc[3] = *abortf;
            __syncthreads();
            if (s_misc[3]) break;
        }
        const unsigned long long step = A.step0 + (unsigned long long)ls;
        const int parity = (int)(step & 1ull);
        // (profiling) a block holding one replica at an ICM temperature
        const bool cold = P.on && icm_on && rpc == 1 && (nt - 1 - (int)(B.rslot[0] % (uint32_t)nt)) < D.nc;
        const long long t_sw = P.on ? clock64() : 0;
        if (A.phase_mask & PHASE_SWEEP) {
            for (int sw = 0; sw < A.sweeps; sw++) {
                const unsigned long long sweep_idx = step * (unsigned long long)A.sweeps + (unsigned long long)sw;
                if (REPLAY) {
                    replay_sweep(A, B, ls, sw, sweep_idx, s_ptab, s_flips, s_bestE);
                    __syncthreads();
                } else {
                    colored_sweep<BLOCKTEAM, BLOCKTEAM && NARROW, SPACE>(A, B, sweep_idx, s_col, s_thr, s_dEp, s_flp, s_flips, s_bestE,
                                             s_improved, s_misc, best_pp);
                }
            }
        }
        P.tick(PROF_SWEEP);
        if (cold) s_prof.c[PROF_SWEEP_ICM] += clock64() - t_sw;
        const bool observe = A.obs != nullptr && D.hist_nbins > 0 && step >= A.hist_from;
        if (observe) {
            // magnetisation of the block's replicas, one warp per replica
            const int warp = tid >> 5, lane = tid & 31;
            for (int j = warp; j < rpc; j += (T >> 5)) {
                long long m = 0;
                for (int i = lane; i < n; i += 32) m += spin_row<SPACE>(B, j)[i];
                for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
                if (lane == 0) s_mag[j] = m;
            }
            __syncthreads();
            if (D.group > 1)
                for (int j = tid; j < rpc; j += T)
                    A.mag_pub[parity * A.energy_pub_half + D.rep_off + B.r0 + j] = s_mag[j];
        }
        // the exchange's draws, before the wait for the energies
        EvenOddDraws xdraw{0.f, 0.f};
        const bool even_odd = !REPLAY && (A.phase_mask & PHASE_EXCHANGE) && (A.flags & ENGINE_EXCHANGE_EVEN_ODD);
        const bool ordered = !REPLAY && (A.phase_mask & PHASE_EXCHANGE) && !(A.flags & ENGINE_EXCHANGE_EVEN_ODD) && nt > 1;
        auto draw = [&]() {
            if (even_odd) xdraw = even_odd_draw(A, D, step);
            if (ordered) {
                exchange_reference_draw(A, D, step, s_xlogu, s_xrand);
                if (tid < 32) exchange_reference_plan(D, s_order, s_xrand, s_tmp, s_lvl);
            }
        };
        // Publishes this block's spins (for ICM partners) as words of 32
        // sites carrying the step's tag: a partner checks the tag of each
        // word it reads, so nothing orders these stores and no fence waits
        // for them (one bit a site: N=2000 goes out in 63 words).
        // A thread packs the 32 spin bytes of a word: the sign bits of four
        // bytes are gathered by one multiplication.
        auto publish_spins = [&]() {
            const int W = (n + 31) >> 5, npw = npad >> 4;
            const unsigned long long tagw = (unsigned long long)(A.pub_base + (uint32_t)ls) << 32;
            unsigned long long* const out = A.spins_pub + parity * A.spins_pub_half + (D.spin_off >> 4) + (long long)B.r0 * npw;
            const int8_t* const sp = B.spin;
            if (SPACE == SP_LARGE4) {
                // (32 interleaved words give a word of each replica)
                for (int k = tid; k < W; k += T) {
                    uint32_t bits[4] = {0, 0, 0, 0};
                    const uint4* const q = reinterpret_cast<const uint4*>(sp + 128 * (long long)k);
#pragma unroll
                    for (int x4 = 0; x4 < 8; x4++) {
                        if (32 * k + 4 * x4 >= npad) break;
                        const uint4 v = q[x4];
                        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int x = 0; x < 4; x++)
#pragma unroll
                            for (int j = 0; j < 4; j++) bits[j] |= ((~w[x] >> (8 * j + 7)) & 1u) << (4 * x4 + x);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) st_relaxed_gpu_u64(out + (long long)j * npw + k, tagw | bits[j]);
                }
            }
            for (int j = 0; space_stride(SPACE) == 1 && j < rpc; j++)
                for (int k = tid; k < W; k += T) {
                    const uint4* const q = reinterpret_cast<const uint4*>(sp + (long long)j * npad + 32 * k);
                    uint32_t v[8] = {};
                    const uint4 lo = q[0];
                    v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
                    if (32 * k + 16 < npad) {
                        const uint4 hi = q[1];
                        v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
                    }
                    uint32_t bits = 0;
#pragma unroll
                    for (int b = 0; b < 8; b++)
                        bits |= ((((~v[b] >> 7) & 0x01010101u) * 0x10204080u) >> 28) << (4 * b);
                    st_relaxed_gpu_u64(out + (long long)j * npw + k, tagw | bits);
                }
        };
        if (D.group > 1 && A.flag_barrier) {
            // publish each of the block's replicas' energy tagged with this
            // step in one 64-bit word, then its spins; wait for every other
            // replica's word of this step.  Every word read across blocks
            // carries its own tag, so the words need no order among
            // themselves: a release and an acquire (two L2 round trips on
            // the step's critical path) are paid only when published
            // magnetisations, which carry no tag, ride along.
            unsigned long long* const ew = reinterpret_cast<unsigned long long*>(A.energy_pub) +
                                           (parity * A.energy_pub_half + D.rep_off) * kPubStride;
            const uint32_t tag = A.pub_base + (uint32_t)ls;
            if (observe) __syncthreads();
            for (int j = tid; j < rpc; j += T) {
                const unsigned long long w = pub_word(tag, B.E[B.r0 + j]);
                if (observe) st_release_gpu_u64(ew + (B.r0 + j) * kPubStride, w);
                else st_relaxed_gpu_u64(ew + (B.r0 + j) * kPubStride, w);
            }
            if (A.publish_delay_ns && (B.rank & 1)) {
                const unsigned long long from = globaltimer_ns();
                while (globaltimer_ns() - from < A.publish_delay_ns) __nanosleep(200);
            }
            if (icm_on) publish_spins();
            draw();
            const unsigned long long limit = A.wait_limit_ns ? A.wait_limit_ns : kWaitLimitNs;
            int ok = 1;
            bool polled = false;
            for (int r0 = tid & ~31; r0 < R && ok; r0 += T) {
                const int r = r0 + (tid & 31);
                const bool need = r < R && (r < B.r0 || r >= B.r0 + rpc);
                unsigned long long w = 0;
                ok = poll_tagged(ew + (need ? r : 0) * kPubStride, need, tag, w, abortf, A.status, limit, 1);
                if (need && ok) B.E[r] = (long long)(int32_t)(uint32_t)w;
                polled |= need;
            }
            if (A.bar_phantom && tid == 0 && ok) {
                // test hook: one more member whose word never comes
                const unsigned long long t0 = globaltimer_ns();
                while (ok) {
                    if (*abortf) ok = 0;
                    else if (globaltimer_ns() - t0 > limit) {
                        dev_fail(A.status, A.abort_flag, DEV_BARRIER_TIMEOUT, 1, blockIdx.x, tag);
                        ok = 0;
                    } else __nanosleep(256);
                }
            }
            if (observe && polled) fence_acq_rel_gpu();
            if (!__syncthreads_and(ok)) break;
        } else if (D.group > 1) {
            // publish this block's energies (and spins, for ICM partners)
            for (int j = tid; j < rpc; j += T) A.energy_pub[parity * A.energy_pub_half + D.rep_off + B.r0 + j] = B.E[B.r0 + j];
            if (icm_on) publish_spins();
            draw();
            if (!group_barrier(A.bar + 2 * inst, (unsigned)(D.group + A.bar_phantom), abortf, A.status, bar_gen,
                               A.wait_limit_ns ? A.wait_limit_ns : kWaitLimitNs))
                break;
            for (int r = tid; r < R; r += T)
                if (r < B.r0 || r >= B.r0 + rpc) B.E[r] = ld_cg(A.energy_pub + parity * A.energy_pub_half + D.rep_off + r);
            __syncthreads();
        } else {
            draw();
        }
        P.tick(PROF_BARRIER);
        if (A.hist != nullptr && D.hist_nbins > 0 && step >= A.hist_from && B.rank == 0) {
            for (int k = tid; k < R; k += T) {
                const int r = (int)B.slot[k];
                const long long bin = (B.E[r] - D.hist_lo) >> 1;
                if (bin >= 0 && bin < D.hist_nbins)
                    atomicAdd(A.hist + D.hist_off + (long long)k * D.hist_nbins + bin, 1u);
                if (observe) {
                    const long long m = (r >= B.r0 && r < B.r0 + rpc)
                                            ? s_mag[r - B.r0]
                                            : ld_cg(A.mag_pub + parity * A.energy_pub_half + D.rep_off + r);
                    unsigned long long* o = reinterpret_cast<unsigned long long*>(A.obs + 2 * (D.rep_off + k));
                    atomicAdd(o, (unsigned long long)m);
                    atomicAdd(o + 1, (unsigned long long)(m * m));
                }
            }
            __syncthreads();
        }
        if (A.phase_mask & PHASE_EXCHANGE) {
            if (REPLAY) exchange_replay(A, B, ls, s_beta, s_att, s_succ);
            else if (A.flags & ENGINE_EXCHANGE_EVEN_ODD) exchange_even_odd(A, B, step, s_dbeta, s_att, s_succ, xdraw);
            else exchange_reference_order(B, s_dbeta, s_att, s_succ, s_xlogu, s_xrand, s_tmp, s_order, s_lvl, P);
            for (int s = tid; s < R; s += T) {
                const uint32_t r = B.slot[s];
                if ((int)r >= B.r0 && (int)r < B.r0 + rpc) {
                    B.rslot[r - B.r0] = (uint32_t)s;
                    B.tb[r - B.r0] = (int)(((uint32_t)s % (uint32_t)nt) * (uint32_t)kst);
                }
            }
            __syncthreads();
        }
        P.tick(PROF_EXCHANGE);
        if (icm_on) {
            // pairs q = cp*nc + kk: slots (2cp)*nt + k and (2cp+1)*nt + k, k = nt-1-kk
            // the block's pairs, found from its own replicas' slots: replica
            // j at slot s (chain c = s / nt, temperature k = s % nt) is in pair
            // q = (c / 2) nc + (nt-1-k) when nt-1-k < nc; a pair with both
            // replicas in the block is taken from its first chain's side
            const int chains_even = D.chains & ~1;
            // the whole block is one team when it holds one replica, or when
            // the instance is configured with one team (large instances: a
            // pair per block-wide team, in sequence, beats a pair per warp)
            if (BLOCKTEAM || D.teams == 1) {
                const Team<true> team{tid, T, s_team_ctl, s_team_keys};
                IcmScratch X = icm_scratch(s_icm, npad);
                if (space_large(SPACE) || (SPACE == SP_ANY && !BLOCKTEAM && !REPLAY && S.icm_split))
                    X.list = reinterpret_cast<int*>(g_icm);
                // Large instances: every pair is worked out once, by the block
                // q mod group whichever it holds, and the owners of its two
                // replicas read the result.  (Each owner for itself, up to
                // rpc pairs in a row in the blocks of cold replicas, none in
                // the others and every pair twice: 294 us a step of N=20000
                // with 136 pairs on 128 blocks; shared 167 us, the time of
                // the two pairs that eight of the blocks get.)
                const bool share = space_large(SPACE) && A.icm_pub != nullptr && D.group > 1 && A.flag_barrier &&
                                   D.icm_algo == ENGINE_ICM_UNION_FIND && !A.icm_exact && A.icm_force == nullptr;
                const int e1 = share ? (chains_even >> 1) * D.nc : rpc, de = share ? D.group : 1;
                for (int e = share ? B.rank : 0; e < e1; e += de) {
                    int cp, kk;
                    if (share) {
                        cp = e / D.nc;
                        kk = e - cp * D.nc;
                    } else {
                        const int sl = (int)B.rslot[e], c = sl / nt;
                        cp = c >> 1;
                        kk = nt - 1 - (sl - c * nt);
                        if (kk >= D.nc || c >= chains_even) continue;
                    }
                    const int k = nt - 1 - kk;
                    const int rA = (int)B.slot[(2 * cp) * nt + k], rB = (int)B.slot[(2 * cp + 1) * nt + k];
                    if (!share && (int)B.rslot[e] >= (2 * cp + 1) * nt && rA >= B.r0 && rA < B.r0 + rpc) continue;
                    icm_pair<true, REPLAY, !REPLAY && (NARROW || !BLOCKTEAM), SPACE, !REPLAY && !BLOCKTEAM>(
                        A, B, team, cp * D.nc + kk, rA, rB, step, ls, X, 30, P,
                        share ? A.icm_pub + (long long)e * A.icm_pub_stride : nullptr);
                }
                if (share) {
                    __syncthreads();
                    if (!__syncthreads_and(apply_pairs<SPACE>(A, B, chains_even, A.pub_base + (uint32_t)ls, abortf))) break;
                }
            } else {
                const int warp = tid >> 5, lane = tid & 31;
                const int teams = min(D.teams, T >> 5);
                if (warp < teams) {
                    const Team<false> team{lane, 32, s_warp_ctl + 2 * warp, nullptr};
                    const IcmScratch X = icm_scratch(s_icm + (size_t)warp * icm_team_bytes(npad), npad);
                    int e = 0;
                    for (int j = 0; j < rpc; j++) {
                        const int sl = (int)B.rslot[j], c = sl / nt, k = sl - c * nt, kk = nt - 1 - k;
                        if (kk >= D.nc || c >= chains_even) continue;
                        const int cp = c >> 1;
                        const int rA = (int)B.slot[(2 * cp) * nt + k], rB = (int)B.slot[(2 * cp + 1) * nt + k];
                        if ((c & 1) && rA >= B.r0 && rA < B.r0 + rpc) continue;
                        if ((e++ % teams) != warp) continue;
                        icm_pair<false, REPLAY, false, SPACE>(A, B, team, cp * D.nc + kk, rA, rB, step, ls, X, 30, P);
                    }
                }
            }
            __syncthreads();
        }
        P.tick(PROF_ICM);
    }
    __syncthreads();
    if (A.job_ns != nullptr && tid == 0 && A.nsteps > 1) A.job_ns[job] = globaltimer_ns() - t_step1;
    if (P.on) {
        s_prof.c[PROF_TOTAL] = clock64() - t_start;
        for (int q = 0; q < PROF_PHASES; q++) A.prof[(size_t)blockIdx.x * PROF_PHASES + q] += (unsigned long long)s_prof.c[q];
    }
    // ---- write the block's state back
    const long long base = D.spin_off + (long long)B.r0 * npad;
    if (SPACE != SP_ANY || !S.state_global)
        for (int idx = tid; idx < rpc * npad; idx += T) {
            const int j = space_stride(SPACE) == 1 ? 0 : idx / npad;
            A.spins[base + idx] = spin_row<SPACE>(B, j)[idx - j * npad];
            if (B.field) A.fields[base + idx] = B.field[idx];
        }
    if (!B.field) {
        // the stored fields of the master copy, gathered once per launch
        for (int idx = tid; idx < rpc * npad; idx += T) {
            const int j = idx / npad, i = idx - j * npad;
            A.fields[base + idx] = i < n ? gather_field(B.row, B.adj, spin_row<SPACE>(B, j), i) : 0;
        }
    }
    for (int j = tid; j < rpc; j += T) {
        const long long g = D.rep_off + B.r0 + j;
        A.energy[g] = B.E[B.r0 + j];
        A.best_E[g] = s_bestE[j];
        A.flips[g] += s_flips[j];
    }
    if (B.rank == 0) {
        for (int r = tid; r < R; r += T) {
            A.slot_rep[D.rep_off + r] = B.slot[r];
            A.attempts[D.rep_off + r] += s_att[r];
            A.successes[D.rep_off + r] += s_succ[r];
        }
        for (int k = tid; k < nt; k += T) A.xorder[D.rep_off + k] = s_order[k];
    }
    // the next job restages shared memory
    __syncthreads();
    }
}

// The variants for blocks of several replicas (their own object file,
// pt_engine_multi.cu: eight variants in one take two minutes to compile).
void* engine_fn_multi(int space);
#ifdef PTICM_ENGINE_MULTI
void* engine_fn_multi(int space) {
    if (space == SP_SHARED || space == SP_STATE) return (void*)pt_engine_kernel<false, false, false, SP_STATE>;
    if (space == SP_LARGE) return (void*)pt_engine_kernel<false, false, false, SP_LARGE>;
    if (space == SP_LARGE4) return (void*)pt_engine_kernel<false, false, false, SP_LARGE4>;
    return (void*)pt_engine_kernel<false, false, false, SP_ANY>;
}
#else
// --------------------------------------------------- from-scratch checks
// For every replica: fields f_i = sum_j J_ij s_j, E = sum h s + 1/2 sum s f
// and the cut sum over edges of w [s_i != s_j] (src/problem.cc:33-162),
// compared with the tracked fields and energy.  One block per replica.
__global__ void recompute_kernel(const EngineArgs A, const int32_t* rep_inst, int total_reps, int write_back,
                                 unsigned long long* mismatches, long long* E_out, long long* cut2_out) {
    const int g = blockIdx.x;
    if (g >= total_reps) return;
    const InstanceDesc D = A.desc[rep_inst[g]];
    const int r = (int)(g - D.rep_off);
    const int8_t* s = A.spins + D.spin_off + (long long)r * D.n_pad;
    int32_t* f = A.fields + D.spin_off + (long long)r * D.n_pad;
    const int32_t* row = A.row + D.row_off;
    const uint32_t* adj = A.adj + D.adj_off;
    long long e2 = 0, cut2 = 0;
    unsigned long long bad = 0;
    for (int i = threadIdx.x; i < D.n; i += blockDim.x) {
        int fi = 0;
        long long ci = 0;
        const int si = s[i];
        for (int a = row[i]; a < row[i + 1]; a++) {
            const uint32_t e = adj[a];
            const int J = (int)(int8_t)(e & 0xffu);
            const int sv = s[e >> 8];
            fi += J * sv;
            if (sv != si) ci += J;
        }
        const int hi = D.has_h ? A.hpool[D.h_off + i] : 0;
        e2 += (long long)si * (2 * hi + fi);
        cut2 += ci;
        if (si != 1 && si != -1) bad++;
        if (write_back) f[i] = fi;
        else if (f[i] != fi) bad++;
    }
    __shared__ long long red[3][32];
    for (int o = 16; o > 0; o >>= 1) {
        e2 += __shfl_xor_sync(0xffffffffu, e2, o);
        cut2 += __shfl_xor_sync(0xffffffffu, cut2, o);
        bad += __shfl_xor_sync(0xffffffffu, bad, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) { red[0][w] = e2; red[1][w] = cut2; red[2][w] = (long long)bad; }
    __syncthreads();
    if (threadIdx.x == 0) {
        long long te = 0, tc = 0, tb = 0;
        for (int k = 0; k < nw; k++) { te += red[0][k]; tc += red[1][k]; tb += red[2][k]; }
        const long long E = te / 2;
        if (write_back) A.energy[g] = E;
        else if (A.energy[g] != E) tb++;
        if (E_out) E_out[g] = E;
        if (cut2_out) cut2_out[g] = tc;
        if (mismatches) atomicAdd(mismatches, (unsigned long long)tb);
    }
}

// Bernoulli(1/2) initial spins from the Philox init stream.
__global__ void init_spins_kernel(const EngineArgs A, const int32_t* rep_inst, int total_reps,
                                  unsigned long long seed) {
    const int g = blockIdx.x;
    if (g >= total_reps) return;
    const InstanceDesc D = A.desc[rep_inst[g]];
    const int r = (int)(g - D.rep_off);
    int8_t* s = A.spins + D.spin_off + (long long)r * D.n_pad;
    const uint2 key = stream_key(seed, STREAM_INIT);
    for (int i4 = threadIdx.x; i4 * 4 < D.n_pad; i4 += blockDim.x) {
        const uint4 x = philox4x32_10(make_uint4((uint32_t)i4, (uint32_t)r, (uint32_t)D.inst_id, 0x5EEDu), key);
        const uint32_t v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int i = i4 * 4 + q;
            if (i < D.n_pad) s[i] = (i < D.n) ? (int8_t)((v[q] >> 31) ? 1 : -1) : (int8_t)1;
        }
    }
}

// States given by the caller (R x n bytes, 0/1, original site order) into
// the device order as +-1 spins: replica r's site i goes to iperm[i];
// padding sites hold +1.
__global__ void load_states_kernel(const uint8_t* src, const int32_t* iperm, int8_t* spins, int R, int n, int n_pad) {
    const long long total = (long long)R * n_pad;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(idx / n_pad), i = (int)(idx - (long long)r * n_pad);
        if (i < n) spins[(long long)r * n_pad + iperm[i]] = src[(long long)r * n + i] ? (int8_t)1 : (int8_t)-1;
        else spins[idx] = 1;
    }
}

// Replica states (0/1 bytes) and fields in the original site order (either may
// be null), from the device order: a row's reads are scattered within L2, its
// writes are lines.
__global__ void export_kernel(const int8_t* spins, const int32_t* fields, const int32_t* iperm, uint8_t* states_out,
                              int32_t* fields_out, int R, int n, int n_pad) {
    const long long total = (long long)R * n;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(idx / n), i = (int)(idx - (long long)r * n);
        const long long at = (long long)r * n_pad + iperm[i];
        if (states_out) states_out[idx] = spins[at] > 0 ? 1 : 0;
        if (fields_out) fields_out[idx] = fields[at];
    }
}

// Philox outputs for host-side known-answer checks.
__global__ void philox_probe_kernel(const uint4* ctr, const uint2* key, uint4* out, int count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) out[i] = philox4x32_10(ctr[i], key[i]);
}

// Problem::energy / maxcut / calculate_dE for a batch of states (device
// order, +-1): E, twice the cut, and dE_i = -2 s_i (h_i + f_i).
__global__ void evaluate_kernel(const int32_t* row, const uint32_t* adj, const int32_t* h, int n, int n_pad,
                                const int8_t* states, int count, long long* E_out, long long* cut2_out,
                                int32_t* dE_out) {
    const int g = blockIdx.x;
    if (g >= count) return;
    const int8_t* s = states + (long long)g * n_pad;
    long long e2 = 0, cut2 = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        int fi = 0;
        long long ci = 0;
        const int si = s[i];
        for (int a = row[i]; a < row[i + 1]; a++) {
            const uint32_t e = adj[a];
            const int J = (int)(int8_t)(e & 0xffu);
            const int sv = s[e >> 8];
            fi += J * sv;
            if (sv != si) ci += J;
        }
        const int hi = h ? h[i] : 0;
        e2 += (long long)si * (2 * hi + fi);
        cut2 += ci;
        if (dE_out) dE_out[(long long)g * n_pad + i] = -2 * si * (hi + fi);
    }
    __shared__ long long red[2][32];
    for (int o = 16; o > 0; o >>= 1) {
        e2 += __shfl_xor_sync(0xffffffffu, e2, o);
        cut2 += __shfl_xor_sync(0xffffffffu, cut2, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) { red[0][w] = e2; red[1][w] = cut2; }
    __syncthreads();
    if (threadIdx.x == 0) {
        long long te = 0, tc = 0;
        for (int k = 0; k < nw; k++) { te += red[0][k]; tc += red[1][k]; }
        E_out[g] = te / 2;
        cut2_out[g] = tc;
    }
}

// The same for states as the caller has them (0/1 bytes, original site order)
// while a state fits shared memory: its spins are placed in the device order
// there, each site gathers its neighbours' from it, and the energy changes
// leave as doubles in the original order, all device-memory accesses but the
// adjacency's whole lines.  (Reordering bytes and doubles on the host was nine
// tenths of a call: 2048 states of N=2000 with dE 20.4 ms.)
__global__ void __launch_bounds__(512) evaluate_states_kernel(const int32_t* row, const uint32_t* adj, const int32_t* h,
                                                              const int32_t* iperm, int n, const uint8_t* states, int count,
                                                              long long* E_out, long long* cut2_out, double* dE_out) {
    extern __shared__ __align__(16) uint8_t eval_sm[];
    int8_t* const s = reinterpret_cast<int8_t*>(eval_sm);
    int32_t* const dE = reinterpret_cast<int32_t*>(eval_sm + ((n + 15) & ~15));
    __shared__ long long red[2][16];
    const int tid = threadIdx.x, T = blockDim.x;
    for (int g = blockIdx.x; g < count; g += gridDim.x) {
        const uint8_t* const src = states + (long long)g * n;
        for (int i = tid; i < n; i += T) s[iperm[i]] = src[i] ? (int8_t)1 : (int8_t)-1;
        __syncthreads();
        long long e2 = 0, cut2 = 0;
        for (int i = tid; i < n; i += T) {
            const int si = s[i];
            int f = 0, w = 0;
            for_each_neighbour(row, adj, i, [&](uint32_t e) {
                const int J = (int)(int8_t)(e & 0xffu);
                f += J * s[e >> 8];
                w += J;
            });
            const int hi = h ? h[i] : 0;
            e2 += (long long)si * (2 * hi + f);
            cut2 += (w - si * f) / 2;   // the couplings to neighbours of the other sign
            if (dE_out) dE[i] = -2 * si * (hi + f);
        }
        for (int o = 16; o > 0; o >>= 1) {
            e2 += __shfl_xor_sync(0xffffffffu, e2, o);
            cut2 += __shfl_xor_sync(0xffffffffu, cut2, o);
        }
        if ((tid & 31) == 0) { red[0][tid >> 5] = e2; red[1][tid >> 5] = cut2; }
        __syncthreads();
        if (tid == 0) {
            long long te = 0, tc = 0;
            for (int k = 0; k < T >> 5; k++) { te += red[0][k]; tc += red[1][k]; }
            E_out[g] = te / 2;
            cut2_out[g] = tc;
        }
        if (dE_out)
            for (int i = tid; i < n; i += T) dE_out[(long long)g * n + i] = (double)dE[iperm[i]];
        __syncthreads();
    }
}

// ------------------------------------------------------------ launchers
static void* engine_fn(bool replay, bool block_team, bool narrow, int space) {
    if (replay) return (void*)pt_engine_kernel<true, false, false, SP_ANY>;
    if (block_team && narrow)
        return space == SP_SHARED ? (void*)pt_engine_kernel<false, true, true, SP_SHARED>
                                  : (void*)pt_engine_kernel<false, true, true, SP_ANY>;
    if (block_team) return (void*)pt_engine_kernel<false, true, false, SP_ANY>;
    return engine_fn_multi(space);
}

// The address spaces of a plan's launch.  (A staged plan of one instance
// stages that instance; a batch stages some of its instances.)
static int plan_space(const SmemPlan& S, bool block_team) {
    if (!S.state_global && !S.field_gather) return S.stage_adj && block_team ? SP_SHARED : SP_STATE;
    if (S.field_gather && S.icm_split) return S.rpc == 4 ? SP_LARGE4 : SP_LARGE;
    return SP_ANY;
}

// Tags of published energy words: one per PT step of every launch in the
// process, never 0 (a zeroed word) and never repeated within 2^32 steps.
static std::atomic<uint32_t> g_pub_tag{1u};

cudaError_t launch_engine(const EngineArgs& A0, int threads, bool replay, bool block_team, bool narrow,
                          bool cooperative, cudaStream_t stream) {
    void* fn = engine_fn(replay, block_team, narrow, plan_space(A0.sm, block_team));
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)A0.sm.total);
    if (e != cudaSuccess) return e;
    EngineArgs A = A0;
    const uint32_t span = (uint32_t)std::max(A.nsteps, 1) + 1u;
    uint32_t base = g_pub_tag.fetch_add(span);
    if (base == 0u || base + span < base) base = g_pub_tag.fetch_add(span);   // (past the wrap: 0 stays unused)
    A.pub_base = base;
    void* args[] = {(void*)&A};
    if (cooperative)
        return cudaLaunchCooperativeKernel(fn, dim3(A.n_blocks), dim3(threads), args, A.sm.total, stream);
    return cudaLaunchKernel(fn, dim3(A.n_blocks), dim3(threads), args, A.sm.total, stream);
}

// Blocks per SM of the variant that a launch with this plan takes (only that
// one is loaded: a variant costs a new process 10-20 ms).  Layouts must not
// depend on how many registers a variant came out with, so the narrow ones
// count as their bound of 128.
cudaError_t engine_max_blocks_per_sm(bool replay, bool block_team, bool narrow, int threads, const SmemPlan& S, int* out) {
    *out = 0;
    const bool bounded = !replay && (narrow || !block_team);
    if (bounded && threads > kNarrowThreads) return cudaSuccess;
    const void* fn = engine_fn(replay, block_team, narrow, plan_space(S, block_team));
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S.total);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, S.total);
    if (e != cudaSuccess) return e;
    *out = bounded ? std::min(per_sm, 65536 / (128 * ((threads + 31) & ~31))) : per_sm;
    return cudaSuccess;
}

cudaError_t launch_recompute(const EngineArgs& A, const int32_t* rep_inst, int total_reps, int write_back,
                             unsigned long long* mismatches, long long* E_out, long long* cut2_out,
                             cudaStream_t stream) {
    recompute_kernel<<<total_reps, 256, 0, stream>>>(A, rep_inst, total_reps, write_back, mismatches, E_out, cut2_out);
    return cudaGetLastError();
}

cudaError_t launch_init_spins(const EngineArgs& A, const int32_t* rep_inst, int total_reps,
                              unsigned long long seed, cudaStream_t stream) {
    init_spins_kernel<<<total_reps, 256, 0, stream>>>(A, rep_inst, total_reps, seed);
    return cudaGetLastError();
}

cudaError_t launch_load_states(const uint8_t* src, const int32_t* iperm, int8_t* spins, int R, int n, int n_pad,
                               cudaStream_t stream) {
    const long long total = (long long)R * n_pad;
    const int blocks = (int)std::min<long long>((total + 255) / 256, 4096);
    load_states_kernel<<<blocks, 256, 0, stream>>>(src, iperm, spins, R, n, n_pad);
    return cudaGetLastError();
}

cudaError_t launch_evaluate(const int32_t* row, const uint32_t* adj, const int32_t* h, int n, int n_pad,
                            const int8_t* states, int count, long long* E_out, long long* cut2_out,
                            int32_t* dE_out, cudaStream_t stream) {
    evaluate_kernel<<<count, 256, 0, stream>>>(row, adj, h, n, n_pad, states, count, E_out, cut2_out, dE_out);
    return cudaGetLastError();
}

cudaError_t launch_export(const int8_t* spins, const int32_t* fields, const int32_t* iperm, uint8_t* states_out,
                          int32_t* fields_out, int R, int n, int n_pad, cudaStream_t stream) {
    const int blocks = (int)std::min<long long>(((long long)R * n + 255) / 256, 4096);
    export_kernel<<<blocks, 256, 0, stream>>>(spins, fields, iperm, states_out, fields_out, R, n, n_pad);
    return cudaGetLastError();
}

size_t evaluate_states_smem(int n, bool with_dE) {
    return (size_t)((n + 15) & ~15) + (with_dE ? 4 * (size_t)n : 0);
}

cudaError_t launch_evaluate_states(const int32_t* row, const uint32_t* adj, const int32_t* h, const int32_t* iperm, int n,
                                   const uint8_t* states, int count, long long* E_out, long long* cut2_out,
                                   double* dE_out, cudaStream_t stream) {
    const size_t smem = evaluate_states_smem(n, dE_out != nullptr);
    const int threads = std::min(512, std::max(64, (n + 31) / 32 * 32));
    cudaError_t e = cudaFuncSetAttribute(evaluate_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    evaluate_states_kernel<<<std::min(count, 4096), threads, smem, stream>>>(row, adj, h, iperm, n, states, count, E_out,
                                                                            cut2_out, dE_out);
    return cudaGetLastError();
}

cudaError_t launch_philox_probe(const uint4* ctr, const uint2* key, uint4* out, int count, cudaStream_t stream) {
    philox_probe_kernel<<<(count + 127) / 128, 128, 0, stream>>>(ctr, key, out, count);
    return cudaGetLastError();
}

#endif  // PTICM_ENGINE_MULTI

}  // namespace pticm
