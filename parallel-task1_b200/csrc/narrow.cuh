// Narrow phases: the small phases of a query, run by one thread-block cluster.
// Included by traverse.cu inside its anonymous namespace (it uses the distance
// words, the stream loads and the schedule network from there).
//
// A phase of the persistent kernels costs some 9 us however little there is to
// do: its chain of steps goes through L2 between SMs five or six times (the
// frontier written by other SMs, the atomics that reserve room for the next
// one, the barrier's arrival and poll, the phase's counters), and on a B200 a
// line that another SM has just written takes about 1500 cycles to read, an L2
// atomic with a result about 1000.  Queries on road-like graphs are thousands of
// such phases, and every query begins with a few.  One cluster of 16 CTAs has
// what those steps need close by: the frontier and all counters live in shared
// memory and are read across the cluster (about 250 cycles), and the cluster
// barrier is hardware.  What is left of the chain is the edge load, the gather
// and the one atomic that decides.
//
// Measured on a B200: a top-down step of the 1100 x 911 grid (662 rows on
// average) 8.9 -> 3.3 us, an SSSP light round there (342 rows) 9.0 -> 4.5 us, BFS
// and SSSP from one source 47 -> 24 ms; a BFS of six steps on 1,024 vertices
// 80 -> 57 us with the call around it.  At RMAT scale 23 the step from a hub's neighbour
// (4,934 edges) takes 6 us instead of 72, because the chunk items of the hubs it
// finds, which the bottom-up step after it does not read, are not written.
//
// A query starts here and goes on in the wide kernel (bfs_persistent /
// sssp_persistent, which then also write the results back) as soon as a phase
// has too many edges, or more than a CTA's shared memory is sure to hold the
// next rows for; a query that stays narrow ends here.
//
// Rows of the frontier stay with the CTA that found them, or are dealt round
// when they are unevenly spread; 2^g lanes to a row and
// four edges to a lane at a time, with g from the mean and the longest row: the
// edges, gathers and atomics of a lane are in flight together.
#pragma once

// One CTA an SM.  512 threads: with 768 or 1024 SSSP on that grid takes 22.3 or
// 24.3 ms instead of 18.3 (the warps without a row still step through the
// phase's bookkeeping).
constexpr int kNarrowBits = 9, kNarrowThreads = 1 << kNarrowBits;
constexpr int kNarrowCtas = 16;         // CTAs of the cluster (8 where the device cannot place 16)
// Edges of the largest narrow phase.  The line is not sharp: with 16k, 64k or
// 128k the grid, a uniform graph of 1M vertices and RMAT scale 16 measure the
// same, since growing frontiers pass through this range in one step.
constexpr unsigned kNarrowEdges = 32768;
constexpr int kNarrowSeg = 128;         // longer rows are cut into segments of this many edges
constexpr int kNarrowSegs = 512;        // segments after a row's first that a CTA's queue holds
constexpr unsigned kNarrowFar = 4096;   // far-pile entries a CTA may split in a bucket opening
constexpr int kNarrowOwn = 131072;      // graphs up to this size are also initialised and written back here
enum NarrowCmd { kNarrowDone, kNarrowWide, kNarrowBudget, kNarrowPush, kNarrowPull, kNarrowHeavy, kNarrowOpen, kNarrowFlush };

// What a CTA adds in one phase.
struct alignas(16) NarrowCount {
    unsigned rows;     // rows in its queue
    unsigned segs;     // further segments of long rows
    unsigned edges;    // and their edges
    unsigned found;    // BFS: vertices found (those without out-edges have no row)
    unsigned scanned;  // edges expanded
    unsigned heavy;    // SSSP: entries added to its heavy list
    unsigned hedges;   // and their heavy edges
    unsigned far;      // vertices for the far pile
    int far_key;       // SSSP: max of 0x7fffffff - distance bits pushed to the far pile
    unsigned longest, hlongest;  // most edges of a row or segment, and of a heavy row
    unsigned pad;
};
static_assert(sizeof(NarrowCount) == 48, "read as three 16-byte words");

struct NarrowShared {
    // frontier rows of two phases (kNarrowRows at most), then the further segments
    int v[2][kNarrowRows + kNarrowSegs], begin[2][kNarrowRows + kNarrowSegs], len[2][kNarrowRows + kNarrowSegs];
    int heavy[2][kNarrowRows];               // SSSP heavy lists
    int far[2][kNarrowRows];                 // vertices for the far pile, of two phases
    NarrowCount cnt[3];                      // ring over phases: being filled, being read, clear
    unsigned first[kNarrowCtas + 1];         // rows and segments of the CTAs before each CTA
    unsigned mains[kNarrowCtas];             // rows among them
    // the phase, from the control warp
    int cmd, g, in, ring, lists, dealt;
    unsigned rows, far_len, hbase;           // hbase: entries this CTA's heavy list holds already
    int level_next;
    float thr, told;
    unsigned round, h_start, f_start;
    int hcur, fcur;
    unsigned far_n, far_at;                  // staged by this CTA in the phase before, and their place in the pile
    int far_buf, far_pile;
    // log of the phase before (written out by an idle warp)
    int log_phase, log_next, log_kind, log_dec, log_choice;  // log_phase -1: none; log_next: index of this phase
    unsigned log_size;
    unsigned long long log_scanned, log_state[5];
    float log_lo, log_hi;
    float mlp[kMlpMaxParams];
};

extern __shared__ unsigned char narrow_smem[];

__device__ __forceinline__ NarrowShared &narrow() { return *reinterpret_cast<NarrowShared *>(narrow_smem); }

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ unsigned cluster_size()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

// All threads of the cluster; orders shared and global memory between them.
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The address of p (in this CTA's shared memory) in CTA `rank`'s.
template <class T>
__device__ __forceinline__ T *on_rank(T *p, unsigned rank)
{
    unsigned long long r;
    asm volatile("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
    return reinterpret_cast<T *>(r);
}

__device__ __forceinline__ unsigned atom_or_if(unsigned *p, unsigned bit, bool on)
{
    unsigned old = 0;
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %3, 0;\n @q atom.global.or.b32 %0, [%1], %2;\n}"
                 : "+r"(old)
                 : "l"(p), "r"(bit), "r"((unsigned)on)
                 : "memory");
    return old;
}

__device__ __forceinline__ unsigned long long atom_min_if(unsigned long long *p, unsigned long long x, bool on)
{
    unsigned long long old = 0;
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %3, 0;\n @q atom.global.min.u64 %0, [%1], %2;\n}"
                 : "+l"(old)
                 : "l"(p), "l"(x), "r"((unsigned)on)
                 : "memory");
    return old;
}

// Totals of a phase over the cluster (control warp; every lane gets them).
struct NarrowTotal {
    unsigned rows, units, edges, found, scanned;  // units: rows and segments
    unsigned longest, most;                       // edges of the longest unit; units of the fullest CTA
    int far_key;
    NarrowCount rank;  // lane c: rank c's
};

__device__ __forceinline__ unsigned scan_ranks(unsigned x)
{
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned y = __shfl_up_sync(kFull, x, d);
        if ((threadIdx.x & 31u) >= (unsigned)d) x += y;
    }
    return x;
}

// Reads every CTA's counters of the phase that just ended.  (A CTA may be ahead
// and add to what the next phase fills, so nothing that a phase adds to is read
// while it runs.)
__device__ __forceinline__ NarrowTotal narrow_totals(int ring)
{
    NarrowShared &s = narrow();
    const unsigned lane = threadIdx.x & 31u, C = cluster_size();
    NarrowCount c{};
    if (lane < C) {
        const uint4 *r = reinterpret_cast<const uint4 *>(&on_rank(&s, lane)->cnt[ring]);
        uint4 *w = reinterpret_cast<uint4 *>(&c);
        w[0] = r[0];
        w[1] = r[1];
        w[2] = r[2];
    }
    c.segs = min(c.segs, (unsigned)kNarrowSegs);
    NarrowTotal t;
    t.rank = c;
    t.rows = __reduce_add_sync(kFull, c.rows);
    t.units = __reduce_add_sync(kFull, c.rows + c.segs);
    t.edges = __reduce_add_sync(kFull, c.edges);
    t.found = __reduce_add_sync(kFull, c.found);
    t.scanned = __reduce_add_sync(kFull, c.scanned);
    t.far_key = __reduce_max_sync(kFull, c.far_key);
    t.longest = __reduce_max_sync(kFull, c.longest);
    t.most = __reduce_max_sync(kFull, c.rows + c.segs);
    return t;
}

// The ranks' shares of the rows and segments a phase expands.
__device__ __forceinline__ void narrow_shares(unsigned rows, unsigned segs)
{
    NarrowShared &s = narrow();
    const unsigned lane = threadIdx.x & 31u, incl = scan_ranks(rows + segs);
    if (lane == 0) s.first[0] = 0;
    if (lane < (unsigned)kNarrowCtas) {
        s.first[lane + 1] = incl;
        s.mains[lane] = rows;
    }
}

// Whether a CTA's queues are sure to hold what a phase of `units` units of at
// most `longest` edges adds to them, beside `held` entries: each edge adds at
// most one row, one heavy entry or one far entry, and a CTA has at most its
// share of the units (dealt round, or within narrow_deal's limit).
__device__ __forceinline__ bool narrow_fits(unsigned units, unsigned edges, unsigned longest, unsigned held, unsigned C)
{
    const unsigned long long share = (unsigned long long)units / C + units / (4 * C) + 17u;
    return min((unsigned long long)edges, share * longest) + held <= (unsigned long long)kNarrowRows;
}

// A phase's units stay with the CTAs that hold them while the fullest has not
// much more than its share; otherwise they are dealt round (which reads them
// across the cluster, some 1000 cycles).
__device__ __forceinline__ bool narrow_deal(unsigned most, unsigned units, unsigned C)
{
    return most > units / C + units / (4 * C) + 16u;
}

// Lanes per unit, as a power of two: four edges a lane for units of the mean
// length, at most a warp; and more, up to a CTA's threads, while the longest unit,
// which is the phase's chain, takes more rounds than there are over the `most`
// units that 2^t threads share (a CTA's, or dealt round the cluster's).  On the
// critical path of every phase: with a formula (count of leading zeros) in place
// of the loops, which end at once on rows of four edges, the grid's SSSP took 3.5%
// longer.  Whole calls, with and without the second loop: SSSP from the hub of a
// star with 5,000 leaves, delta 0.1, 197 us and 617 (258 in the wide kernel); four
// Bellman-Ford queries on RMAT, 2,048 vertices and 8,192 edges, 353 and 750 (455).
__device__ __forceinline__ int narrow_lanes(unsigned units, unsigned edges, unsigned longest, unsigned most, int t)
{
    int g = 0;
    while (g < 5 && (edges >> (g + 2)) > units) g++;
    while (g < kNarrowBits && ((int)longest - 1 >> (g + 2)) > (int)(most << g >> t)) g++;
    return g;
}

// Rank and index of row or segment r of the phase (dealt: of all, otherwise of this CTA's).
__device__ __forceinline__ unsigned narrow_owner(unsigned r, unsigned &index, bool dealt, unsigned rank)
{
    const NarrowShared &s = narrow();
    if (!dealt) {
        index = r < s.mains[rank] ? r : r + (kNarrowRows - s.mains[rank]);
        return rank;
    }
    unsigned c = 0;
#pragma unroll
    for (unsigned d = kNarrowCtas / 2; d; d >>= 1)
        if (s.first[c + d] <= r) c += d;
    index = r - s.first[c];
    if (index >= s.mains[c]) index += kNarrowRows - s.mains[c];
    return c;
}

// Row i of queue `out`; `longest` is raised to its edges (or its segments').
__device__ __forceinline__ void narrow_put_row(int out, NarrowCount &c, unsigned i, int v, int begin, int len, unsigned &longest)
{
    NarrowShared &s = narrow();
    if (len > kNarrowSeg && len <= kNarrowRows) {
        // A long row in few lanes would be a long chain: its segments are units
        // of their own.  Where they do not fit, the row stays whole: the first
        // such row fills the segments' places left with empty ones, and none
        // after it finds room (narrow_totals counts no more than the places).
        // That takes more than 64k edges in one CTA's queue, which only a graph
        // that runs here alone goes on with.
        const int more = (len - 1) / kNarrowSeg;
        unsigned at = atomicAdd(&c.segs, (unsigned)more);
        if (at + (unsigned)more <= (unsigned)kNarrowSegs) {
            at += kNarrowRows;
            for (int k = 1; k <= more; k++, at++) {
                s.v[out][at] = v;
                s.begin[out][at] = begin + k * kNarrowSeg;
                s.len[out][at] = min(kNarrowSeg, len - k * kNarrowSeg);
            }
            len = kNarrowSeg;
        } else {
            for (; at < (unsigned)kNarrowSegs; at++) {
                s.v[out][kNarrowRows + at] = v;
                s.begin[out][kNarrowRows + at] = begin;
                s.len[out][kNarrowRows + at] = 0;
            }
        }
    }
    longest = max(longest, (unsigned)len);
    s.v[out][i] = v;
    s.begin[out][i] = begin;
    s.len[out][i] = len;
}

// Log records of the phase before and the decision for this one, by an idle warp's first lane.
__device__ __noinline__ void narrow_write_log(Ctl *ctl)
{
    const NarrowShared &s = narrow();
    if (s.log_phase >= 0) {
        const int i = s.log_phase;
        if (i < kMaxTrace) {
            ctl->ph_kind[i] = (unsigned char)s.log_kind;
            ctl->ph_size[i] = s.log_size;
            ctl->ph_end_ns[i] = globaltimer();
            ctl->ph_scanned[i] = s.log_scanned;
        }
    }
    if (s.log_dec >= 0 && s.log_dec < kMaxDec) {
        const int i = s.log_dec;
        unsigned long long *x = reinterpret_cast<unsigned long long *>(ctl->dec_x[i]);  // the features' place until the end
#pragma unroll
        for (int k = 0; k < 5; k++) x[k] = s.log_state[k];
        ctl->dec_choice[i] = (unsigned char)s.log_choice;
        ctl->dec_phase[i] = s.log_next;
        ctl->dec_lo[i] = s.log_lo;
        ctl->dec_hi[i] = s.log_hi;
    }
}

__device__ __forceinline__ bool narrow_logger()
{
    return cluster_rank() == cluster_size() - 1 && threadIdx.x == kNarrowThreads - 32;
}

// ------------------------------------------------------------------- BFS
__device__ __forceinline__ void bfs_init(const TravArgs &a, unsigned tid, unsigned nth)
{
    const int s = a.source;
    for (unsigned v = tid; v < (unsigned)a.V; v += nth) reinterpret_cast<int *>(a.value)[v] = (int)v == s ? 0 : -1;
    if (!a.color) {
        for (unsigned w = tid; w < (unsigned)a.W; w += nth) a.visited[w] = (int)w == (s >> 5) ? 1u << (s & 31) : 0u;
        return;
    }
    // vertex mask: vertices of another color start out visited, so no step
    // (top-down or bottom-up) ever reaches them; their levels stay -1
    for (unsigned w = tid >> 5; w < (unsigned)a.W; w += nth >> 5) {
        const int v = (int)(w * 32 + (threadIdx.x & 31u));
        const bool pre = v < a.V && (v == s || __ldg(&a.color[v]) != a.color_want);
        const unsigned m = __ballot_sync(kFull, pre);
        if ((threadIdx.x & 31u) == 0) a.visited[w] = m;
    }
}

__global__ void __launch_bounds__(256) bfs_init_kernel(TravArgs a)
{
    bfs_init(a, blockIdx.x * 256 + threadIdx.x, gridDim.x * 256);
}

// Hand rows over to the wide kernel (whole ones, also where the queue holds segments): short ones to its queue, longer ones as
// chunk items (written by the whole warp).  Counts go to `n`.
__device__ __forceinline__ void narrow_hand_over(const TravArgs &a, bool on, int v, int begin, int len, int32_t *q, int2 *chunks,
                                                 Ctl::Rows &n)
{
    const unsigned lane = threadIdx.x & 31u;
    const bool big = on && len > a.small_deg;
    if (on && !big && len > 0) q[atomicAdd(&n.q, 1u)] = v;
    unsigned m = __ballot_sync(kFull, big);
    if (lane == 0 && m) atomicAdd(&n.big, (unsigned)__popc(m));
    const int items = big ? (len + a.item - 1) / a.item : 0;
    unsigned at = 0;
    if (big) at = atomicAdd(&n.chunks, (unsigned)items);
    while (m) {
        const int o = __ffs(m) - 1;
        m &= m - 1;
        const int ov = __shfl_sync(kFull, v, o), ob = __shfl_sync(kFull, begin, o), on_ = __shfl_sync(kFull, items, o);
        const unsigned oa = __shfl_sync(kFull, at, o);
        for (int c = (int)lane; c < on_; c += 32) chunks[oa + c] = make_int2(ov, ob + c * a.item);
    }
}

__device__ __forceinline__ void narrow_write_back(const TravArgs &a, bool dist, unsigned tid, unsigned nth)
{
    if (!a.out) return;
    for (unsigned v = tid; v < (unsigned)a.V; v += nth) {
        const int r = __ldg(&a.new_of_old[v]);
        const unsigned x = dist ? (unsigned)(__ldcg(&a.dist[r]) >> 32) : __ldcg(&a.value[dist ? 0 : r]);
        if (a.out_kind <= 1) reinterpret_cast<unsigned *>(a.out)[v] = x;
        else reinterpret_cast<unsigned char *>(a.out)[v] = (int32_t)x >= 0 ? 1 : 0;
    }
}

// alone: the whole query runs here (small graphs); otherwise the wide kernel follows.
__global__ void __launch_bounds__(kNarrowThreads, 1) bfs_narrow(const __grid_constant__ TravArgs a, int alone)
{
    NarrowShared &s = narrow();
    const unsigned C = cluster_size(), rank = cluster_rank(), tid = threadIdx.x;
    const unsigned gtid = tid * C + rank, nth = C * kNarrowThreads;  // consecutive units go to different CTAs
    const int cluster_bits = kNarrowBits + 31 - __clz((int)C);
    Ctl *ctl = a.ctl;
    const int src = a.source;
    const bool own = a.V <= kNarrowOwn;
    if (own) bfs_init(a, rank * kNarrowThreads + tid, nth);
    if (tid == 0) {
        for (int k = 0; k < 3; k++) s.cnt[k] = NarrowCount{};
        if (rank == 0) {
            const int b = __ldg(&a.out_off[src]), d = __ldg(&a.out_off[src + 1]) - b;
            s.cnt[0].found = 1;
            s.cnt[0].edges = (unsigned)d;
            if (d > 0) {
                s.cnt[0].rows = 1;
                narrow_put_row(0, s.cnt[0], 0, src, b, d, s.cnt[0].longest);
            }
        }
    }
    cluster_sync();
    if (rank == 0 && tid == 0) ctl->t0_ns = globaltimer();
    // state of the control warp
    unsigned long long nf_prev = 0, nf = 0, mu = (unsigned long long)a.E, scanned = 0;
    int L = 0, dir = 0, bu = 0;
    for (int p = 0;; p++) {
        if (tid < 32) {
            const NarrowTotal t = narrow_totals(p % 3);
            const bool deal = narrow_deal(t.most, t.units, C);
            const int lanes = narrow_lanes(t.units, t.edges, t.longest, deal ? t.units : t.most, deal ? cluster_bits : kNarrowBits);
            narrow_shares(t.rank.rows, t.rank.segs);
            const unsigned long long done_nf = nf;
            if (p > 0) {
                nf_prev = nf;
                L++;
            }
            nf = t.found;
            mu -= t.edges;
            scanned += t.scanned;
            int plain = dir;
            if (dir == 0) {
                if ((double)t.edges * a.alpha > (double)mu) plain = 1;
            } else if (!(nf >= nf_prev || (double)nf * a.beta > (double)a.V)) {
                plain = 0;
            }
            const int d = a.force_dir >= 0 ? (L == 0 ? 0 : a.force_dir) : plain;
            int cmd = d ? kNarrowPull : kNarrowPush;
            if (nf == 0) cmd = kNarrowDone;
            else if (L >= a.max_steps) cmd = kNarrowBudget;
            else if (!alone && (d || t.edges > kNarrowEdges || !narrow_fits(t.units, t.edges, t.longest, 0, C))) cmd = kNarrowWide;
            const bool step = cmd == kNarrowPush || cmd == kNarrowPull;
            if (tid == 0) {
                s.cmd = cmd;
                s.rows = t.units;
                s.dealt = deal;
                s.g = lanes;
                s.in = p & 1;
                s.ring = (p + 1) % 3;
                s.level_next = L + 1;
                s.lists = cmd == kNarrowWide && !d;  // a bottom-up step needs none
                s.cnt[(p + 2) % 3] = NarrowCount{};
            }
            if (tid == 0 && rank == C - 1) {  // for the log
                s.log_phase = p - 1;
                s.log_next = p;
                s.log_kind = dir;
                s.log_size = (unsigned)done_nf;
                s.log_scanned = scanned;
                s.log_dec = step ? L : -1;
                s.log_choice = d;
                s.log_lo = s.log_hi = 0.0f;
                s.log_state[0] = nf;
                s.log_state[1] = t.edges;
                s.log_state[2] = mu;
                s.log_state[3] = nf_prev;
                s.log_state[4] = (unsigned long long)(unsigned)L | (unsigned long long)dir << 32 | (unsigned long long)plain << 33;
                if (step && L < kMaxTrace) {
                    ctl->dirs[L] = (unsigned char)d;
                    ctl->frontier[L] = (unsigned)nf;
                }
            }
            if (tid == 0 && rank == 0) {
                if (!step) {
                    ctl->steps = L;
                    ctl->bottom_up_steps = bu;
                    ctl->buckets = 0;
                    ctl->nphase = p;
                    ctl->ndec = L;
                    ctl->edges_scanned = scanned;
                    if (cmd == kNarrowBudget) ctl->err = kErrBudget;
                    Ctl::Resume &r = ctl->resume;
                    r.active = cmd == kNarrowWide;
                    r.wrote = own;
                    r.nf = nf;
                    r.mf = t.edges;
                    r.mu = mu;
                    r.nf_prev = nf_prev;
                    r.steps = L;
                    r.scanned = scanned;
                }
            }
            if (step) {
                dir = d;
                bu += d;
            }
        }
        __syncthreads();
        if (narrow_logger()) narrow_write_log(ctl);
        const int cmd = s.cmd, in = s.in, out = in ^ 1;
        NarrowCount &c = s.cnt[s.ring];
        unsigned edges = 0, found = 0, expanded = 0, longest = 0;
        if (cmd == kNarrowPush) {
            const bool dealt = s.dealt;
            const unsigned rows = dealt ? s.rows : s.first[rank + 1] - s.first[rank];
            const int g = s.g, sub = (int)(tid & ((1u << g) - 1u));
            const unsigned r0 = dealt ? (tid >> g) * C + rank : tid >> g, step = (kNarrowThreads >> g) * (dealt ? C : 1u);
            for (unsigned r = r0; r < rows; r += step) {
                unsigned i;
                const unsigned owner = narrow_owner(r, i, dealt, rank);
                const NarrowShared *o = dealt ? on_rank(&s, owner) : &s;
                const int len = o->len[in][i], b = o->begin[in][i], end = b + len;
                if (sub == 0) expanded += (unsigned)len;
                for (int e = b + 4 * sub; e < end; e += 4 << g) {
                    int v[4], o0[4], o1[4];
                    unsigned old[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) v[j] = e + j < end ? __ldg(&a.out_adj[e + j]) : 0;
                    // straight to the atomic: reading the word first would save
                    // atomics, but it is one more round trip
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const bool ok = e + j < end;
                        old[j] = atom_or_if(a.visited + (v[j] >> 5), 1u << (v[j] & 31), ok);
                        o0[j] = ok ? __ldg(&a.out_off[v[j]]) : 0;
                        o1[j] = ok ? __ldg(&a.out_off[v[j] + 1]) : 0;
                    }
                    unsigned rows_new = 0;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const bool fresh = e + j < end && !(old[j] >> (v[j] & 31) & 1u);
                        if (fresh) reinterpret_cast<int *>(a.value)[v[j]] = s.level_next;
                        found += fresh;
                        if (!fresh) o1[j] = o0[j];
                        rows_new += o1[j] > o0[j];
                    }
                    if (rows_new) {
                        unsigned at = atomicAdd(&c.rows, rows_new);
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            if (o1[j] <= o0[j]) continue;
                            edges += (unsigned)(o1[j] - o0[j]);
                            narrow_put_row(out, c, at++, v[j], o0[j], o1[j] - o0[j], longest);
                        }
                    }
                }
            }
        } else if (cmd == kNarrowPull) {
            // bottom-up (graphs that run here alone): every unvisited vertex
            // looks for a parent of the current level, and a long in-row that has
            // none among its first is left to the whole warp (500 dense vertices
            // beside one with 4,500 in-edges from vertices that are never reached,
            // whole call: 690 us four parents at a time by one thread, 82 us so, 172
            // us in the wide kernel; 512 vertices of 512 edges, where nearly every
            // first parent is one: four queries 131 us, and 145 with the warp at once)
            constexpr int kOwn = 32;  // parents a lane looks at in a long row
            const int level = s.level_next - 1;
            const unsigned lane = tid & 31u;
            for (unsigned v = gtid; __any_sync(kFull, v < (unsigned)a.V); v += nth) {
                const bool open = v < (unsigned)a.V && !(__ldcg(&a.visited[v >> 5]) >> (v & 31u) & 1u);
                const int b = open ? __ldg(&a.in_off[v]) : 0, end = open ? __ldg(&a.in_off[v + 1]) : 0;
                const int own = end - b > kBuCoop ? b + kOwn : end;
                bool hit = false;
                for (int e = b; e < own && !hit; e += 4) {
                    int u[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) u[j] = e + j < own ? __ldg(&a.in_adj[e + j]) : -1;
#pragma unroll
                    for (int j = 0; j < 4; j++) hit |= u[j] >= 0 && (int)__ldcg(&a.value[u[j]]) == level;
                }
                for (unsigned coop = __ballot_sync(kFull, own < end && !hit); coop; coop &= coop - 1) {
                    const int owner = __ffs(coop) - 1;
                    const int rb = __shfl_sync(kFull, own, owner), re = __shfl_sync(kFull, end, owner);
                    bool h = false;
                    for (int e = rb; e < re && !__any_sync(kFull, h); e += 128) {
                        int u[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const int k = e + 32 * j + (int)lane;
                            u[j] = k < re ? __ldg(&a.in_adj[k]) : -1;
                        }
#pragma unroll
                        for (int j = 0; j < 4; j++) h |= u[j] >= 0 && (int)__ldcg(&a.value[u[j]]) == level;
                    }
                    h = __any_sync(kFull, h);
                    if ((int)lane == owner) hit = h;
                }
                if (!hit) continue;
                reinterpret_cast<int *>(a.value)[v] = level + 1;
                atomicOr(&a.visited[v >> 5], 1u << (v & 31u));
                const int o0 = __ldg(&a.out_off[v]), o1 = __ldg(&a.out_off[v + 1]);
                found++;
                edges += (unsigned)(o1 - o0);
                if (o1 > o0) narrow_put_row(out, c, atomicAdd(&c.rows, 1u), (int)v, o0, o1 - o0, longest);
            }
        } else {
            break;
        }
        __syncwarp();
        if (__any_sync(kFull, (edges | found | expanded) != 0u)) {
            edges = __reduce_add_sync(kFull, edges);
            found = __reduce_add_sync(kFull, found);
            expanded = __reduce_add_sync(kFull, expanded);
            longest = __reduce_max_sync(kFull, longest);
            if ((tid & 31u) == 0) {
                atomicAdd(&c.edges, edges);
                atomicAdd(&c.found, found);
                atomicAdd(&c.scanned, expanded);
                atomicMax(&c.longest, longest);
            }
        }
        cluster_sync();
    }
    // over, or over to the wide kernel
    if (s.lists) {
        const unsigned mine = s.mains[rank];
        for (unsigned i0 = 0; i0 < mine; i0 += kNarrowThreads) {
            const bool on = i0 + tid < mine;
            const int v = on ? s.v[s.in][i0 + tid] : 0;
            const int b = on ? __ldg(&a.out_off[v]) : 0, e = on ? __ldg(&a.out_off[v + 1]) : 0;
            narrow_hand_over(a, on, v, b, e - b, a.q0, a.chunks0, ctl->resume.frontier);
        }
    }
    cluster_sync();  // the logs are written
    const int decisions = min((int)__ldcg(&ctl->ndec), kMaxDec);
    for (int i = (int)gtid; i < decisions; i += (int)nth) {
        unsigned long long x[5];
#pragma unroll
        for (int k = 0; k < 5; k++) x[k] = __ldcg(reinterpret_cast<unsigned long long *>(ctl->dec_x[i]) + k);
        const Feat f = bfs_features((int)(unsigned)x[4], x[0], x[1], x[2], x[3], a.V, a.E, (int)(x[4] >> 32 & 1u),
                                    (int)(x[4] >> 33 & 1u));
#pragma unroll
        for (int k = 0; k < kDecFeat; k++) ctl->dec_x[i][k] = f.x[k];
    }
    if (s.cmd == kNarrowDone && own) narrow_write_back(a, false, rank * kNarrowThreads + tid, nth);
}

// ------------------------------------------------------------------ SSSP
__device__ __forceinline__ void sssp_init(const TravArgs &a, unsigned tid, unsigned nth)
{
    for (unsigned v = tid; v < (unsigned)a.V; v += nth) {
        const unsigned cls = row_class(a, (int)v);
        a.rcls[v] = (unsigned char)cls;
        a.dist[v] = pack_dist((int)v == a.source ? 0.0f : FLT_MAX, cls);
    }
}

__global__ void __launch_bounds__(256) sssp_init_kernel(TravArgs a)
{
    sssp_init(a, blockIdx.x * 256 + threadIdx.x, gridDim.x * 256);
}

// Per-thread sums of a phase.
struct NarrowSums {
    unsigned edges, hedges, expanded, longest, hlongest;
    int far_key;
};

// What a thread adds for its N vertices v[j] at once, one reservation a list:
// bit 0 of push[j]: its light row [lb, le) joins the next frontier; bit 1: its
// heavy row (hlen edges) the heavy list hcur; bit 2: it joins the far pile.
template <int N>
__device__ __forceinline__ void narrow_add(NarrowCount &c, int out, int hcur, unsigned hbase, const int (&v)[N],
                                           const unsigned (&push)[N], const int (&lb)[N], const int (&le)[N],
                                           const int (&hlen)[N], NarrowSums &n)
{
    NarrowShared &s = narrow();
    unsigned nl = 0, nh = 0, nf = 0;
#pragma unroll
    for (int j = 0; j < N; j++) {
        nl += push[j] & 1u;
        nh += push[j] >> 1 & 1u;
        nf += push[j] >> 2;
    }
    unsigned al = 0, ah = 0, af = 0;
    if (nl) al = atomicAdd(&c.rows, nl);
    if (nh) ah = hbase + atomicAdd(&c.heavy, nh);
    if (nf) af = atomicAdd(&c.far, nf);
#pragma unroll
    for (int j = 0; j < N; j++) {
        if (push[j] & 1u) {
            n.edges += (unsigned)(le[j] - lb[j]);
            narrow_put_row(out, c, al++, v[j], lb[j], le[j] - lb[j], n.longest);
        }
        if (push[j] & 2u) {
            n.hedges += (unsigned)hlen[j];
            n.hlongest = max(n.hlongest, (unsigned)hlen[j]);
            s.heavy[hcur][ah++] = v[j];
        }
        if (push[j] & 4u) s.far[out][af++] = v[j];
    }
}

__global__ void __launch_bounds__(kNarrowThreads, 1) sssp_narrow(const __grid_constant__ TravArgs a, int alone)
{
    NarrowShared &s = narrow();
    const unsigned C = cluster_size(), rank = cluster_rank(), tid = threadIdx.x, lane = tid & 31u;
    const unsigned gtid = tid * C + rank, nth = C * kNarrowThreads;
    const int cluster_bits = kNarrowBits + 31 - __clz((int)C);
    Ctl *ctl = a.ctl;
    const int src = a.source;
    const bool own = a.V <= kNarrowOwn;
    const int32_t *const lo_off = a.nlight ? a.loff : a.out_off;  // light rows (every edge light without nlight)
    if (own) sssp_init(a, rank * kNarrowThreads + tid, nth);
    if (a.mlp)
        for (unsigned i = tid; i < (unsigned)mlp_param_count(kSsspOut); i += kNarrowThreads) s.mlp[i] = __ldg(&a.mlp[i]);
    if (tid == 0) {
        for (int k = 0; k < 3; k++) s.cnt[k] = NarrowCount{};
        if (rank == 0) {
            const int b = __ldg(&lo_off[src]), d = __ldg(&lo_off[src + 1]) - b;
            const int deg = __ldg(&a.out_off[src + 1]) - __ldg(&a.out_off[src]);
            s.cnt[0].edges = (unsigned)d;
            if (d > 0) {
                s.cnt[0].rows = 1;
                narrow_put_row(0, s.cnt[0], 0, src, b, d, s.cnt[0].longest);
            }
            if (deg > d) {
                s.cnt[0].heavy = 1;
                s.cnt[0].hedges = s.cnt[0].hlongest = (unsigned)(deg - d);
                s.heavy[0][0] = src;
            }
        }
    }
    cluster_sync();
    if (rank == 0 && tid == 0) ctl->t0_ns = globaltimer();
    // state of the control warp
    float thr = a.delta > 0.0f ? a.delta : INFINITY, lo = 0.0f;
    unsigned nheavy = 0, hedges = 0, hlongest = 0;  // lane c: entries, edges and longest row of rank c's heavy list
    unsigned far_len = 0;             // far pile in memory
    int hcur = 0, fcur = 0, steps = 0, buckets = 1, last = -1, flushes = 0, min_far = (int)kFltMaxBits;
    unsigned round = 1, h_start = 1, f_start = 1, last_size = 0;
    unsigned long long scanned = 0;
    for (int p = 0;; p++) {
        if (tid < 32) {
            const NarrowTotal t = narrow_totals(p % 3);
            nheavy += t.rank.heavy;
            hedges += t.rank.hedges;
            hlongest = max(hlongest, t.rank.hlongest);
            const unsigned heavy = __reduce_add_sync(kFull, nheavy), heavy_edges = __reduce_add_sync(kFull, hedges);
            const unsigned max_heavy = __reduce_max_sync(kFull, nheavy), heavy_longest = __reduce_max_sync(kFull, hlongest);
            scanned += t.scanned;
            const int far_bits = t.far_key > 0 ? 0x7fffffff - t.far_key : (int)kFltMaxBits;
            min_far = last == 4 ? far_bits : min(min_far, far_bits);
            // what the last phase staged for the far pile joins it after what is there
            const unsigned staged_incl = scan_ranks(t.rank.far);
            const unsigned staged = __shfl_sync(kFull, staged_incl, 31), most_staged = __reduce_max_sync(kFull, t.rank.far);
            const unsigned far_n = __shfl_sync(kFull, t.rank.far, (int)rank);
            const unsigned far_at = far_len + __shfl_sync(kFull, staged_incl, (int)rank) - far_n;
            // the next phase
            int cmd;
            unsigned size = 0;
            if (t.rows > 0) {
                cmd = kNarrowPush;
                size = t.rows;
                if (!alone && (t.edges > kNarrowEdges || !narrow_fits(t.units, t.edges, t.longest, max_heavy, C))) cmd = kNarrowWide;
            } else if (heavy > 0) {
                cmd = kNarrowHeavy;
                size = heavy;
                if (!alone && (heavy_edges > kNarrowEdges || !narrow_fits(heavy, heavy_edges, heavy_longest, 0, C))) cmd = kNarrowWide;
            } else if (far_len + staged > 0) {
                // every entry may join a CTA's queue or its next staging; where a
                // CTA would get too many, they are written out first
                cmd = kNarrowOpen;
                size = far_len + staged;
                if (!alone && far_len + staged > kNarrowFar * C) cmd = kNarrowWide;
                else if (staged > 0 && far_len / C + kNarrowThreads + most_staged > (unsigned)kNarrowRows) cmd = kNarrowFlush;
            } else {
                cmd = kNarrowDone;
            }
            if (cmd != kNarrowDone && steps + buckets >= a.max_steps) cmd = kNarrowBudget;
            const bool hv = cmd == kNarrowHeavy;
            const bool deal = narrow_deal(hv ? max_heavy : t.most, hv ? heavy : t.units, C);
            const unsigned n_units = hv ? heavy : t.units;
            const int lanes = narrow_lanes(n_units, hv ? heavy_edges : t.edges, hv ? heavy_longest : t.longest,
                                           deal ? n_units : hv ? max_heavy : t.most, deal ? cluster_bits : kNarrowBits);
            narrow_shares(hv ? nheavy : t.rank.rows, hv ? 0u : t.rank.segs);
            const unsigned mine = __shfl_sync(kFull, nheavy, (int)rank);
            if (cmd == kNarrowHeavy) nheavy = hedges = hlongest = 0;  // the list is used up; the other one starts empty
            int option = -1;
            float told = thr;
            unsigned long long st0 = 0, st1 = 0, st2 = 0;
            if (cmd == kNarrowOpen) {
                // bound = max(old, min far) + width, as in sssp_query
                option = 0;
                st0 = (unsigned long long)size | (unsigned long long)(unsigned)steps << 32;
                st1 = (unsigned long long)(unsigned)buckets;
                st2 = (unsigned long long)(unsigned)min_far | (unsigned long long)__float_as_uint(thr) << 32;
                if (a.mlp)
                    option = mlp_argmax_warp<kSsspOut>(s.mlp,
                                                       sssp_features(steps, size, __int_as_float(min_far), thr, a.delta, a.V,
                                                                     a.E, buckets, a.mean_w, a.max_deg),
                                                       0, a.mlp_margin);
                const float width = a.delta * sssp_width_scale(option);
                float hi = __fadd_rn(fmaxf(thr, __int_as_float(min_far)), width);
                if (!(hi > thr)) hi = nextafterf(thr, INFINITY);
                thr = hi;
                lo = fmaxf(told, __int_as_float(min_far));
                h_start = f_start = round;
            }
            if (cmd == kNarrowHeavy) h_start = round;
            const bool more = cmd >= kNarrowPush;
            if (tid == 0) {
                s.cmd = cmd;
                s.rows = cmd == kNarrowPush ? t.units : size;
                s.far_len = far_len;
                s.far_n = far_n;
                s.far_at = far_at;
                s.far_buf = p & 1;
                s.far_pile = fcur;
                s.hbase = cmd == kNarrowHeavy ? 0u : mine;
                s.dealt = deal;
                s.g = lanes;
                s.in = p & 1;
                s.ring = (p + 1) % 3;
                s.thr = thr;
                s.told = told;
                s.round = round;
                s.h_start = h_start;
                s.f_start = f_start;
                s.hcur = hcur;
                s.fcur = fcur;
                s.cnt[(p + 2) % 3] = NarrowCount{};
            }
            if (tid == 0 && rank == C - 1) {  // for the log
                s.log_phase = last >= 0 ? p - 1 - flushes : -1;
                s.log_next = p - flushes;
                s.log_kind = last;
                s.log_size = last_size;
                s.log_scanned = scanned;
                s.log_dec = option >= 0 ? buckets - 1 : -1;
                s.log_choice = option;
                s.log_lo = told;
                s.log_hi = thr;
                s.log_state[0] = st0;
                s.log_state[1] = st1;
                s.log_state[2] = st2;
                s.log_state[3] = s.log_state[4] = 0;
                if (cmd == kNarrowPush && steps < kMaxTrace) ctl->frontier[steps] = size;
            }
            if (tid == 0 && rank == 0) {
                if (!more) {
                    ctl->steps = steps;
                    ctl->buckets = buckets;
                    ctl->bottom_up_steps = 0;
                    ctl->nphase = p - flushes;
                    ctl->ndec = buckets - 1;
                    ctl->edges_scanned = scanned;
                    if (cmd == kNarrowBudget) ctl->err = kErrBudget;
                    Ctl::Resume &r = ctl->resume;
                    r.active = cmd == kNarrowWide;
                    r.wrote = own;
                    r.steps = steps;
                    r.buckets = buckets;
                    r.scanned = scanned;
                    r.far_len = far_len + staged;
                    r.fcur = fcur;
                    r.min_far = min_far;
                    r.thr = thr;
                    r.lo = lo;
                    r.round = round;
                    r.h_start = h_start;
                    r.f_start = f_start;
                }
            }
            far_len = cmd == kNarrowOpen ? 0 : far_len + staged;
            if (cmd == kNarrowFlush) {
                last = -1;  // no phase of the query: nothing to count or log
                flushes++;
            } else {
                last = cmd == kNarrowPush ? 3 : cmd == kNarrowHeavy ? 5 : 4;
                last_size = size;
            }
            round++;
            if (cmd == kNarrowOpen) {
                fcur ^= 1;
                buckets++;
            } else if (cmd != kNarrowFlush) {
                steps++;
                if (cmd == kNarrowHeavy) hcur ^= 1;
            }
        }
        __syncthreads();
        if (narrow_logger()) narrow_write_log(ctl);
        const int cmd = s.cmd, in = s.in, out = in ^ 1;
        NarrowCount &c = s.cnt[s.ring];
        NarrowSums n{0, 0, 0, 0, 0, 0};
        if (cmd != kNarrowOpen) {
            int32_t *pile = s.far_pile ? a.far1 : a.far0;
            for (unsigned i = tid; i < s.far_n; i += kNarrowThreads) pile[s.far_at + i] = s.far[s.far_buf][i];
        }
        if (cmd == kNarrowPush || cmd == kNarrowHeavy) {
            const bool heavy_rows = cmd == kNarrowHeavy, packed = !heavy_rows && a.nlight;
            const int hc = heavy_rows ? s.hcur ^ 1 : s.hcur;  // the heavy list that grows
            const bool dealt = s.dealt;
            const unsigned rows = dealt ? s.rows : s.first[rank + 1] - s.first[rank], round_ = s.round;
            const int g = s.g, sub = (int)(tid & ((1u << g) - 1u));
            const unsigned r0 = dealt ? (tid >> g) * C + rank : tid >> g, step = (kNarrowThreads >> g) * (dealt ? C : 1u);
            const float bound = s.thr;
            const unsigned hbase = s.hbase;
            for (unsigned r = r0; r < rows; r += step) {
                unsigned i;
                const unsigned owner = narrow_owner(r, i, dealt, rank);
                const NarrowShared *o = dealt ? on_rank(&s, owner) : &s;
                int u, b, end;
                if (heavy_rows) {
                    u = o->heavy[s.hcur][i];
                    b = __ldg(&a.out_off[u]) + __ldg(&a.nlight[u]);
                    end = __ldg(&a.out_off[u + 1]);
                } else {
                    u = o->v[in][i];
                    b = o->begin[in][i];
                    end = b + o->len[in][i];
                }
                if (sub == 0) n.expanded += (unsigned)(end - b);
                const float du = dist_of(__ldcg(&a.dist[u]));
                for (int e = b + 4 * sub; e < end; e += 4 << g) {
                    int v[4];
                    float nd[4];
                    unsigned long long cur[4], old[4];
                    int l0[4], l1[4], o0[4], o1[4];
                    bool ok[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        ok[j] = e + j < end;
                        if (packed) {
                            const int2 x = ok[j] ? __ldg(&a.ledge[e + j]) : make_int2(0, 0);
                            v[j] = x.x;
                            nd[j] = __int_as_float(x.y);
                        } else {
                            v[j] = ok[j] ? __ldg(&a.out_adj[e + j]) : 0;
                            nd[j] = ok[j] ? __ldg(&a.out_w[e + j]) : 0.0f;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) cur[j] = ok[j] ? __ldcg(&a.dist[v[j]]) : 0ull;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        nd[j] = __fadd_rn(du, nd[j]);  // one rounded add, as sssp.hpp:56
                        ok[j] = ok[j] && nd[j] < dist_of(cur[j]);
                        old[j] = atom_min_if(&a.dist[v[j]], pack_dist(nd[j], round_ << kClsBits | ((unsigned)cur[j] & kClsMask)),
                                             ok[j]);
                        l0[j] = ok[j] ? __ldg(&lo_off[v[j]]) : 0;
                        l1[j] = ok[j] ? __ldg(&lo_off[v[j] + 1]) : 0;
                        o0[j] = ok[j] ? __ldg(&a.out_off[v[j]]) : 0;
                        o1[j] = ok[j] ? __ldg(&a.out_off[v[j] + 1]) : 0;
                    }
                    unsigned push[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        // push decisions as in SsspVisit::drain
                        const float od = dist_of(old[j]);
                        const unsigned cls = (unsigned)old[j] & kClsMask, orr = (unsigned)old[j] >> kClsBits;
                        push[j] = 0;
                        if (ok[j] && nd[j] < od) {
                            if (nd[j] < bound) {
                                const bool below = od < bound;
                                push[j] = ((cls & kClsLight) && !(below && orr >= round_) ? 1u : 0u) |
                                          ((cls & kClsHeavy) && !(below && orr >= s.h_start) ? 2u : 0u);
                            } else {
                                push[j] = orr >= s.f_start ? 0u : 4u;
                                n.far_key = max(n.far_key, 0x7fffffff - __float_as_int(nd[j]));
                            }
                        }
                        o0[j] = (o1[j] - o0[j]) - (l1[j] - l0[j]);  // heavy edges
                    }
                    narrow_add(c, out, hc, hbase, v, push, l0, l1, o0, n);
                }
            }
        } else if (cmd == kNarrowOpen) {
            // the pile in memory, shared out over the cluster, and what this CTA
            // staged in the phase before
            const int32_t *fp = s.fcur ? a.far1 : a.far0;
            const unsigned share = s.far_len > gtid ? (s.far_len - gtid + nth - 1) / nth : 0u;
            const unsigned staged = s.far_n > tid ? (s.far_n - tid + kNarrowThreads - 1) / kNarrowThreads : 0u;
            for (unsigned k = 0; k < share + staged; k++) {
                const int v = k < share ? __ldcg(&fp[gtid + k * nth]) : s.far[s.far_buf][tid + (k - share) * kNarrowThreads];
                const unsigned long long dv = __ldcg(&a.dist[v]);
                const unsigned cls = (unsigned)dv & kClsMask;
                const float d = dist_of(dv);
                if (!(d >= s.told)) continue;
                // stamp the word with this round, keeping the distance
                atomicMax(&a.dist[v], pack_dist(d, s.round << kClsBits | cls));
                const bool in_bucket = d < s.thr;
                const int vs[1] = {v};
                int l0[1] = {0}, l1[1] = {0}, hl[1] = {0};
                const unsigned push[1] = {in_bucket ? (cls & kClsLight ? 1u : 0u) | (cls & kClsHeavy ? 2u : 0u) : 4u};
                if (in_bucket) {
                    l0[0] = __ldg(&lo_off[v]);
                    l1[0] = __ldg(&lo_off[v + 1]);
                    hl[0] = __ldg(&a.out_off[v + 1]) - __ldg(&a.out_off[v]) - (l1[0] - l0[0]);
                } else {
                    n.far_key = max(n.far_key, 0x7fffffff - __float_as_int(d));
                }
                narrow_add(c, out, s.hcur, s.hbase, vs, push, l0, l1, hl, n);
            }
        } else if (cmd != kNarrowFlush) {
            break;
        }
        __syncwarp();
        if (__any_sync(kFull, (n.edges | n.hedges | n.expanded | (unsigned)n.far_key) != 0u)) {
            n.edges = __reduce_add_sync(kFull, n.edges);
            n.hedges = __reduce_add_sync(kFull, n.hedges);
            n.expanded = __reduce_add_sync(kFull, n.expanded);
            n.far_key = __reduce_max_sync(kFull, n.far_key);
            n.longest = __reduce_max_sync(kFull, n.longest);
            n.hlongest = __reduce_max_sync(kFull, n.hlongest);
            if (lane == 0) {
                atomicAdd(&c.edges, n.edges);
                atomicAdd(&c.hedges, n.hedges);
                atomicAdd(&c.scanned, n.expanded);
                atomicMax(&c.far_key, n.far_key);
                atomicMax(&c.longest, n.longest);
                atomicMax(&c.hlongest, n.hlongest);
            }
        }
        cluster_sync();
    }
    // over, or over to the wide kernel
    if (s.cmd == kNarrowWide) {
        const int in = s.in, hc = s.hcur;
        const unsigned mine = s.mains[rank], nh = s.hbase;
        for (unsigned i0 = 0; i0 < mine; i0 += kNarrowThreads) {
            const bool on = i0 + tid < mine;
            const int v = on ? s.v[in][i0 + tid] : 0;
            const int b = on ? __ldg(&lo_off[v]) : 0, e = on ? __ldg(&lo_off[v + 1]) : 0;
            narrow_hand_over(a, on, v, b, e - b, a.q0, a.chunks0, ctl->resume.frontier);
        }
        for (unsigned i0 = 0; i0 < nh; i0 += kNarrowThreads) {
            const unsigned i = i0 + tid;
            const bool on = i < nh;
            const int v = on ? s.heavy[hc][i] : 0;
            const int b = on ? __ldg(&a.out_off[v]) + __ldg(&a.nlight[v]) : 0, e = on ? __ldg(&a.out_off[v + 1]) : 0;
            narrow_hand_over(a, on, v, b, e - b, a.hq0, a.hch0, ctl->resume.heavy);
        }
    }
    cluster_sync();  // the logs are written
    const int decisions = min((int)__ldcg(&ctl->ndec), kMaxDec);
    for (int i = (int)gtid; i < decisions; i += (int)nth) {
        unsigned long long x[3];
#pragma unroll
        for (int k = 0; k < 3; k++) x[k] = __ldcg(reinterpret_cast<unsigned long long *>(ctl->dec_x[i]) + k);
        const Feat f = sssp_features((int)(x[0] >> 32), (unsigned)x[0], __uint_as_float((unsigned)x[2]),
                                     __uint_as_float((unsigned)(x[2] >> 32)), a.delta, a.V, a.E, (int)x[1], a.mean_w, a.max_deg);
#pragma unroll
        for (int k = 0; k < kDecFeat; k++) ctl->dec_x[i][k] = f.x[k];
    }
    if (s.cmd == kNarrowDone && own) narrow_write_back(a, true, rank * kNarrowThreads + tid, nth);
}
