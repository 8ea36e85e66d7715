/*
 * sampler_stream.cu — the logits -> token kernel (sm_100a).
 *
 * Every logits row crosses the chip exactly once. A row is cut into slices of at most 8192 floats; the work item
 * is (row, slice); the grid is two thread blocks of 8 warps per SM, and every thread block owns a contiguous run
 * of the row-major item list. The consecutive slices of one row inside a run are a PART of that row.
 *
 *   Streaming. Every warp owns a fixed share of each slice (256 float4) and keeps its own ring of two stages
 *   full with bulk asynchronous copies (global -> this thread block's shared memory, signalled on the warp's own
 *   mbarriers): it waits for its share, applies the penalties that fall into it, lifts it into registers, asks
 *   for the share two items ahead and works on the registers. Inside a part no warp waits for another one.
 *
 *   Greedy rows keep (maximum, first id) per warp. Top-k / top-p rows keep, per thread, the maximum of its 32
 *   floats of every slice (a group) and its maximum over the part: nothing else of the select happens while the
 *   part streams. When it is through, the kq-th largest of the 256 thread maxima is a threshold that k and a few
 *   more values of the part reach; the few dozen groups that hold them are read again. Temperature rows sum
 *   e^((x - maximum) / T) per warp and slice, top-p rows per thread over the part.
 *
 *   Before any of this a row's share may pass the soft cap tanhf(x / c) * c and the mask of allowed columns,
 *   in place in the stage (head.c:145-159; only launches that carry one pay for it).
 *
 *   Part boundaries. The thread block meets and writes the part's record (maximum, first id, threshold, sums;
 *   two 16-byte slots) followed by its candidates to the part's place in global scratch. Nothing else is
 *   shared between the stream kernel's thread blocks: no counters, no thread block waits for another one.
 *
 *   Finishing is left to a kernel of its own behind the stream kernel, launched as a programmatic dependent so
 *   that its thread blocks are placed while the stream kernel drains: one thread block per row merges the parts'
 *   records; greedy rows end there; top-k rows (k <= 256) get their surviving candidates ordered, their
 *   probabilities evaluated exactly (double exp rounded once) and the draw made; temperature rows walk the
 *   per-warp segment sums and re-read the one segment that the draw falls into; top-p rows with a small nucleus
 *   are served from the candidates and the sums of the rest; wide nuclei are worked on by all thread blocks that
 *   have no row left (sampler_wide.cuh); top-k rows beyond 256 and what neither serves take a private copy of the row
 *   in global scratch (the multi-pass path; ROW_SLOW_PATH in both cases). finish_rows_kernel<false> carries all of that; finish_rows_kernel<true> carries greedy
 *   and top-k alone and is launched instead when the caller vouched for such rows (F_FAST_ONLY); with
 *   F_GREEDY_ONLY, and with F_INLINE_TOPK (whole rows per thread block, greedy and top-k rows), the stream kernel
 *   writes the tokens itself and no finishing kernel runs.
 *   Histories of more than kRowIdsMax ids are counted per row by row_ids_kernel ahead of all this.
 *
 *   The stream kernel is a template over what a launch can meet (kinds of rows vouched for, penalties at all,
 *   plain input, short histories), chosen by the host at the launch: an instantiation carries no code for the
 *   rest, and no call to an out-of-line function is left inside its slice loop.
 *
 * Semantics follow geistlib's CPU sampler:
 *   mode dispatch ............ src/archs/transformer/forward/head.c:172-183
 *   argmax ................... src/engine/sampler.c:52-62
 *   softmax / inverse CDF .... src/engine/sampler.c:68-102
 *   temperature / top-k / top-p  src/engine/sampler.c:106-132, :178-228, :232-305
 *   xorshift64* .............. src/engine/sampler.c:27-48
 *   rows of one session share one generator, in order  head.c:282-303
 * Penalties and vocabulary shards have no counterpart there; they are defined
 * in the header of include/geist_b200.h.
 */
#include <stddef.h>

#include "sampler_device.cuh"

namespace gb {

/* Optional instrumentation, compiled in with -DGB_PROFILE (and -DGB_PROFILE_CYC): PROF(i) stamps %globaltimer
 * at fixed points of a thread block's life (stream kernel 0-4, finishing kernels 5-13), MP(i) at the stages of
 * the multi-pass path, CYC(i) adds up a warp's cycles per section of the stream kernel's slice loop (0 wait for
 * data, 2 maxima or sums with the refill, 4 loop top, 5 part set-up, 6 part end with the select). The arrays are
 * read back through geist_b200_debug_*. All of it is empty otherwise. */
#ifdef GB_PROFILE
__device__ long long g_prof[1024][16];
__device__ __forceinline__ long long gtime() {
    long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
#define PROF(i)                                        \
    if (threadIdx.x == 0 && blockIdx.x < 1024) {       \
        g_prof[blockIdx.x][i] = gtime();               \
    }
#define PROF_ONCE(i)                                                       \
    if (threadIdx.x == 0 && blockIdx.x < 1024 && g_prof[blockIdx.x][i] == 0) { \
        g_prof[blockIdx.x][i] = gtime();                                   \
    }
__device__ long long g_mp[1024][24];
#define MP(i)                                          \
    if (threadIdx.x == 0 && blockIdx.x < 1024) {       \
        g_mp[blockIdx.x][i] = gtime();                 \
    }
#ifdef GB_PROFILE_CYC
__device__ long long g_cyc[1024][kWarps][8];
#define CYC_INIT()              \
    long long cyc_acc[8] = {0}; \
    long long cyc_t      = clock64()
#define CYC(i)                          \
    {                                   \
        const long long t_ = clock64(); \
        cyc_acc[i] += t_ - cyc_t;       \
        cyc_t = t_;                     \
    }
#define CYC_DONE()                                                  \
    if ((threadIdx.x & 31) == 0 && blockIdx.x < 1024) {             \
        for (int i_ = 0; i_ < 8; i_++) {                            \
            g_cyc[blockIdx.x][threadIdx.x >> 5][i_] = cyc_acc[i_];  \
        }                                                           \
    }
#else
#define CYC_INIT()
#define CYC(i)
#define CYC_DONE()
#endif
#else
#define MP(i)
#define PROF(i)
#define PROF_ONCE(i)
#define CYC_INIT()
#define CYC(i)
#define CYC_DONE()
#endif

struct PenEntry {
    int   li;
    float orig;
};

__device__ __forceinline__ float key_to_float(unsigned k) { return __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k); }


/* The threads that share a reduction: here always the whole thread block. */
struct Grp {
    int tid, lane, warp; /* position inside the group */
    int n, nw;           /* threads, warps */
    int bar;             /* unused: the group is the thread block */
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};

__device__ __forceinline__ Grp whole_block() {
    Grp g;
    g.tid  = (int) threadIdx.x;
    g.lane = g.tid & 31;
    g.warp = g.tid >> 5;
    g.n    = kThreads;
    g.nw   = kWarps;
    g.bar  = 0;
    return g;
}

/* Reduction scratch, one instance per group. */
struct __align__(16) GroupShared {
    float     wred_f[32];
    int       wred_a[32];
    double    wred_d[32];
    long long wred_l[32];
    double    S;
    float     blk_max;
    int       blk_arg;
    int       n_dlist;
    int       n_sel;
    int       b_star;
    int       n_hi;
    int       flag;
    int       pick;
};

static_assert(kSliceMax / kWarps <= 1024, "an offset in a share takes ten bits of an id list entry");
static_assert(kNV4 == 1 << kNV4Log, "the float4 of a group are named by bits");

enum Mode { M_ARGMAX, M_TOPK, M_TOPP, M_TEMP };

constexpr int ST_DEFERRED = 1 << 30; /* inside the kernel only: the one-pass finish could not serve the row (the multi-pass path has to, or the kernel lacks the code) */

/* Everything a row needs that does not depend on the slice. */
struct RowCfg {
    int                row, seq0, seq, rr;
    float              T, top_p, inv_t;
    int                top_k, k, kq;
    Mode               mode;
    bool               select_only, pen_on;
    int                H, E;
    float              rep, freq, pres;
    float              cap;  /* > 0: the row is sampled from tanhf(x / cap) * cap */
    const unsigned    *mrow; /* the sequence's mask of allowed columns, or null */
    const int         *hrow, *erow;
    unsigned long long rng; /* generator state this row starts from */
    int                draws_per_row;
};

/* The part of a row's configuration that costs memory round trips; workers
 * fetch it one item ahead. */
struct RawCfg {
    int   seq;
    float T, top_p;
    int   top_k, hist_len;
    float rep, freq, pres;
    float cap;
    unsigned long long rng; /* the sequence's generator word (only when asked for) */
};

__device__ __forceinline__ RawCfg raw_config(const SampleParams &p, int row, bool want_rng = false) {
    RawCfg    c;
    const int seq0 = p.rows_per_seq == 1 ? row : row / p.rows_per_seq;
    c.seq          = p.slot ? p.slot[seq0] : seq0;
    c.T            = p.temperature[c.seq];
    c.top_k        = p.top_k[c.seq];
    c.top_p        = p.top_p[c.seq];
    c.hist_len     = p.hist ? p.hist_len[c.seq] : 0;
    c.rep          = p.rep ? p.rep[c.seq] : 1.0f;
    c.freq         = p.freq ? p.freq[c.seq] : 0.0f;
    c.pres         = p.pres ? p.pres[c.seq] : 0.0f;
    c.cap          = p.softcap ? p.softcap[c.seq] : 0.0f;
    c.rng          = (want_rng && p.rng_in) ? p.rng_in[c.seq] : 1ull; /* travels with the other parameters */
    return c;
}

__device__ __forceinline__ RowCfg row_config(const SampleParams &p, int row, const RawCfg &c, bool want_rng) {
    RowCfg r;
    r.row   = row;
    r.seq0  = p.rows_per_seq == 1 ? row : row / p.rows_per_seq;
    r.rr    = row - r.seq0 * p.rows_per_seq;
    r.seq   = c.seq;
    r.T     = c.T;
    r.top_k = c.top_k;
    r.top_p = c.top_p;
    /* head.c:172-183 folded with the early-outs of the three sampler functions */
    if (!(r.T > 0.0f)) {
        r.mode = M_ARGMAX;
    } else if (r.top_k > 1) {
        r.mode = r.top_k >= p.V ? M_TEMP : M_TOPK;
    } else if (r.top_p > 0.0f && r.top_p < 1.0f) {
        r.mode = M_TOPP;
    } else {
        r.mode = M_TEMP;
    }
    r.select_only = (p.flags & F_SELECT_ONLY) != 0;
    r.k           = min(r.top_k, kTopKClamp);
    if (r.select_only) {
        r.mode = M_TOPK;
        r.k    = min(max(r.top_k, 1), min(p.V, kTopKClamp));
    }
    r.kq            = r.mode == M_TOPK ? r.k : (r.mode == M_TOPP ? min(kNucleusProbe, p.V) : 0);
    r.inv_t         = r.T > 0.0f ? __fdiv_rn(1.0f, r.T) : 1.0f;
    r.draws_per_row = (r.T > 0.0f && !r.select_only) ? 1 : 0;
    r.rng           = 1ull;
    if (want_rng) {
        r.rng = c.rng;
        for (int i = 0; i < r.rr * r.draws_per_row; i++) {
            (void) xorshift_next(r.rng);
        }
    }
    r.pen_on = p.hist != nullptr || p.extra != nullptr;
    r.H      = p.hist ? (int) min((long long) max(c.hist_len, 0), p.hist_stride) : 0;
    r.E      = p.extra ? r.rr : 0; /* proposals fed before this row: extra[1..rr] */
    r.rep    = c.rep > 0.0f ? c.rep : 1.0f;
    r.freq   = c.freq;
    r.pres   = c.pres;
    /* head.c:145-159: the cap is skipped for greedy rows (monotone, the argmax is the same) */
    r.cap    = (c.cap > 0.0f && r.T > 0.0f) ? c.cap : 0.0f;
    r.mrow   = p.mask ? p.mask + (size_t) r.seq * (size_t) p.mask_stride : nullptr;
    r.hrow   = p.hist ? p.hist + (size_t) r.seq * (size_t) p.hist_stride : nullptr;
    r.erow   = p.extra ? p.extra + (size_t) r.seq0 * (size_t) p.extra_stride : nullptr; /* per call, not per slot */
    return r;
}

__device__ __forceinline__ int hist_id(const RowCfg &r, int j, int vocab_offset) {
    return (j < r.H ? r.hrow[j] : r.erow[1 + j - r.H]) - vocab_offset;
}

/* What happens to a logit before the penalties: the final-logit soft cap in the reference's own expression
 * (head.c:154, :286), then the mask of allowed columns (bit i of the sequence's mask row: column i may be
 * sampled; a masked column reads as -inf). `i` is the column inside this call's logits. */
__device__ __forceinline__ float soft_cap(float x, float c) {
    return __fmul_rn(tanhf(__fdiv_rn(x, c)), c);
}
__device__ __forceinline__ float prologue_one(float x, int i, float cap, const unsigned *mrow) {
    if (cap > 0.0f) {
        x = soft_cap(x, cap);
    }
    if (mrow != nullptr && ((mrow[i >> 5] >> (i & 31)) & 1u) == 0u) {
        x = -CUDART_INF_F;
    }
    return x;
}

/* The mask words of a warp's share of a slice, at most 1024 columns: a word per lane, and the one behind them where the share
 * begins inside a word. Asked for a slice ahead: read where they were used, every slice waited for them. */
struct ShareMask {
    unsigned w, x;
};
__device__ __forceinline__ ShareMask share_mask(const unsigned *mrow, int V, int lane, int column) {
    ShareMask m;
    const int at = column >> 5, words = (V + 31) >> 5;
    m.w          = at + lane < words ? __ldg(mrow + at + lane) : 0u;
    m.x          = (column & 31) != 0 && at + 32 < words ? __ldg(mrow + at + 32) : 0u;
    return m;
}

/* The same over a warp's share of a slice in its stage (sl: the share's first float; e0: its index inside the
 * slice; mine4 float4 groups, lane-strided; n: the slice's length, what lies behind it stays -inf). Kept out of
 * line: the stream kernel's loop stays short for the launches that have neither cap nor mask. */
__device__ __noinline__ void prologue_share(float *sl, int lane, int mine4, int e0, int n, int s0, float cap, bool masked, const ShareMask &words) {
    float4  *w4 = reinterpret_cast<float4 *>(sl) + lane;
    unsigned allowed[kNV4]; /* four columns each: a float4 lies on a multiple of four, so inside one word of the mask */
    if (masked) {
#pragma unroll
        for (int i = 0; i < kNV4; i++) {
            const int      at = ((s0 + e0) & 31) + 4 * (lane + 32 * i);
            const unsigned in = __shfl_sync(0xffffffffu, words.w, (at >> 5) & 31);
            allowed[i]        = ((at >> 5) < 32 ? in : words.x) >> (at & 31);
        }
    }
#pragma unroll
    for (int i = 0; i < kNV4; i++) {
        if (lane + 32 * i < mine4) {
            const int e = e0 + 4 * (lane + 32 * i);
            float4    v = w4[32 * i];
            if (cap > 0.0f) {
                if (e + 0 < n) v.x = soft_cap(v.x, cap);
                if (e + 1 < n) v.y = soft_cap(v.y, cap);
                if (e + 2 < n) v.z = soft_cap(v.z, cap);
                if (e + 3 < n) v.w = soft_cap(v.w, cap);
            }
            if (masked) { /* what lies behind the row's end is -inf already */
                v.x = (allowed[i] & 1u) != 0u ? v.x : -CUDART_INF_F;
                v.y = (allowed[i] & 2u) != 0u ? v.y : -CUDART_INF_F;
                v.z = (allowed[i] & 4u) != 0u ? v.z : -CUDART_INF_F;
                v.w = (allowed[i] & 8u) != 0u ? v.w : -CUDART_INF_F;
            }
            w4[32 * i] = v;
        }
    }
    __syncwarp();
}

/* The same with the division by rep done as a double product with 1 / rep (rounded to double once per part): the
 * float nearest to x * rcp is the correctly rounded x / rep for every pair of floats (a quotient of two 24-bit
 * numbers is at least 2^-49 of itself away from every midpoint of two floats, the product's error is below 2^-52),
 * and the slice loop keeps clear of the division's out-of-line slow path: a call inside that loop costs every
 * slice. */
__device__ __forceinline__ float penalise_rcp(float x, int cnt, double rcp, float rep, float freq, float pres) {
    x = x > 0.0f ? __double2float_rn(__dmul_rn((double) x, rcp)) : __fmul_rn(x, rep);
    x = __fsub_rn(x, __fmul_rn((float) cnt, freq));
    return __fsub_rn(x, pres);
}

__device__ __forceinline__ float penalise(float x, int cnt, float rep, float freq, float pres) {
    x = x > 0.0f ? __fdiv_rn(x, rep) : __fmul_rn(x, rep);
    x = __fsub_rn(x, __fmul_rn((float) cnt, freq));
    return __fsub_rn(x, pres);
}

/*
 * Penalties on a run of n values that hold the global ids [s0, s0 + n). `buf`
 * may be shared or global memory; `bitmap` has (n + 31) / 32 zeroed words;
 * `dlist` has room for `cap` distinct ids; *n_dlist is zero. `first_id` is the
 * caller's pre-fetched history id for j = g.tid (or any value when the caller
 * did not prefetch: have_first = false). All threads of the group call this.
 * Returns status bits.
 */
__device__ int apply_penalties(const Grp &g, float *buf, int s0, int n, const RowCfg &r, int V, int vocab_offset, unsigned *bitmap, PenEntry *dlist, int cap, int *n_dlist,
                               bool have_first, int first_id) {
    int       st    = 0;
    const int total = r.H + r.E;
    auto      id_at = [&](int j) { return (have_first && j == g.tid) ? first_id : hist_id(r, j, vocab_offset); };
    if (r.freq == 0.0f) {
        /* multiplicities do not matter: the first thread to mark an id rewrites it, one pass */
        for (int j = g.tid; j < total; j += g.n) {
            const int id = id_at(j);
            const int li = id - s0;
            if (id >= 0 && id < V && li >= 0 && li < n) {
                const unsigned bit = 1u << (li & 31);
                if (!(atomicOr(&bitmap[li >> 5], bit) & bit)) {
                    buf[li] = penalise(buf[li], 1, r.rep, 0.0f, r.pres);
                }
            }
        }
        g.sync();
        return st;
    }
    /* (a) the first thread to mark an id owns it and saves the original value */
    for (int j = g.tid; j < total; j += g.n) {
        const int id = id_at(j);
        const int li = id - s0;
        if (id >= 0 && id < V && li >= 0 && li < n) {
            const unsigned bit = 1u << (li & 31);
            if (!(atomicOr(&bitmap[li >> 5], bit) & bit)) {
                const int pos = atomicAdd(n_dlist, 1);
                if (pos < cap) {
                    dlist[pos].li   = li;
                    dlist[pos].orig = buf[li];
                }
            }
        }
    }
    g.sync();
    int nd = *n_dlist;
    if (nd > cap) { /* cannot happen: the callers have room for an entry per value of the run, or per id; keep the run consistent anyway */
        st |= ST_HIST_OVERFLOW;
        nd = 0;
    }
    /* (b) the slot becomes an integer counter */
    for (int i = g.tid; i < nd; i += g.n) {
        reinterpret_cast<int *>(buf)[dlist[i].li] = 0;
    }
    g.sync();
    if (nd > 0) {
        for (int j = g.tid; j < total; j += g.n) {
            const int id = id_at(j);
            const int li = id - s0;
            if (id >= 0 && id < V && li >= 0 && li < n) {
                atomicAdd(reinterpret_cast<int *>(buf) + li, 1);
            }
        }
    }
    g.sync();
    /* (c) one thread per distinct id writes the penalised value */
    for (int i = g.tid; i < nd; i += g.n) {
        const int li = dlist[i].li;
        buf[li]      = penalise(dlist[i].orig, reinterpret_cast<int *>(buf)[li], r.rep, r.freq, r.pres);
    }
    g.sync();
    return st;
}

/* ------------------------------------------------------- sums over a row -- */

/* The sums of temperature and top-p rows are formed of 2^((x - ref) * scale), ref a value of the row and scale =
 * log2(e) / T in two floats (their sum is good to 2^-48): the difference comes first, so a term's argument is rounded at
 * its own size, whatever the sizes of x and T. The high float is rounded down, both are at least the
 * smallest float and the low one is finite, so that an x of -inf (which pads a row) gives 0 and the x that is ref gives
 * 1 at every T whose inverse is finite. */
__device__ __forceinline__ double sum_scale(float inv_t) { return (double) inv_t * 1.4426950408889634; }
struct SumScale {
    float hi, lo;
};
__device__ __forceinline__ SumScale sum_scale2(float inv_t) {
    SumScale k;
    const float hi = __double2float_rz(sum_scale(inv_t));
    k.hi           = fmaxf(hi, 0x1p-149f);
    k.lo           = fminf(fmaxf(__double2float_rn(sum_scale(inv_t) - (double) hi), 0x1p-149f), 3.4028235e38f);
    return k;
}
__device__ __forceinline__ float sum_term(float x, const SumScale &k, float ref) {
    const float d = __fsub_rn(x, ref);
    return exp2_fast(__fmaf_rn(d, k.lo, __fmul_rn(d, k.hi)));
}
/* what a sum relative to `from` is multiplied with to be relative to `to`; nothing has been summed relative to -inf */
__device__ __forceinline__ double ref_move(float from, float to, float inv_t) {
    return from == -CUDART_INF_F ? 0.0 : exp(((double) from - (double) to) * (double) inv_t);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

/* ------------------------------------------------------- group reductions -- */

/* (max, first id) over the group; every thread gets the result. */
__device__ __forceinline__ void group_argmax(const Grp &g, GroupShared *sh, float &v, int &a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int   oa = __shfl_xor_sync(0xffffffffu, a, o);
        if (pair_before(ov, oa, v, a)) {
            v = ov;
            a = oa;
        }
    }
    g.sync(); /* earlier readers of the scratch are done */
    if (g.lane == 0) {
        sh->wred_f[g.warp] = v;
        sh->wred_a[g.warp] = a;
    }
    g.sync();
    if (g.warp == 0) {
        v = g.lane < g.nw ? sh->wred_f[g.lane] : -CUDART_INF_F;
        a = g.lane < g.nw ? sh->wred_a[g.lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int   oa = __shfl_xor_sync(0xffffffffu, a, o);
            if (pair_before(ov, oa, v, a)) {
                v = ov;
                a = oa;
            }
        }
        if (g.lane == 0) {
            sh->blk_max = v;
            sh->blk_arg = a;
        }
    }
    g.sync();
    v = sh->blk_max;
    a = sh->blk_arg;
}

/* Every thread gets the same total (fixed order of additions). */
__device__ __forceinline__ double group_sum_d(const Grp &g, GroupShared *sh, double v) {
    v = warp_sum_d(v);
    g.sync(); /* the previous result has been read */
    if (g.lane == 0) {
        sh->wred_d[g.warp] = v;
    }
    g.sync();
    double t = 0.0;
    for (int w = 0; w < g.nw; w++) {
        t += sh->wred_d[w];
    }
    return t;
}

__device__ __forceinline__ long long group_sum_ll(const Grp &g, GroupShared *sh, long long v) {
    v = warp_sum_ll(v);
    g.sync();
    if (g.lane == 0) {
        sh->wred_l[g.warp] = v;
    }
    g.sync();
    long long t = 0;
    for (int w = 0; w < g.nw; w++) {
        t += sh->wred_l[w];
    }
    return t;
}

/* ------------------------------------------------------------ multi-pass path -- */

template <class F>
__device__ __forceinline__ void row_sweep(const Grp &g, const float *row, int V, F &&f) {
    const int     V4 = V >> 2;
    const float4 *p4 = reinterpret_cast<const float4 *>(row);
    int           j  = g.tid;
    for (; j + 7 * g.n < V4; j += 8 * g.n) { /* eight loads in flight per thread */
        float4 v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            v[q] = p4[j + q * g.n];
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int b = 4 * (j + q * g.n);
            f(v[q].x, b), f(v[q].y, b + 1), f(v[q].z, b + 2), f(v[q].w, b + 3);
        }
    }
    for (; j < V4; j += g.n) {
        const float4 x = p4[j];
        f(x.x, 4 * j);
        f(x.y, 4 * j + 1);
        f(x.z, 4 * j + 2);
        f(x.w, 4 * j + 3);
    }
    for (int i = (V4 << 2) + g.tid; i < V; i += g.n) {
        f(row[i], i);
    }
}

template <class F>
__device__ __forceinline__ void row_rewrite(const Grp &g, float *row, int V, F &&f) {
    /* private copies start on 16-byte boundaries: four values per access, four accesses in flight per thread */
    const int V4 = V >> 2;
    float4   *p4 = reinterpret_cast<float4 *>(row);
    int       j  = g.tid;
    for (; j + 3 * g.n < V4; j += 4 * g.n) {
        float4 a = p4[j], b = p4[j + g.n], c = p4[j + 2 * g.n], d = p4[j + 3 * g.n];
        a.x = f(a.x, 4 * j), a.y = f(a.y, 4 * j + 1), a.z = f(a.z, 4 * j + 2), a.w = f(a.w, 4 * j + 3);
        p4[j] = a;
        b.x = f(b.x, 4 * (j + g.n)), b.y = f(b.y, 4 * (j + g.n) + 1), b.z = f(b.z, 4 * (j + g.n) + 2), b.w = f(b.w, 4 * (j + g.n) + 3);
        p4[j + g.n] = b;
        c.x = f(c.x, 4 * (j + 2 * g.n)), c.y = f(c.y, 4 * (j + 2 * g.n) + 1), c.z = f(c.z, 4 * (j + 2 * g.n) + 2), c.w = f(c.w, 4 * (j + 2 * g.n) + 3);
        p4[j + 2 * g.n] = c;
        d.x = f(d.x, 4 * (j + 3 * g.n)), d.y = f(d.y, 4 * (j + 3 * g.n) + 1), d.z = f(d.z, 4 * (j + 3 * g.n) + 2), d.w = f(d.w, 4 * (j + 3 * g.n) + 3);
        p4[j + 3 * g.n] = d;
    }
    for (; j < V4; j += g.n) {
        float4 x = p4[j];
        x.x = f(x.x, 4 * j), x.y = f(x.y, 4 * j + 1), x.z = f(x.z, 4 * j + 2), x.w = f(x.w, 4 * j + 3);
        p4[j] = x;
    }
    for (int i = (V4 << 2) + g.tid; i < V; i += g.n) {
        row[i] = f(row[i], i);
    }
}

/* out[i] = f(in[i], i): both rows on 16-byte boundaries (in may be out). */
template <class F>
__device__ __forceinline__ void row_map(const Grp &g, const float *in, float *out, int V, F &&f) {
    const int     V4 = V >> 2;
    const float4 *i4 = reinterpret_cast<const float4 *>(in);
    float4       *o4 = reinterpret_cast<float4 *>(out);
    int           j  = g.tid;
    for (; j + 3 * g.n < V4; j += 4 * g.n) {
        float4 v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[q] = i4[j + q * g.n];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int b = 4 * (j + q * g.n);
            v[q].x = f(v[q].x, b), v[q].y = f(v[q].y, b + 1), v[q].z = f(v[q].z, b + 2), v[q].w = f(v[q].w, b + 3);
            o4[j + q * g.n] = v[q];
        }
    }
    for (; j < V4; j += g.n) {
        float4 x = i4[j];
        x.x = f(x.x, 4 * j), x.y = f(x.y, 4 * j + 1), x.z = f(x.z, 4 * j + 2), x.w = f(x.w, 4 * j + 3);
        o4[j] = x;
    }
    for (int i = (V4 << 2) + g.tid; i < V; i += g.n) {
        out[i] = f(in[i], i);
    }
}

/* A walk is written against "something that calls f(value, id) for every entry": the whole private copy of a
 * row, or a short list of (value, id) pairs picked out of it. */
template <class F>
__device__ __forceinline__ void list_sweep(const Grp &g, const Pair *list, int n, F &&f) {
    int j = g.tid;
    for (; j + 3 * g.n < n; j += 4 * g.n) {
        const Pair a = list[j], b = list[j + g.n], c = list[j + 2 * g.n], d = list[j + 3 * g.n];
        f(a.v, a.idx), f(b.v, b.idx), f(c.v, c.idx), f(d.v, d.idx);
    }
    for (; j < n; j += g.n) {
        const Pair a = list[j];
        f(a.v, a.idx);
    }
}

/* Largest composite word t with mass{word >= t} >= target (inclusive) or > target. The search may
 * start from a known prefix of the word: the bits above top_bit are taken from `prefix`. */
template <class Sweep, class KeyF, class MassF>
__device__ unsigned long long bisect_mass(const Grp &g, GroupShared *sh, Sweep &&sweep, int idx_bits, double target, bool inclusive, KeyF &&key, MassF &&mass,
                                          unsigned long long prefix = 0ull, int top_bit = -1) {
    for (int bit = top_bit >= 0 ? top_bit : 31 + idx_bits; bit >= 0; bit--) {
        const unsigned long long t = prefix | (1ull << bit);
        double                   m = 0.0;
        sweep([&](float x, int i) {
            if (composite(key(x), i, idx_bits) >= t) {
                m += mass(x, i);
            }
        });
        const double tot = group_sum_d(g, sh, m);
        if (inclusive ? (tot >= target) : (tot > target)) {
            prefix = t;
        }
    }
    return prefix;
}

/* Where a walk over the row in descending key order first reaches a target mass. */
struct RadixOut {
    bool      found;  /* false: the whole row stays below the target */
    unsigned  key;    /* the key at which the running mass crosses */
    double    above;  /* mass of the entries with a larger key */
    long long n_above; /* how many those are */
    long long ties;   /* entries with exactly this key (and mass > 0) */
};

/*
 * The same answer as the top 32 bits of bisect_mass, in four sweeps instead of thirty-two: one
 * byte of the key per sweep, masses and counts per byte value in shared memory (`copies` private
 * histograms, one per warp where the room allows), then a scan from the top value down. hm / hc
 * hold copies * 256 doubles / ints.
 */
template <bool kUnit = false, class Sweep, class KeyF, class MassF>
__device__ RadixOut radix_mass(const Grp &g, GroupShared *sh, double *hm, int *hc, int copies, double scale, Sweep &&sweep, double target, bool inclusive, KeyF &&key,
                               MassF &&mass, int last_level = 0, bool top_filled = false) {
    /* masses are summed as 64-bit fixed point (mass * scale, truncated): integer adds in shared memory are one
     * instruction whatever the conflicts, and the sums do not depend on the order. The caller picks a scale that
     * keeps the row's total below 2^63. */
    unsigned long long *hq = reinterpret_cast<unsigned long long *>(hm);
    RadixOut out;
    out.found   = true;
    out.key     = 0u;
    out.above   = 0.0;
    out.n_above = 0;
    out.ties    = 0;
    for (int level = 3; level >= last_level; level--) { /* last_level 3: the top byte alone; the histograms then stay as they are for the caller */
        const int shift = 8 * level;
        if (!(top_filled && level == 3)) { /* top_filled: the caller binned the top byte itself while it had the entries in hand */
        for (int i = g.tid; i < copies * 256; i += g.n) {
            hq[i] = 0ull;
            hc[i] = 0;
        }
        g.sync();
        unsigned long long *mym = hq + (g.warp % copies) * 256;
        int           *myc = hc + (g.warp % copies) * 256;
        const unsigned pre = out.key;
        sweep([&](float x, int i) {
            const unsigned k = key(x);
            if (level == 3 || (k >> (shift + 8)) == (pre >> (shift + 8))) {
                const unsigned d = (k >> shift) & 255u;
                if (kUnit) { /* every entry weighs one: the counts are the masses */
                    atomicAdd(&myc[d], 1);
                } else {
                    const double m = mass(x, i);
                    if (m > 0.0) {
                        atomicAdd(&mym[d], __double2ull_rz(m * scale));
                        atomicAdd(&myc[d], 1);
                    }
                }
            }
        });
        }
        g.sync();
        if (g.warp == 0) {
            /* lane l owns the byte values 255 - 8 l down to 248 - 8 l: the walk order */
            double m8[8];
            int    c8[8];
            double lane_m = 0.0;
            int    lane_c = 0;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int b = 255 - (8 * g.lane + q);
                unsigned long long q8 = 0ull;
                c8[q]                 = 0;
                for (int w = 0; w < copies; w++) {
                    q8 += hq[w * 256 + b];
                    c8[q] += hc[w * 256 + b];
                }
                m8[q] = kUnit ? (double) c8[q] : (double) q8 / scale;
                lane_m += m8[q];
                lane_c += c8[q];
            }
            double incl_m = lane_m;
            int    incl_c = lane_c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double um = __shfl_up_sync(0xffffffffu, incl_m, o);
                const int    uc = __shfl_up_sync(0xffffffffu, incl_c, o);
                if (g.lane >= o) {
                    incl_m += um;
                    incl_c += uc;
                }
            }
            const double   before = out.above + (incl_m - lane_m);
            const bool     cross  = inclusive ? (before + lane_m >= target) : (before + lane_m > target);
            const unsigned ball   = __ballot_sync(0xffffffffu, cross);
            if (ball == 0u) {
                if (g.lane == 0) {
                    sh->b_star = -1;
                }
            } else if (g.lane == __ffs(ball) - 1) {
                double run = before;
                int    cnt = incl_c - lane_c;
                int    b   = 255 - 8 * g.lane - 7;
                int    tc  = c8[7];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const bool hit = inclusive ? (run + m8[q] >= target) : (run + m8[q] > target);
                    if (hit) {
                        b  = 255 - (8 * g.lane + q);
                        tc = c8[q];
                        break;
                    }
                    run += m8[q];
                    cnt += c8[q];
                }
                sh->b_star = b;
                sh->S      = run;
                sh->n_hi   = cnt;
                sh->n_sel  = tc;
            }
        }
        g.sync();
        if (sh->b_star < 0) {
            out.found = false;
            g.sync();
            return out;
        }
        out.key |= (unsigned) sh->b_star << shift;
        out.above = sh->S;
        out.n_above += (long long) sh->n_hi;
        out.ties = (long long) sh->n_sel;
        g.sync();
    }
    return out;
}

/*
 * From the key at which a walk crosses to the composite word of the crossing entry: entries with
 * equal keys are walked by ascending id, and `j` of them (1-based) are needed. One of a kind: one
 * sweep finds its id. Several: the low bits of the word are bisected as before.
 */
template <class Sweep, class KeyF, class MassF>
__device__ unsigned long long resolve_ties(const Grp &g, GroupShared *sh, Sweep &&sweep, int idx_bits, const RadixOut &ro, double target, bool inclusive, KeyF &&key,
                                           MassF &&mass) {
    if (ro.ties <= 1) {
        if (g.tid == 0) {
            sh->pick = 0x7fffffff;
        }
        g.sync();
        sweep([&](float x, int i) {
            if (key(x) == ro.key && mass(x, i) > 0.0) {
                atomicMin(&sh->pick, i);
            }
        });
        g.sync();
        const int id = sh->pick;
        g.sync();
        return composite(ro.key, id == 0x7fffffff ? 0 : id, idx_bits);
    }
    return bisect_mass(g, sh, sweep, idx_bits, target, inclusive, key, mass, (unsigned long long) ro.key << idx_bits, idx_bits - 1);
}

/* Where a row is read again once it has been streamed, and whether it starts on a 16-byte boundary there. A launch that
 * asks for the rows as they are sampled from reads those back and changes nothing a second time: they may lie over the
 * logits themselves. */
__device__ __forceinline__ const float *row_again(const SampleParams &p, int row) {
    return p.out_logits != nullptr ? p.out_logits + (size_t) row * (size_t) p.V : p.logits + (size_t) row * (size_t) p.row_stride;
}
__device__ __forceinline__ bool again_aligned(const SampleParams &p) {
    return p.out_logits != nullptr ? (reinterpret_cast<unsigned long long>(p.out_logits) & 15ull) == 0ull && (p.V & 3) == 0 : p.aligned != 0;
}

/* All threads of the thread block serve a row whose kept set does not fit the one-pass path. The row's configuration comes
 * in shared memory: handed on by reference it, and the group, would lie in the callers' frames. */
__device__ __noinline__ int multipass_row(const SampleParams &p, GroupShared *sh, const RowCfg *cfg, float row_max, int row_arg, void *hist_mem, int hist_bytes, int slot, void *save_mem) {
    const Grp g = whole_block();
    RowCfg    r = *cfg;
    /* room for the byte histograms of the radix walks: per warp where it fits, else one for all */
    const int copies = hist_bytes >= g.nw * 256 * 12 ? g.nw : 1;
    double   *hm     = reinterpret_cast<double *>(hist_mem);
    int      *hc     = reinterpret_cast<int *>(hm + copies * 256);
    const int    V        = p.V;
    const int    idx_bits = 32 - __clz(max(V - 1, 1));
    int          st       = ST_SLOW_PATH;
    float       *gr       = p.gen_rows + (size_t) slot * (size_t) p.gen_stride;
    const float *src      = row_again(p, r.row);
    const bool   src_al   = again_aligned(p);
    int         *kept_i   = p.kept_cap > 0 ? p.kept_idx + (size_t) r.row * (size_t) p.kept_cap : nullptr;
    float       *kept_v   = p.kept_cap > 0 ? p.kept_val + (size_t) r.row * (size_t) p.kept_cap : nullptr;
    /* Nothing changes the row's values (no penalties, cap or mask) and it lies on a 16-byte boundary: it is read
     * where it is, and the private copy only takes what a top-p row is rewritten into. */
    const bool   in_place = !r.pen_on && !(r.cap > 0.0f) && r.mrow == nullptr && src_al;
    const float *cur      = in_place ? src : gr; /* what the sweeps read */
    auto         row_sw   = [&](auto &&f) { row_sweep(g, cur, V, f); };
    /* the entries that pred(value, id) names, picked out of the row into this thread block's list (any order);
     * every thread gets their number, which may exceed the list's room: the caller checks */
    Pair *list     = p.gen_list + (size_t) slot * (size_t) p.gen_list_cap;
    auto  pick_out = [&](auto &&pred) {
        if (g.tid == 0) {
            sh->n_sel = 0;
        }
        g.sync();
        row_sweep(g, cur, V, [&](float x, int i) {
            if (pred(x, i)) {
                const int pos = atomicAdd(&sh->n_sel, 1);
                if (pos < p.gen_list_cap) {
                    list[pos].v   = x;
                    list[pos].idx = i;
                }
            }
        });
        __threadfence_block();
        g.sync();
        const int n = sh->n_sel;
        g.sync();
        return n;
    };
    MP(0);
    /* private copy of the row, penalties applied once */
    if (in_place) {
    } else if (src_al) { /* rows start on 16-byte boundaries: four values per load */
        const float4 *s4 = reinterpret_cast<const float4 *>(src);
        float4       *d4 = reinterpret_cast<float4 *>(gr);
        for (int i = g.tid; i < (V >> 2); i += g.n) {
            d4[i] = s4[i];
        }
        for (int i = (V & ~3) + g.tid; i < V; i += g.n) {
            gr[i] = src[i];
        }
    } else {
        for (int i = g.tid; i < V; i += g.n) {
            gr[i] = src[i];
        }
    }
    if (r.cap > 0.0f || r.mrow != nullptr) {
        g.sync();
        const float     cap  = r.cap;
        const unsigned *mrow = r.mrow;
        row_rewrite(g, gr, V, [&](float x, int i) { return prologue_one(x, i, cap, mrow); });
    }
    if (r.pen_on) {
        unsigned *bm = p.gen_bitmap + (size_t) slot * (size_t) p.gen_bitmap_words;
        for (int i = g.tid; i < p.gen_bitmap_words; i += g.n) {
            bm[i] = 0u;
        }
        if (g.tid == 0) {
            sh->n_dlist = 0;
        }
        g.sync();
        st |= apply_penalties(g, gr, 0, V, r, V, p.vocab_offset, bm, reinterpret_cast<PenEntry *>(p.gen_dlist + (size_t) slot * (size_t) p.gen_hist_cap), p.gen_hist_cap,
                              &sh->n_dlist, false, 0);
    } else {
        g.sync();
    }
    MP(1);
    /* the fast path's slice records need not carry the maximum: take it from the copy */
    row_max = -CUDART_INF_F;
    row_arg = 0x7fffffff;
    row_sweep(g, cur, V, [&](float x, int i) {
        if (row_arg == 0x7fffffff || pair_before(x, i, row_max, row_arg)) {
            row_max = x;
            row_arg = i;
        }
    });
    group_argmax(g, sh, row_max, row_arg);
    MP(2);
    if (r.mode == M_TOPK) {
        /* the k-th entry in (value desc, id asc) order: a radix walk on counts, then the ids of its ties */
        auto                     okey   = [](float x) { return order_key(x); };
        auto                     one    = [](float, int) { return 1.0; };
        /* The set's last entry, the short way: one sweep counts the entries per top byte of the key, the byte value
         * in which the k-th falls is picked out into the list and the k-th is found there. The long way (four
         * sweeps, ties by bisection) stays for what does not fit the list. */
        unsigned long long t_set    = 0ull;
        bool               have_set = false;
        int                n_list   = 0;
        auto               lst_sw   = [&](auto &&f) { list_sweep(g, list, n_list, f); };
        if (p.gen_list_cap > 0) {
            const RadixOut r3 = radix_mass<true>(g, sh, hm, hc, copies, 1.0, row_sw, (double) r.k, true, okey, one, 3);
            if (r3.found && r3.ties <= (long long) p.gen_list_cap) {
                const unsigned top = r3.key >> 24;
                n_list             = pick_out([&](float x, int) { return (order_key(x) >> 24) == top; });
                if (n_list <= p.gen_list_cap) {
                    const double   tgt = (double) r.k - r3.above;
                    const RadixOut rc  = radix_mass<true>(g, sh, hm, hc, copies, 1.0, lst_sw, tgt, true, okey, one);
                    if (rc.found) {
                        t_set    = resolve_ties(g, sh, lst_sw, idx_bits, rc, tgt, true, okey, one);
                        have_set = true;
                    }
                }
            }
        }
        if (!have_set) {
            const RadixOut rs = radix_mass<true>(g, sh, hm, hc, copies, 1.0, row_sw, (double) r.k, true, okey, one);
            t_set             = rs.found ? resolve_ties(g, sh, row_sw, idx_bits, rs, (double) r.k, true, okey, one) : 0ull;
        }
        auto in_set = [&](float x, int i) { return composite(order_key(x), i, idx_bits) >= t_set; };
        /* the kept set itself (at most 8192 entries) goes into the list: its sum and the draw are found there */
        n_list            = p.gen_list_cap > 0 ? pick_out(in_set) : p.gen_list_cap + 1;
        const bool listed = n_list <= p.gen_list_cap;
        if (r.select_only) {
            if (listed) {
                for (int j = g.tid; j < min(n_list, p.kept_cap); j += g.n) {
                    kept_i[j] = list[j].idx + p.vocab_offset;
                    kept_v[j] = list[j].v;
                }
            } else {
                if (g.tid == 0) {
                    sh->n_sel = 0;
                }
                g.sync();
                row_sweep(g, cur, V, [&](float x, int i) {
                    if (in_set(x, i)) {
                        const int pos = atomicAdd(&sh->n_sel, 1);
                        if (pos < p.kept_cap) {
                            kept_i[pos] = i + p.vocab_offset;
                            kept_v[pos] = x;
                        }
                    }
                });
            }
            if (g.tid == 0) {
                p.kept_n[r.row] = r.k;
                p.tokens[r.row] = row_arg + p.vocab_offset;
            }
        } else {
            auto   qof = [&](float x) { return (double) exp_exact(scaled_arg(x, row_max, r.inv_t)); };
            double m   = 0.0;
            auto   set_sw = [&](auto &&f) { /* the kept set: from the list, else filtered out of the row */
                if (listed) {
                    list_sweep(g, list, n_list, f);
                } else {
                    row_sweep(g, cur, V, [&](float x, int i) {
                        if (in_set(x, i)) {
                            f(x, i);
                        }
                    });
                }
            };
            set_sw([&](float x, int) { m += qof(x); });
            const double S = group_sum_d(g, sh, m);
            const double u = (double) unit_from(xorshift_next(r.rng)) * S;
            /* the pick is the earliest walk position whose running sum exceeds u: the largest
             * word t with mass{word >= t} > u */
            auto                     qmass  = [&](float x, int) { return qof(x); };
            const RadixOut           rp     = radix_mass(g, sh, hm, hc, copies, 0x1p49, set_sw, u, false, okey, qmass); /* weights <= 1, at most 8192 of them */
            unsigned long long       t_pick = rp.found ? resolve_ties(g, sh, set_sw, idx_bits, rp, u, false, okey, qmass) : 0ull;
            if (t_pick < t_set) {
                t_pick = t_set;
            }
            if (g.tid == 0) { /* the word names its entry */
                const unsigned long long id_mask = (1ull << idx_bits) - 1ull;
                p.tokens[r.row]                  = min((int) (id_mask - (t_pick & id_mask)), V - 1) + p.vocab_offset;
            }
            if (g.tid == 0 && p.kept_cap > 0) {
                p.kept_n[r.row] = r.k;
            }
            if (p.kept_cap > 0) {
                st |= ST_KEPT_PARTIAL;
            }
        }
    } else {
        /* top-p with any nucleus size: the copy becomes e_i, then p_i (sampler.c:245-255) */
        double acc = 0.0;
        /* e_i as a correctly rounded expf gives it: with a nucleus of tens of thousands of ids an
         * exponential that is off by a fraction of an ulp on average moves the running sum by more than
         * the distance between two neighbours of the walk */
        row_map(g, cur, gr, V, [&](float x, int) {
            const float e = exp_exact(scaled_arg(x, row_max, r.inv_t));
            acc += (double) e;
            return e;
        });
        cur            = gr; /* from here on the sweeps read the rewritten copy */
        const double S = group_sum_d(g, sh, acc);
        MP(3);
        /* p_i; and while every p_i is in hand it is binned by the top byte of the window's key (what the short way
         * below starts from) */
        const unsigned k_top_w   = __float_as_uint(__double2float_rn(1.0 / S));
        const float    p_floor_w = __double2float_rn(0.5 * (1.0 - (double) r.top_p) / (double) V);
        const unsigned k_floor_w = (p_floor_w > 0.0f && __float_as_uint(p_floor_w) < k_top_w) ? __float_as_uint(p_floor_w) : 0u;
        const unsigned span_w    = k_top_w > k_floor_w ? k_top_w - k_floor_w : 0u;
        const int      ls_w      = span_w > 0u ? __clz(span_w) : 0;
        {
            unsigned long long *hq = reinterpret_cast<unsigned long long *>(hm);
            for (int i = g.tid; i < copies * 256; i += g.n) {
                hq[i] = 0ull;
                hc[i] = 0;
            }
            g.sync();
            unsigned long long *mym = hq + (g.warp % copies) * 256;
            int                *myc = hc + (g.warp % copies) * 256;
            row_rewrite(g, gr, V, [&](float e, int) {
                const float    pv = __double2float_rn((double) e / S);
                const unsigned k  = __float_as_uint(pv);
                if (k >= k_floor_w && pv > 0.0f) {
                    const unsigned d = ((min(k, k_top_w) - k_floor_w) << ls_w) >> 24;
                    atomicAdd(&mym[d], __double2ull_rz((double) pv * 0x1p62));
                    atomicAdd(&myc[d], 1);
                }
                return pv;
            });
        }
        g.sync();
        MP(4);
        auto keyf  = [](float pv) { return __float_as_uint(pv); }; /* p >= 0: the bits are ordered */
        auto massf = [](float pv, int) { return (double) pv; };
        /* cutoff: first walk position whose running sum reaches top_p, inclusive */
        /* The radix walks look at a window of keys stretched over all 32 bits, so that the entries
         * spread over the byte values instead of piling up in a few. Cutoff: entries with
         * p < (1 - top_p) / V add up to less than 1 - top_p, so the walk crosses above them. */
        auto windowed = [&](unsigned k_lo, unsigned k_hi, double target, bool inclusive, auto &&mass_in) {
            const unsigned span = k_hi > k_lo ? k_hi - k_lo : 0u;
            const int      ls   = span > 0u ? __clz(span) : 0;
            auto           kw   = [&](float pv) {
                const unsigned k = keyf(pv);
                return k >= k_lo ? (min(k, k_hi) - k_lo) << ls : 0u;
            };
            auto mw = [&](float pv, int i) { return keyf(pv) >= k_lo ? mass_in(pv, i) : 0.0; };
            RadixOut ro = radix_mass(g, sh, hm, hc, copies, 0x1p62, row_sw, target, inclusive, kw, mw); /* probabilities: the row adds up to 1 */
            ro.key      = (ro.key >> ls) + k_lo; /* back to the key itself */
            return ro;
        };
        const unsigned k_top   = keyf(__double2float_rn(1.0 / S)); /* the largest p: e = 1 at the row maximum */
        const float    p_floor = __double2float_rn(0.5 * (1.0 - (double) r.top_p) / (double) V);
        const unsigned k_floor = (p_floor > 0.0f && keyf(p_floor) < k_top) ? keyf(p_floor) : 0u;
        const unsigned long long id_mask = (1ull << idx_bits) - 1ull;
        unsigned long long t_cut = 0ull, t_pick = 0ull;
        long long          cut   = 0;
        bool               have_cut = false, have_pick = false;
        double             N = 0.0, u = 0.0;
        /*
         * Short way. One sweep bins the row by the top byte of the window's key (mass and count per bin). The
         * walk crosses top_p inside one bin: its entries (a few hundred on rows of this kind) are picked out into
         * a list, and the crossing entry is found on the list, target reduced by the mass of the bins above. The
         * draw is walked the same way: the bins' masses are known already (the crossing bin's is what of it lies
         * in the nucleus), the bin it falls into is picked out if it is another one, and the entry is found on
         * that list. Three sweeps of the row instead of a dozen and more. Whatever does not fit (a bin with more
         * entries than the list holds, sums that round apart) takes the long way below.
         */
        {
            const unsigned span = k_top > k_floor ? k_top - k_floor : 0u;
            const int      ls   = span > 0u ? __clz(span) : 0;
            auto           kw   = [&](float pv) {
                const unsigned k = keyf(pv);
                return k >= k_floor ? (min(k, k_top) - k_floor) << ls : 0u;
            };
            auto mwin = [&](float pv, int) { return keyf(pv) >= k_floor ? (double) pv : 0.0; };
            unsigned long long *sq   = reinterpret_cast<unsigned long long *>(save_mem); /* the bins' masses and counts, kept */
            int                *sc   = reinterpret_cast<int *>(sq + 256);
            auto in_bin_of = [&](int bin) { return [&, bin](float pv, int) { return keyf(pv) >= k_floor && (int) (kw(pv) >> 24) == bin && pv > 0.0f; }; };
            const RadixOut r3 = radix_mass(g, sh, hm, hc, copies, 0x1p62, row_sw, (double) r.top_p, true, kw, mwin, 3, true);
            MP(11);
            if (r3.found && r3.ties <= (long long) p.gen_list_cap && p.gen_list_cap > 0) {
                const int b_cut = (int) (r3.key >> 24);
                if (g.tid < 256) { /* the histograms of the sweep are still there: their sums are kept for the draw */
                    unsigned long long q = 0ull;
                    int                c = 0;
                    for (int w = 0; w < copies; w++) {
                        q += reinterpret_cast<unsigned long long *>(hm)[w * 256 + g.tid];
                        c += hc[w * 256 + g.tid];
                    }
                    sq[g.tid] = q;
                    sc[g.tid] = c;
                }
                g.sync();
                int  n_list = pick_out(in_bin_of(b_cut));
                MP(12);
                auto lst_sw = [&](auto &&f) { list_sweep(g, list, n_list, f); };
                if (n_list <= p.gen_list_cap) {
                    const double   tgt = (double) r.top_p - r3.above;
                    const RadixOut rc  = radix_mass(g, sh, hm, hc, copies, 0x1p62, lst_sw, tgt, true, keyf, massf);
                    if (rc.found) {
                        MP(13);
                        t_cut      = resolve_ties(g, sh, lst_sw, idx_bits, rc, tgt, true, keyf, massf);
                        MP(14);
                        double nm  = 0.0;
                        long long ncnt = 0;
                        lst_sw([&](float pv, int i) {
                            if (composite(keyf(pv), i, idx_bits) >= t_cut) {
                                nm += (double) pv;
                                ncnt++;
                            }
                        });
                        const double in_bin = group_sum_d(g, sh, nm);
                        N                   = r3.above + in_bin;
                        cut                 = r3.n_above + group_sum_ll(g, sh, ncnt);
                        have_cut            = true;
                        u                   = (double) unit_from(xorshift_next(r.rng)) * N;
                        /* the bin the draw falls into: a walk over the kept bins from the top, the crossing bin with
                         * its share of the nucleus */
                        if (g.tid == 0) {
                            double run = 0.0;
                            int    bp  = -1;
                            for (int bin = 255; bin >= b_cut && bp < 0; bin--) {
                                const double mb = bin == b_cut ? in_bin : (double) sq[bin] / 0x1p62;
                                if (u < run + mb) {
                                    bp = bin;
                                } else {
                                    run += mb;
                                }
                            }
                            sh->b_star = bp;
                            sh->S      = run;
                        }
                        g.sync();
                        MP(15);
                        const int    b_pick  = sh->b_star;
                        const double above_p = sh->S;
                        g.sync();
                        if (b_pick < 0) {
                            have_pick = true; /* rounding left u at the very end: the last nucleus entry (sampler.c:292) */
                        } else if (b_pick == b_cut) {
                            auto           nml = [&](float pv, int i) { return composite(keyf(pv), i, idx_bits) >= t_cut ? (double) pv : 0.0; };
                            const double   ut  = u - above_p;
                            const RadixOut rk  = radix_mass(g, sh, hm, hc, copies, 0x1p62, lst_sw, ut, false, keyf, nml);
                            t_pick             = rk.found ? resolve_ties(g, sh, lst_sw, idx_bits, rk, ut, false, keyf, nml) : 0ull;
                            have_pick          = true;
                        } else if (sc[b_pick] <= p.gen_list_cap) {
                            n_list = pick_out(in_bin_of(b_pick));
                            MP(16);
                            if (n_list <= p.gen_list_cap) {
                                const double   ut = u - above_p;
                                const RadixOut rk = radix_mass(g, sh, hm, hc, copies, 0x1p62, lst_sw, ut, false, keyf, massf);
                                t_pick            = rk.found ? resolve_ties(g, sh, lst_sw, idx_bits, rk, ut, false, keyf, massf) : 0ull;
                                have_pick         = true;
                            }
                        }
                    }
                }
            }
        }
        if (!have_cut) { /* the long way: radix walks over the whole row */
            RadixOut rc = windowed(k_floor, k_top, (double) r.top_p, true, massf);
            if (!rc.found && k_floor != 0u) {
                rc = windowed(0u, k_top, (double) r.top_p, true, massf); /* rounding kept the window short of top_p */
            }
            MP(5);
            t_cut = rc.found ? resolve_ties(g, sh, row_sw, idx_bits, rc, (double) r.top_p, true, keyf, massf) : 0ull;
            MP(6);
            double    nm   = 0.0;
            long long ncnt = 0;
            row_sweep(g, gr, V, [&](float pv, int i) {
                if (composite(keyf(pv), i, idx_bits) >= t_cut) {
                    nm += (double) pv;
                    ncnt++;
                }
            });
            N   = group_sum_d(g, sh, nm);
            MP(7);
            cut = group_sum_ll(g, sh, ncnt);
            u   = (double) unit_from(xorshift_next(r.rng)) * N;
        }
        if (!have_pick) {
            auto           nmass = [&](float pv, int i) { return composite(keyf(pv), i, idx_bits) >= t_cut ? (double) pv : 0.0; };
            const RadixOut rk    = windowed((unsigned) (t_cut >> idx_bits), k_top, u, false, nmass);
            MP(8);
            t_pick = rk.found ? resolve_ties(g, sh, row_sw, idx_bits, rk, u, false, keyf, nmass) : 0ull;
            MP(9);
        }
        if (t_pick < t_cut) {
            t_pick = t_cut; /* default: the last nucleus entry (sampler.c:292) */
        }
        if (g.tid == 0) { /* the word names its entry: the id is in its low bits */
            p.tokens[r.row] = min((int) (id_mask - (t_pick & id_mask)), V - 1) + p.vocab_offset;
        }
        if (g.tid == 0 && p.kept_cap > 0) {
            p.kept_n[r.row] = (int) cut;
        }
        if (p.kept_cap > 0) {
            st |= ST_KEPT_PARTIAL;
        }
    }
    g.sync();
    MP(10);
    return st;
}

/* Status of a finished row and, behind a sequence's last row, its generator. One thread. */
__device__ __forceinline__ void row_epilogue(const SampleParams &p, const RowCfg &r, int row, int st, unsigned long long rng0) {
    p.status[row] = st;
    if (p.rng_out != nullptr && r.rr == p.rows_per_seq - 1) {
        /* the sequence's generator (rng0: the word it came with) after all of its rows drew */
        unsigned long long s = rng0;
        for (int i = 0; i < p.rows_per_seq * r.draws_per_row; i++) {
            (void) xorshift_next(s);
        }
        p.rng_out[r.seq] = s;
    }
}

} /* namespace gb */

#include "sampler_wide.cuh"

namespace gb {

/* ------------------------------------------------------------ shared state -- */

constexpr int kTagAt  = 21; /* above an entry's ten bits of offset and eleven of count (kRowIdsMax at most) */
constexpr int kIdBits = 4 * kSliceMax;
/* Where the bit of a value lies: slice of the part, warp, offset in the share. */
__device__ __forceinline__ int id_bit(int s, int w, int off) { return ((s & 3) * kWarps + w) * (kSliceMax / kWarps) + off; }

constexpr int kKeyBins = 512; /* among which the threshold is sought */

/* A part whose candidates outran their list, for raise_threshold. */
struct PartAgain {
    int             row, c0, part_len, gm_shift, kq;
    bool            pro, sums; /* cap or mask to apply; top-p: the candidates leave the sum */
    float           inv_t;
    bool            pen, long_ids;
    float           rep, freq, pres;
    double          rep_rcp;
    const int      *long_off;  /* long histories: where the part's shares' runs start ... */
    const unsigned *list;      /* the ids' entries */
    bool            long_smem; /* where the runs start lies in shared memory, as for ids counted here */
};

/* What the warps of one thread block share. The ring (every warp's two stages) lies in front of it in dynamic
 * shared memory, the group maxima of the part in work behind it. */
struct __align__(16) StreamShared {
    unsigned long long full[kWarps][kStages]; /* warp w's share of item j has landed in its stage j % kStages */
    /* the part in work */
    int                st;        /* status bits of the part */
    unsigned long long best[kWarps];               /* (key of the maximum, ~first id) per warp */
    float              wb_ref[kWarps];             /* top-p: what the warp's sum is relative to ... */
    double             wb_acc[kWarps];             /* ... that sum ... */
    double             wb_sum[kWarps];             /* ... and the sum without the candidates, relative to the part's reference */
    float              ref_at[kSliceRefs][kWarps]; /* top-p: what a slice's terms were formed relative to */
    unsigned           rl_id[kRowIds]; /* the row's distinct history ids as (offset in the share | count << 10 | tag << kTagAt),
                                        * grouped by the (slice, warp) share they fall into (rows that can bring more: behind the group maxima) ... */
    alignas(16) int    rl_cnt[kRowIds + 4]; /* ... and where each group's run starts */
    alignas(16) unsigned id_bits[kIdBits / 32];             /* which values of the part an id has changed (slices s and s + 4 share their bits) */
    /* the part's select */
    uint2              key_ends[kWarps];      /* smallest and largest key of a warp's thread maxima */
    int                n_grp, n_cand;         /* groups that reach the threshold; candidates in them */
    int                max_cnt;               /* how often the part's most frequent id occurs (asked where that raises a value) */
    alignas(16) unsigned short grp[kGroupSlots * kThreads]; /* (slot << 8) | thread; at a part's set-up, how many ids each group of them has */
    alignas(8) Pair    cand[kPartCand];
    PartAgain          again;                 /* what raise_threshold needs to know of the part */
    /* finishing inside the stream kernel (F_INLINE_TOPK): the k best in order, their weights */
    int                cur_rr;
    union {
        alignas(16) Pair fin_s[kFastKMax];
        int              key_bins[kKeyBins]; /* before that, while the threshold is sought */
    };
    alignas(8) float   fin_q[kFastKMax];
    unsigned long long cur_rng;         /* the generator word the part's sequence came with, its sequence, and whether the row is the sequence's last */
    int                cur_seq, cur_last;
    float              cap;             /* the part's soft cap and mask row (0 / null: none) */
    const unsigned    *mrow;
    const unsigned    *raw_word[kRawWords]; /* SampleParams::raw_word: lanes that read different words of a constant take turns */
    RawCfg             raw_nxt;         /* parameters of the next row of this run, copied in while the part streams */
    alignas(16) int    nxt_ids[kRowIds]; /* that row's history ids (raw): the first words of its history row ... */
    int                nxt_ext[kRowIds]; /* ... and the tokens fed before it */
};

/* What comes in of every part in one round trip, before its count of candidates is known: its record and the first
 * candidates behind it, kStageWords words of 8 bytes shared out over the parts, an even number each and no more than kStageMost. */
constexpr int kStageWords = 1024;
constexpr int kStageMost  = 128;

/* What the threads of one finishing thread block share; the merged candidate list lies behind it. */
struct __align__(16) FinishShared {
    GroupShared gs; /* reductions of the whole thread block */
    int         poff[kMaxParts]; /* where a part's candidates begin among those that did not come in with the records */
    alignas(16) int bhist[kHistBins]; /* select histogram */
    int         n_sel, n_ent, slot;
    unsigned    fin_bitmap[kFinBitmapWords];
    Pair        fsort[kFastKMax];
    alignas(8) float fq[kFastKMax];
    alignas(16) unsigned long long stage[kStageWords]; /* the records and first candidates of the row's parts */
    unsigned long long save[256 + 128];                      /* the multi-pass path keeps a histogram here */
    RowCfg      cfg;    /* the row's: in registers it had left none for the code that finishes it */
    unsigned long long rng0; /* the generator word that the row's sequence came with */
    double      wide_S; /* a top-p row that the candidates could not serve: its sum, 0 where it is not known */
};

constexpr int kGroupBytes = kGroupSlots * kThreads * 4; /* one maximum per slot and thread */
constexpr int kListSmem   = kRowIdsMax;       /* id-list entries of a part that are kept in shared memory */
constexpr int kRankWords  = 2 * (kHistBins + 1) + 3; /* what puts candidates in order, beside them */
constexpr int kFinCap     = 2048;             /* candidates the finisher can order per row (8 per thread) */
static_assert(kPartCand * (int) sizeof(Pair) + kRankWords * 4 <= kGroupBytes, "a part's candidates are put in order there");
constexpr int kFinBytes   = 2 * kFinCap * (int) sizeof(Pair) + (kRankWords + 1) * 4; /* finisher: the merged candidate list, what puts it in order; the multi-pass path keeps one byte histogram per warp there */
static_assert(kFinBytes >= kWarps * 256 * 12, "a byte histogram per warp fits");
constexpr int kFinGeneralBytes = sizeof(WideShared) > (size_t) kFinBytes ? (int) sizeof(WideShared) : kFinBytes; /* the general kernel works on wide rows there as well */
static_assert(kGroupBytes >= 2 * kRowIdsMax * 8, "the id table of a part's set-up lies in the group maxima's memory");
static_assert(kGroupSlots <= 256 && kThreads == 256, "a group's name fits 16 bits");

/* Part `k` of a row in global scratch: its record (two int4), then its candidates. */
__device__ __forceinline__ int4 *part_rec(const SampleParams &p, int row, int k) {
    return reinterpret_cast<int4 *>(p.parts + ((size_t) row * (size_t) p.parts_max + (size_t) k) * (size_t) kPartBytes);
}

/* n things dealt out in runs of q + 1 (the first r runs) and q: which run holds thing i */
__device__ __forceinline__ int run_of(int i, int q, int r) { return i < r * (q + 1) ? i / (q + 1) : r + (i - r * (q + 1)) / q; }

/* a / d for a quotient of at most 1024, given 1 / d: the float product is off by one at most */
__device__ __forceinline__ int quotient(int a, int d, float rcp) {
    int       q = __float2int_rz((float) a * rcp);
    const int r = a - q * d;
    return q + (r >= d ? 1 : 0) - (r < 0 ? 1 : 0);
}

/* The thread block that streams item i, and the run [first, first + count) of thread block b (RunMap). */
__device__ __forceinline__ int cta_of_item(const SampleParams &p, int i) {
    const RunMap &m = p.map;
    if (m.mode == RUN_ITEMS) {
        return run_of(i, m.q, m.r);
    }
    const int row = i / p.n_slices;
    if (m.mode == RUN_ROWS) {
        return run_of(row, m.q, m.r);
    }
    return row * m.P + run_of(i - row * p.n_slices, m.q, m.r);
}
__device__ __forceinline__ void run_of_cta(const SampleParams &p, int b, int &first, int &count) {
    const RunMap &m = p.map;
    if (m.mode == RUN_ITEMS) {
        first = b * m.q + min(b, m.r);
        count = m.q + (b < m.r ? 1 : 0);
    } else if (m.mode == RUN_ROWS) {
        first = (b * m.q + min(b, m.r)) * p.n_slices;
        count = (m.q + (b < m.r ? 1 : 0)) * p.n_slices;
    } else {
        const int row = b / m.P, j = b - row * m.P;
        first         = row * p.n_slices + j * m.q + min(j, m.r);
        count         = m.q + (j < m.r ? 1 : 0);
    }
}

/* Highest bin b with at least kq entries in bins >= b (0 when there is none); the whole warp calls, every lane gets it. */
__device__ __forceinline__ int top_bin(const int *hist, int lane, int kq) {
    int cc[8], mine = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        cc[i] = *reinterpret_cast<const volatile int *>(&hist[8 * lane + i]);
        mine += cc[i];
    }
    int suffix = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int dn = __shfl_down_sync(0xffffffffu, suffix, o);
        if (lane + o < 32) {
            suffix += dn;
        }
    }
    const unsigned ball = __ballot_sync(0xffffffffu, suffix >= kq);
    int            b    = 0;
    if (ball != 0u && lane == 31 - __clz(ball)) {
        int run = suffix - mine;
        b       = 8 * lane;
#pragma unroll
        for (int i = 7; i >= 0; i--) {
            run += cc[i];
            if (run >= kq) {
                b = 8 * lane + i;
                break;
            }
        }
    }
    return __shfl_sync(0xffffffffu, b, ball != 0u ? 31 - __clz(ball) : 0);
}

/* ------------------------------------------------------ few candidates, weights -- */

/* At most kRankFew candidates in order, the k best to out_s, with kWeigh their weights e^((x - max) / T) to out_q. Four threads (two beyond
 * 64 candidates) compare a candidate with a share of the others each, eight at a time without a branch between them.
 * All threads call; the caller's barrier follows. */
constexpr int kRankFew = 128;
static_assert(2 * kRankFew == kThreads, "two threads per candidate");
template <bool kWeigh>
__device__ __forceinline__ void rank_few(const Pair *cand, int total, int k, float inv_t, Pair *out_s, float *out_q) {
    const int  log = total <= kRankFew / 2 ? 2 : 1, i = (int) threadIdx.x >> log, step = 1 << log, sub = (int) threadIdx.x & (step - 1);
    const Pair me   = cand[min(i, total - 1)];
    int        rank = 0;
    float      top  = -CUDART_INF_F;
#pragma unroll 1
    for (int j0 = sub; j0 < total; j0 += 8 * step) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const Pair o = cand[min(j0 + j * step, total - 1)];
            rank += j0 + j * step < total && pair_before(o.v, o.idx, me.v, me.idx) ? 1 : 0;
            top = kWeigh ? fmaxf(top, o.v) : top;
        }
    }
    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
    top = kWeigh ? fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1)) : top;
    if (log == 2) {
        rank += __shfl_xor_sync(0xffffffffu, rank, 2);
        top = kWeigh ? fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2)) : top;
    }
    if (sub == 0 && i < total && rank < k) {
        out_s[rank] = me;
        if (kWeigh) {
            out_q[rank] = exp_exact(scaled_arg(me.v, top, inv_t));
        }
    }
}

/* `total` candidates dealt out to kHistBins bins, the highest in front, in srt; entry b of start: candidates in the bins before b.
 * Whether the bin that the k-th falls into holds more than kRankMost. All threads call. */
constexpr int kRankMost = 256; /* entries of that bin that are ranked against each other: dealing them out again costs as much */
template <class Bin>
__device__ __forceinline__ bool deal_out(const Pair *in, int total, int k, Pair *srt, int *start, Bin &&bin_of) {
    const int tid = (int) threadIdx.x, lane = tid & 31;
    int      *next = start + kHistBins + 1;
    for (int i = tid; i <= kHistBins; i += kThreads) {
        start[i] = 0; /* entry b + 1: candidates in bin b, until the scan */
    }
    __syncthreads();
    for (int i = tid; i < total; i += kThreads) {
        atomicAdd(&start[bin_of(in[i].v) + 1], 1);
    }
    __syncthreads();
    if (tid < 32) {
        int v[kHistBins / 32], run = 0;
#pragma unroll
        for (int i = 0; i < kHistBins / 32; i++) {
            run += start[1 + kHistBins / 32 * lane + i];
            v[i] = run;
        }
        int before = run;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, before, d);
            if (lane >= d) {
                before += o;
            }
        }
        before -= run;
#pragma unroll
        for (int i = 0; i < kHistBins / 32; i++) {
            start[1 + kHistBins / 32 * lane + i] = before + v[i];
            next[1 + kHistBins / 32 * lane + i]  = before + v[i];
        }
        if (lane == 0) {
            next[0] = 0;
        }
    }
    __syncthreads();
    for (int i = tid; i < total; i += kThreads) {
        const Pair me                           = in[i];
        srt[atomicAdd(&next[bin_of(me.v)], 1)] = me;
    }
    static_assert(kHistBins == kThreads, "a bin per thread");
    return __syncthreads_or(start[tid] < k && start[tid + 1] - start[tid] > kRankMost) != 0; /* bins further up hold less than k */
}
/* What deal_out left, each candidate ranked against its own bin. */
template <class Bin>
__device__ __forceinline__ void rank_dealt(const Pair *srt, int total, int k, const int *start, Pair *out_s, Bin &&bin_of) {
    for (int i = (int) threadIdx.x; i < total; i += kThreads) {
        const Pair me   = srt[i];
        const int  b    = bin_of(me.v), end = start[b + 1];
        int        rank = start[b];
        if (rank < k) {
            for (int j = rank; j < end; j++) {
                rank += pair_before(srt[j].v, srt[j].idx, me.v, me.idx) ? 1 : 0;
            }
            if (rank < k) {
                out_s[rank] = me;
            }
        }
    }
}
/* Bins of keys: those from lo to hi, 2^shift each, are dealt out to bins 1 to 254, what lies above to bin 0. */
struct KeyBins {
    unsigned lo, hi;
    int      shift;
    __device__ __forceinline__ int operator()(float v) const {
        const unsigned key = order_key(v);
        return key > hi ? 0 : key < lo ? kHistBins - 1 : kHistBins - 2 - (int) ((key - lo) >> shift);
    }
};
/* Bins of values from lo on, scale of them to a unit, the highest in front; by_octave: of the values' bits. */
struct ValueBins {
    float lo, scale;
    bool  by_octave;
    __device__ __forceinline__ int operator()(float v) const {
        return kHistBins - 1 - min(kHistBins - 1, max(0, __float2int_rz(((by_octave ? (float) __float_as_int(v) : v) - lo) * scale)));
    }
};
/* The bin of `first` that the k-th of the candidates dealt out falls into holds too many: it is cut again between its smallest and its
 * largest key, until the bin that the k-th is in holds few, or equal ones. Fewer than k lie above it, what lies below is not ranked. False:
 * its entries are equal, what has been dealt out stays as it is. Out of line: rare. */
__device__ __noinline__ bool rank_crowded(const Pair *in, int total, int k, const ValueBins first, Pair *srt, int *start, Pair *out_s) {
    const int tid  = (int) threadIdx.x;
    unsigned *ends = reinterpret_cast<unsigned *>(start + 2 * (kHistBins + 1)); /* smallest and largest key of the bin, and which it is */
    KeyBins   bins{0u, 0u, -1};
    do {
        if (start[tid] < k && start[tid + 1] >= k) {
            ends[0] = 0xffffffffu;
            ends[1] = 0u;
            ends[2] = (unsigned) tid;
        }
        __syncthreads();
        const int b  = (int) ends[2];
        unsigned  lo = 0xffffffffu, hi = 0u;
        for (int i = tid; i < total; i += kThreads) {
            const float v = in[i].v;
            if ((bins.shift < 0 ? first(v) : bins(v)) == b) {
                lo = min(lo, order_key(v));
                hi = max(hi, order_key(v));
            }
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if ((tid & 31) == 0) {
            atomicMin(&ends[0], lo);
            atomicMax(&ends[1], hi);
        }
        __syncthreads();
        if (bins.shift < 0 && ends[0] == ends[1]) {
            return false;
        }
        bins.lo              = ends[0];
        bins.hi              = ends[1];
        const unsigned range = bins.hi - bins.lo;
        bins.shift           = max(0, 32 - __clz(range) - 8);
        bins.shift += (range >> bins.shift) > (unsigned) (kHistBins - 3) ? 1 : 0;
    } while (deal_out(in, total, k, srt, start, bins) && bins.shift > 0);
    rank_dealt(srt, total, k, start, out_s, bins);
    return true;
}
/* More than kRankFew candidates in order, the k best to out_s; they lie between lo and hi. They are dealt out to 256 bins of
 * values, the highest in front (srt takes them), and ranked against their own bin: one against all costs a thread block
 * total^2 / 32 rounds of six instructions. 1000 rows of 8192, us: top-k 128 54.3 -> 45.8, 200 81.5 -> 53.7, 250 105 -> 59.9;
 * 256 x 128256 top-k 200 48.9 -> 41.0. by_octave: bins of the values' bits, for probabilities (lo is not used); in even bins all but
 * a few share the last, and eight top-p rows of 19 parts took 67 us instead of 41. A value far above the rest does the same to the bins
 * of values: rank_crowded (64 x 32000 with a value of 4000 in each row, top-k 256: 197 us without it, 30; 8 x 128256, top-k 129: 248 and 27).
 * start: room for kRankWords words. All threads call; the caller's barrier follows. */
__device__ __noinline__ void rank_in_bins(const Pair *in, int total, int k, float lo, float hi, bool by_octave, Pair *srt, int *start, Pair *out_s) {
    if (by_octave) {
        hi = (float) __float_as_int(hi);
        lo = hi - (float) (20 << 23); /* what is a millionth of the largest or less shares the last bin */
    }
    const ValueBins bins{lo, hi > lo && hi - lo < CUDART_INF_F ? (float) kHistBins / (hi - lo) : 0.0f, by_octave}; /* 0: one bin for all */
    if (!deal_out(in, total, k, srt, start, bins) || !rank_crowded(in, total, k, bins, srt, start, out_s)) {
        rank_dealt(srt, total, k, start, out_s, bins);
    }
}

/*
 * The reference's draw over k <= 256 weights in descending order (sampler.c:90-102): the sum and the walk in its order, in
 * double. Where the smallest weight is at least 2^-22 every partial sum is a whole number of 2^-45 below 2^53 of them, so
 * exact in any order, and the warp adds in parallel; else one lane adds one by one. The whole warp calls: the place that
 * u01 times the sum falls on, and the sum. (Between the candidates and the token of one row, top-k 40: 1.9 us with a thread per
 * candidate to rank them, the exponentials behind a barrier and one thread over the weights, twice; 1.25 us.)
 */
__device__ __forceinline__ int draw_sorted(int lane, const float *q, int k, float u01, double *S_out) {
    const float2 two = 2 * lane < k ? *reinterpret_cast<const float2 *>(q + 2 * lane) : make_float2(0.0f, 0.0f); /* what lies behind the k-th weight is not used */
    if (q[k - 1] >= 0x1p-22f) {
        const int per  = k <= 64 ? 2 : (k + 31) >> 5, i0 = lane * per;
        double    incl = (double) two.x + (2 * lane + 1 < k ? (double) two.y : 0.0);
        if (k > 64) {
            incl = 0.0;
#pragma unroll 1
            for (int i = i0; i < min(i0 + per, k); i++) {
                incl += (double) q[i];
            }
        }
        const double mine = incl;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) {
                incl += up;
            }
        }
        const double S = __shfl_sync(0xffffffffu, incl, 31), u = (double) u01 * S;
        const int    from = __ffs(__ballot_sync(0xffffffffu, u < incl)) - 1; /* the lane whose run crosses u, -1: none */
        double       a    = incl - mine;
        int          pick = i0;
        if (k <= 64) {
            pick += u < a + (double) two.x ? 0 : 1;
        } else {
#pragma unroll 1
            for (; pick < min(i0 + per, k) - 1; pick++) {
                a += (double) q[pick];
                if (u < a) {
                    break;
                }
            }
        }
        *S_out = S;
        return from < 0 ? k - 1 : __shfl_sync(0xffffffffu, pick, from);
    }
    double S    = 0.0;
    int    pick = k - 1;
    if (lane == 0) {
#pragma unroll 1
        for (int i0 = 0; i0 < k; i0 += 8) { /* eight weights per round: their loads overlap, the sum keeps its order */
            float w8[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                w8[i] = i0 + i < k ? q[i0 + i] : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                S += (double) w8[i]; /* adding +0 behind the last weight changes nothing */
            }
        }
        const double u = (double) u01 * S;
        double       a = 0.0;
#pragma unroll 1
        for (int i = 0; i < k; i++) {
            a += (double) q[i];
            if (u < a) {
                pick = i;
                break;
            }
        }
    }
    *S_out = __shfl_sync(0xffffffffu, S, 0);
    return __shfl_sync(0xffffffffu, pick, 0);
}

/* ---------------------------------------------------------------- finisher -- */

/* A row's parameters, as the finishing kernels need them. */
__device__ __forceinline__ RowCfg finish_config(const SampleParams &p, int row, const RawCfg &rc) {
    RowCfg r = row_config(p, row, rc, true);
    if (p.out_logits != nullptr) { /* read back as it is sampled from (row_again) */
        r.cap    = 0.0f;
        r.mrow   = nullptr;
        r.pen_on = false;
    }
    return r;
}
/* Nobody has to wait for a row of another kind. The thread that has written its parameters. */
template <bool kFast>
__device__ __forceinline__ void not_wide(const SampleParams &p, const FinishShared *sh) {
    if (!kFast && sh->cfg.mode != M_TOPP) {
        atomicAdd(&p.wide_head->rows, 1ull);
    }
}

/*
 * One row, all threads of a finishing thread block. Merges the parts' records, then by mode: argmax; temperature
 * (segment sums, then the crossing segment re-read and walked); top-k / top-p over the merged candidates. cmem:
 * room for the merged list. first: the thread block's. Returns the row's status bits (ST_DEFERRED: the multi-pass path has to serve it).
 */
template <bool kFast>
__device__ __forceinline__ int finish_row(const Grp &g, const SampleParams &p, FinishShared *sh, int row, int n_parts, bool first, bool temp, unsigned char *cmem) {
    const RowCfg &r    = sh->cfg; /* the thread block's first row's is there, any other's behind the second barrier */
    int       *kept_i  = p.kept_cap > 0 ? p.kept_idx + (size_t) row * (size_t) p.kept_cap : nullptr;
    float     *kept_v  = p.kept_cap > 0 ? p.kept_val + (size_t) row * (size_t) p.kept_cap : nullptr;
    Pair      *cbuf    = reinterpret_cast<Pair *>(cmem);
    GroupShared *gs    = &sh->gs;
    int        st      = 0;

    g.sync(); /* the staging of the row before is no longer read */
    if (g.tid == 0) {
        sh->wide_S = 0.0;
        sh->n_sel  = 0;
    }
    sh->bhist[g.tid] = 0;
    static_assert(kHistBins == kThreads, "a bin per thread");
    const int st_parts = min(n_parts, kStageWords / 4), st_w = min(kStageMost, (kStageWords / st_parts) & ~1), st_cand = st_w - 4; /* words of a part that are staged */
    const float st_rcp = 1.0f / (float) st_w;
    auto part_of = [&](int t, int &i) { /* which part staged word t is of, and its place behind that part's record */
        const int k = quotient(t, st_w, st_rcp);
        i           = t - k * st_w - 4;
        return k;
    };
    constexpr int      kOwnWords = kStageWords / kThreads;
    unsigned long long tv[kOwnWords];
    /* a segment per thread: asked for with the records, where the first row, or the one before any other, is a temperature row (temp); a
     * temperature row behind one of another kind reads its segments further down, as rows of more segments do */
    const bool by_segs = !kFast && temp && p.n_slices * kWarps <= kThreads;
    float      seg_ref = 0.0f;
    double     seg_sum = 0.0;
    {
        /* one round trip: the records and the first candidates of the parts, whatever their counts are, and the parameters of a row
         * behind the first (with a round trip of their own: 2000 x 16384 top-k 40, unhinted, 87.8 us, so 82.3) */
#pragma unroll
        for (int q = 0; q < kStageWords / kThreads; q++) {
            int       i;
            const int t = g.tid + q * kThreads, k = part_of(t, i);
            tv[q]       = q * kThreads < st_parts * st_w && k < st_parts ? __ldcg(reinterpret_cast<const unsigned long long *>(part_rec(p, row, k)) + 4 + i) : 0ull;
        }
        if (by_segs && g.tid < p.n_slices * kWarps) {
            const SegRec *seg = p.segs + (size_t) row * (size_t) (p.n_slices * kWarps) + g.tid;
            seg_ref           = __ldcg(&seg->ref);
            seg_sum           = __ldcg(&seg->sum);
        }
        RawCfg rc{};
        if (!first && g.tid == 0) {
            rc = raw_config(p, row, true);
        }
#pragma unroll
        for (int q = 0; q < kStageWords / kThreads; q++) {
            if (q * kThreads < st_parts * st_w) {
                sh->stage[g.tid + q * kThreads] = tv[q];
            }
        }
        if (!first && g.tid == 0) {
            sh->cfg  = finish_config(p, row, rc);
            sh->rng0 = rc.rng;
            not_wide<kFast>(p, sh);
        }
    }
    g.sync();
    unsigned long long rng = r.rng;
    if (n_parts > kMaxParts) {
        /* a row spread over that many thread blocks (a handful of rows on the whole chip): its maximum is
         * taken from the records one by one, everything else is left to the multi-pass path */
        float m = -CUDART_INF_F;
        int   a = 0x7fffffff;
        for (int i = g.tid; i < n_parts; i += g.n) {
            const int4  h  = __ldcg(part_rec(p, row, i));
            const float pm = __int_as_float(h.x);
            st |= h.w;
            if (pair_before(pm, h.y, m, a)) {
                m = pm;
                a = h.y;
            }
        }
        st = __reduce_or_sync(0xffffffffu, st);
        if (g.lane == 0) {
            gs->wred_l[g.warp] = st;
        }
        group_argmax(g, gs, m, a);
        for (int w = 0; w < g.nw; w++) {
            st |= (int) gs->wred_l[w];
        }
        if (r.mode == M_ARGMAX) {
            if (g.tid == 0) {
                p.tokens[row] = a + p.vocab_offset;
                if (p.kept_cap > 0) {
                    p.kept_n[row] = 0;
                }
            }
            return st;
        }
        if (g.tid == 0) {
            gs->blk_max = m;
            gs->blk_arg = a;
        }
        g.sync();
        return st | ST_DEFERRED;
    }
    /* The parts' records, two per lane, by every warp for itself: one after the other they took a microsecond of a row of
     * sixteen parts. Rows of up to kMaxParts parts have all their records among the staged words. */
    static_assert(kMaxParts == 64 && kStageWords / kMaxParts >= 4, "two parts per lane, their records are staged");
    unsigned max_key = 0u, tau_key = 0u;
    int      row_arg = 0x7fffffff, others = 0;
    bool     overflow = false;
    {
        int args[2], more[2];
        unsigned keys[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int part = g.lane + 32 * h;
            keys[h]        = 0u;
            args[h]        = 0x7fffffff;
            more[h]        = 0;
            if (part < n_parts) {
                const int4 a = *reinterpret_cast<const int4 *>(&sh->stage[part * st_w]), b = *reinterpret_cast<const int4 *>(&sh->stage[part * st_w + 2]);
                keys[h] = order_key(__int_as_float(a.x));
                args[h] = a.y;
                overflow |= a.z > kPartCand;
                more[h] = max(0, min(a.z, kPartCand + 1) - st_cand); /* what is not staged */
                st |= a.w;
                tau_key = max(tau_key, order_key(__int_as_float(b.x)));
            }
        }
        max_key  = __reduce_max_sync(0xffffffffu, max(keys[0], keys[1]));
        row_arg  = __reduce_min_sync(0xffffffffu, min(keys[0] == max_key ? args[0] : 0x7fffffff, keys[1] == max_key ? args[1] : 0x7fffffff)); /* rows that are not greedy carry no id */
        st       = __reduce_or_sync(0xffffffffu, st);
        overflow = __any_sync(0xffffffffu, overflow);
        if (r.mode == M_TOPK || r.mode == M_TOPP) {
            tau_key = __reduce_max_sync(0xffffffffu, tau_key);
            others  = __reduce_add_sync(0xffffffffu, more[0] + more[1]);
            if (others > 0 && g.warp == 0) { /* for the passes over candidates that are not staged */
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    int upto = more[h];
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int up = __shfl_up_sync(0xffffffffu, upto, o);
                        upto += g.lane >= o ? up : 0;
                    }
                    const int base = h == 0 ? 0 : __reduce_add_sync(0xffffffffu, more[0]);
                    if (g.lane + 32 * h < n_parts) {
                        sh->poff[g.lane + 32 * h] = base + upto - more[h];
                    }
                }
            }
        }
    }
    const float row_max = key_to_float(max_key), tau_row = key_to_float(tau_key);

    if (r.mode == M_ARGMAX) {
        if (g.tid == 0) {
            p.tokens[row] = row_arg + p.vocab_offset;
            if (p.kept_cap > 0) {
                p.kept_n[row] = 0;
            }
        }
        return st;
    }

    if (kFast && r.mode != M_TOPK) {
        return st | ST_DEFERRED; /* temperature and top-p rows: the general finishing kernel's */
    }
    if constexpr (!kFast) {
    if (r.mode == M_TEMP) {
        /* segment sums (one per warp and slice, ids in order), moved from their own maximum to the row maximum */
        const int     nseg   = p.n_slices * kWarps;
        const SegRec *segs   = p.segs + (size_t) row * (size_t) nseg;
        auto          seg_at = [&](int t) {
            const float  ref = __ldcg(&segs[t].ref);
            const double sm  = __ldcg(&segs[t].sum);
            return sm * ref_move(ref, row_max, r.inv_t);
        };
        int    found = -1;
        double u, fbase = -CUDART_INF; /* nothing crosses: the walk ends on its last id */
        if (by_segs) {
            /* a segment per thread: its sum is read and moved once, the scan's total is the row's sum */
            const double val  = g.tid < nseg ? seg_sum * ref_move(seg_ref, row_max, r.inv_t) : 0.0;
            double       incl = val;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double up = __shfl_up_sync(0xffffffffu, incl, o);
                if (g.lane >= o) {
                    incl += up;
                }
            }
            if (g.lane == 31) {
                gs->wred_d[g.warp] = incl;
            }
            if (g.tid == 0) {
                gs->pick = -1;
            }
            g.sync();
            double S = 0.0, woff = 0.0;
#pragma unroll
            for (int w = 0; w < kWarps; w++) {
                woff = w == g.warp ? S : woff;
                S += gs->wred_d[w];
            }
            u = (double) unit_from(xorshift_next(rng)) * S;
            /* The first segment whose end lies beyond u. Every thread has the same sums up to each warp and, as lane 31's, with it:
             * one warp takes it. Which of its lanes is asked of those that add something; their sums may end a last bit away from
             * lane 31's, and the last of them takes it where none of theirs lies beyond u. */
            const unsigned over = __ballot_sync(0xffffffffu, u < incl + woff);
            if ((over >> 31) != 0u && !(u < woff)) {
                const unsigned adds = __ballot_sync(0xffffffffu, val > 0.0);
                if (g.lane == ((over & adds) != 0u ? __ffs(over & adds) - 1 : 31 - __clz(adds))) {
                    gs->pick = g.tid;
                    gs->S    = incl + woff - val;
                }
            }
            g.sync();
            found = gs->pick;
            fbase = found >= 0 ? gs->S : fbase;
        } else {
            double part = 0.0;
            for (int t = g.tid; t < nseg; t += g.n) {
                part += seg_at(t);
            }
            const double S = group_sum_d(g, gs, part);
            u = (double) unit_from(xorshift_next(rng)) * S;
            double carry = 0.0;
            for (int t0 = 0; t0 < nseg; t0 += g.n) {
                const int    t    = t0 + g.tid;
                const double val  = t < nseg ? seg_at(t) : 0.0;
                double       incl = val;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double up = __shfl_up_sync(0xffffffffu, incl, o);
                    if (g.lane >= o) {
                        incl += up;
                    }
                }
                g.sync();
                if (g.lane == 31) {
                    gs->wred_d[g.warp] = incl;
                }
                if (g.tid == 0) {
                    gs->pick = 0x7fffffff;
                }
                g.sync();
                double woff = carry;
                for (int w = 0; w < g.warp; w++) {
                    woff += gs->wred_d[w];
                }
                incl += woff;
                if (val > 0.0 && u < incl) {
                    atomicMin(&gs->pick, t);
                }
                g.sync();
                const int pk = gs->pick;
                if (pk != 0x7fffffff) {
                    if (t == pk) {
                        gs->S = incl - val;
                    }
                    g.sync();
                    found = pk;
                    fbase = gs->S;
                    break;
                }
                for (int w = 0; w < g.nw; w++) {
                    carry += gs->wred_d[w];
                }
            }
        }
        if (found < 0) {
            found = nseg - 1;
        }
        /* the crossing segment, re-read from the row (L2), penalised, walked with the row maximum */
        const int    cc    = found / kWarps, w = found % kWarps;
        const int    s0c   = cc * p.slice;
        const int    nc    = max(0, min(p.slice, p.V - s0c));
        const int    nv4c  = (nc + 3) >> 2;
        const int    Lc    = share_len(nv4c);
        const int    e0    = min(4 * w * Lc, nc);
        const int    e1    = min(4 * min((w + 1) * Lc, nv4c), nc);
        const int    seg_n = max(e1 - e0, 0);
        const float *src   = row_again(p, row) + s0c + e0;
        /* every thread takes a run of consecutive entries; the runs' sums are scanned over the group and the thread whose run
         * crosses u walks it */
        const int per = (seg_n + g.n - 1) / g.n; /* <= 4 */
        const int i0  = g.tid * per;
        float     ev[4];
        g.sync();
        if (r.pen_on) {
            constexpr int kSegMost = kSliceMax / kWarps; /* entries of a segment, and so distinct ids in it */
            static_assert(kSegMost * (sizeof(float) + sizeof(PenEntry)) <= (size_t) kFinBytes, "a segment and its ids fit");
            float    *wbuf = reinterpret_cast<float *>(cmem);
            PenEntry *ids  = reinterpret_cast<PenEntry *>(wbuf + kSegMost);
            for (int i = g.tid; i < seg_n; i += g.n) {
                wbuf[i] = prologue_one(src[i], s0c + e0 + i, r.cap, r.mrow);
            }
            for (int i = g.tid; i < kFinBitmapWords; i += g.n) {
                sh->fin_bitmap[i] = 0u;
            }
            if (g.tid == 0) {
                gs->n_dlist = 0;
            }
            g.sync();
            if (seg_n > 0) {
                st |= apply_penalties(g, wbuf, s0c + e0, seg_n, r, p.V, p.vocab_offset, sh->fin_bitmap, ids, kSegMost, &gs->n_dlist, false, 0);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                ev[q] = q < per && i0 + q < seg_n ? wbuf[i0 + q] : -CUDART_INF_F;
            }
        } else { /* nothing to change: each thread reads its own */
#pragma unroll
            for (int q = 0; q < 4; q++) {
                ev[q] = q < per && i0 + q < seg_n ? prologue_one(src[i0 + q], s0c + e0 + i0 + q, r.cap, r.mrow) : -CUDART_INF_F;
            }
        }
        {
            double mine = 0.0;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                ev[q] = q < per && i0 + q < seg_n ? expf(scaled_arg(ev[q], row_max, r.inv_t)) : 0.0f;
                mine += (double) ev[q];
            }
            double incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double up = __shfl_up_sync(0xffffffffu, incl, o);
                if (g.lane >= o) {
                    incl += up;
                }
            }
            if (g.lane == 31) {
                gs->wred_d[g.warp] = incl;
            }
            g.sync();
            u           = u < fbase ? fbase : u; /* the difference that fbase is may be a last bit too large */
            double base = fbase, upto = fbase;   /* up to the thread's warp, and in all */
#pragma unroll
            for (int ww = 0; ww < kWarps; ww++) {
                base = ww == g.warp ? upto : base;
                upto += gs->wred_d[ww];
            }
            const unsigned over = __ballot_sync(0xffffffffu, u < base + incl);
            if (u < upto) {
                if ((over >> 31) != 0u && !(u < base)) { /* one warp takes it, and which of its lanes is asked as above */
                    const unsigned adds = __ballot_sync(0xffffffffu, mine > 0.0);
                    if (g.lane == ((over & adds) != 0u ? __ffs(over & adds) - 1 : 31 - __clz(adds))) {
                        double a   = base + (incl - mine);
                        int    hit = i0;
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            a += (double) ev[q];
                            hit = ev[q] > 0.0f ? i0 + q : hit;
                            if (ev[q] > 0.0f && u < a) {
                                break;
                            }
                        }
                        p.tokens[row] = s0c + e0 + hit + p.vocab_offset;
                    }
                }
            } else {
                /* The segment's share came out a hair larger than its entries add up to: the last entry that adds something. Nothing
                 * does, or the row's sum is no number: its last id, as the reference's walk ends. */
                if (g.tid == 0) {
                    gs->pick = -1;
                }
                g.sync();
                int last = -1;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    last = ev[q] > 0.0f ? i0 + q : last;
                }
                last = __reduce_max_sync(0xffffffffu, u == u ? last : -1);
                if (g.lane == 0 && last >= 0) {
                    atomicMax(&gs->pick, last);
                }
                g.sync();
                if (g.tid == 0) {
                    p.tokens[row] = max(s0c + e0 + (gs->pick >= 0 ? gs->pick : seg_n - 1), 0) + p.vocab_offset;
                }
            }
            if (g.tid == 0 && p.kept_cap > 0) {
                p.kept_n[row] = 0;
            }
        }
        g.sync();
        return st;
    }

    }
    /* ---- top-k and top-p: merge the parts' candidates ---- */
    bool need_multipass = !(r.kq > 0 && r.kq <= kFastKMax) || overflow; /* what counts is how many stay above the row's threshold: checked below */
    const bool keep_all = r.mode == M_TOPP; /* every marked entry was left out of the bulk sums */
    const float u01     = unit_from(xorshift_next(rng)); /* the row's draw */
    int         n_rank  = 0;   /* entries of cbuf, the kq best among them; top-p: their probabilities */
    float       rank_hi = row_max;
    static_assert(kStageWords <= kFinCap, "what is staged fits the list");
    if (!need_multipass && others == 0) {
        /* All candidates came in with the records, four words per thread. Those that cannot be among the kq best, by the bins
         * their values fall into, are dropped where they are; the rest is ranked. Bound by latency: three barriers and a dozen
         * shared-memory round trips. From the records to the token, one row of 128256 in 16 parts, top-k 40: 8.0 -> 5.1 us (the
         * parts one after the other, lists written and read between the steps, one thread over the weights); 64 x 32000 top-k 40
         * in 4 parts each 18.0 -> 14.0 us a pass, 4 x 128256 top-p 19.0 -> 14.9. */
        const float range = row_max - tau_row, scale = row_max > tau_row && range < CUDART_INF_F ? (float) kHistBins / range : 0.0f;
        int         bin[kOwnWords]; /* -1: nothing to keep */
        float       v[kOwnWords];
        double      part = 0.0;
#pragma unroll
        for (int q = 0; q < kOwnWords; q++) {
            int       i;
            const int t = g.tid + q * kThreads, k = part_of(t, i), held = k < n_parts ? (int) (unsigned) sh->stage[k * st_w + 1] : 0;
            v[q]   = __uint_as_float((unsigned) tv[q]);
            bin[q] = i >= 0 && i < held && (keep_all || v[q] >= tau_row) ? min(kHistBins - 1, max(0, __float2int_rz((v[q] - tau_row) * scale))) : -1;
            if (bin[q] >= 0) {
                atomicAdd(&sh->bhist[bin[q]], 1);
            }
        }
        if constexpr (!kFast) {
            if (r.mode == M_TOPP) { /* the candidates' weights, exact, and what the parts added up of the rest */
#pragma unroll 1
                for (int q = 0; q < kOwnWords; q++) {
                    const bool one = bin[q] >= 0;
                    if (__any_sync(0xffffffffu, one)) {
                        const float e = exp_exact(scaled_arg(v[q], row_max, r.inv_t));
                        v[q]          = e;
                        part += one ? (double) e : 0.0;
                    }
                }
                if (g.tid < n_parts) {
                    const unsigned long long *rec = &sh->stage[g.tid * st_w + 2];
                    part += ref_move(__uint_as_float((unsigned) (rec[0] >> 32)), row_max, r.inv_t) * __longlong_as_double((long long) rec[1]);
                }
                part = warp_sum_d(part);
                if (g.lane == 0) {
                    gs->wred_d[g.warp] = part;
                }
            }
        }
        g.sync();
        const int few_min = top_bin(sh->bhist, g.lane, r.kq);
        double    S       = 0.0;
        if constexpr (!kFast) {
            if (r.mode == M_TOPP) {
#pragma unroll
                for (int w = 0; w < kWarps; w++) {
                    S += gs->wred_d[w];
                }
                rank_hi = __double2float_rn(1.0 / S); /* the row's maximum is a candidate */
                if (g.tid == 0) {
                    sh->wide_S = S;
                }
            }
        }
        unsigned in[kOwnWords];
        int      mine = 0;
#pragma unroll
        for (int q = 0; q < kOwnWords; q++) {
            in[q] = __ballot_sync(0xffffffffu, bin[q] >= 0 && bin[q] >= few_min);
            mine += __popc(in[q]);
        }
        int at = g.lane == 0 && mine > 0 ? atomicAdd(&sh->n_sel, mine) : 0;
        at     = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
        for (int q = 0; q < kOwnWords; q++) {
            const int pos = at + __popc(in[q] & ((1u << g.lane) - 1u));
            if (((in[q] >> g.lane) & 1u) != 0u) {
                cbuf[pos] = Pair{!kFast && r.mode == M_TOPP ? __double2float_rn((double) v[q] / S) : v[q], (int) (tv[q] >> 32)}; /* top-p: p_i as the reference normalises it */
            }
            at += __popc(in[q]);
        }
        g.sync();
        need_multipass = sh->n_sel < r.kq;
        n_rank         = sh->n_sel;
    }
    if (!need_multipass && others > 0) {
        /* The candidates of all parts are merged in up to three passes of one rolled loop. The first keeps what
         * passes the row's threshold (the largest of the parts' thresholds). A row cut into many parts can have far
         * more of those than k (every part kept at least k of its own): if they do not fit, a second pass bins them
         * by value between the threshold and the row's maximum, and a third keeps the bins from the top down to the
         * one in which the kq-th falls. */
        float bin_scale = 0.0f;
        int   bin_min   = 0;
        auto  bin_of    = [&](float v) { return min(kHistBins - 1, max(0, __float2int_rz((v - tau_row) * bin_scale))); };
        int   pass      = 0; /* 0 keep by threshold, 1 bin, 2 keep by bin */
        /* The whole warp calls: the entries that stay are counted over the warp and get their places with one atomic
         * per warp. */
        auto place = [&](bool valid, const Pair &e) {
            bool keep = valid && (keep_all || e.v >= tau_row);
            if (pass == 1) {
                if (keep) {
                    atomicAdd(&sh->bhist[bin_of(e.v)], 1);
                }
                return;
            }
            if (pass == 2) {
                keep = keep && bin_of(e.v) >= bin_min;
            }
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            if (m == 0u) {
                return;
            }
            int base = 0;
            if (g.lane == 0) {
                base = atomicAdd(&sh->n_ent, __popc(m));
            }
            const int pos = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << g.lane) - 1u));
            if (keep && pos < kFinCap) {
                cbuf[pos] = e;
            }
        };
        int total = 0;
#pragma unroll 1
        for (pass = 0; pass < 3; pass++) {
            if (g.tid == 0) {
                sh->n_ent = 0;
            }
            if (pass == 1 && g.tid < kHistBins) {
                sh->bhist[g.tid] = 0;
            }
            g.sync();
            /* what is staged, then one loop over the rest of all parts (rolled: code that runs once per row costs what it weighs) */
#pragma unroll 1
            for (int t0 = 0; t0 < st_parts * st_w; t0 += kThreads) {
                int                      i;
                const int                t = t0 + g.tid, k = part_of(t, i);
                const bool               ok = k < st_parts && i >= 0 && i < (int) (unsigned) sh->stage[min(k, st_parts - 1) * st_w + 1];
                const unsigned long long w  = ok ? sh->stage[t] : 0ull;
                place(ok, Pair{__uint_as_float((unsigned) w), (int) (w >> 32)});
            }
#pragma unroll 1
            for (int f0 = 0; f0 < others; f0 += g.n) {
                const int  f  = f0 + g.tid;
                const bool ok = f < others;
                /* the last part that begins at f or before: offsets ascend. One after the other they were most of a row of many
                 * parts: 2 x 262144 in 32 parts, top-k 256, 156 -> 107 us. */
                int pi = 0;
#pragma unroll
                for (int step = kMaxParts / 2; step > 0; step >>= 1) {
                    if (pi + step < n_parts && f >= sh->poff[pi + step]) {
                        pi += step;
                    }
                }
                const int i = f - sh->poff[pi] + (pi < st_parts ? st_cand : 0);
                Pair      e{0.0f, 0};
                if (ok) {
                    const unsigned long long w = __ldcg(reinterpret_cast<const unsigned long long *>(part_rec(p, row, pi)) + 4 + i);
                    e.v                        = __uint_as_float((unsigned) w);
                    e.idx                      = (int) (w >> 32);
                }
                place(ok, e);
            }
            g.sync();
            if (pass == 1) { /* the bin in which the kq-th candidate from the top falls */
                if (g.warp == 0) {
                    const int bb = top_bin(sh->bhist, g.lane, r.kq);
                    if (g.lane == 0) {
                        gs->b_star = bb;
                    }
                }
                g.sync();
                bin_min = gs->b_star;
                g.sync();
                if (bin_min <= 0) {
                    break; /* nothing to gain: the candidates sit in the lowest bin (many equal values) */
                }
                continue;
            }
            total = sh->n_ent;
            if (pass == 2 || total <= kFinCap || keep_all || !(row_max > tau_row) || !(row_max - tau_row < CUDART_INF_F)) {
                break;
            }
            bin_scale = (float) kHistBins / (row_max - tau_row);
            g.sync(); /* every thread has read n_ent: the next pass puts it back to zero */
        }
        PROF(10);
        if (total > kFinCap || total < r.kq) {
            need_multipass = true;
        }
        n_rank = total;
        if constexpr (!kFast) {
            if (!need_multipass && r.mode == M_TOPP) {
                /* Candidates get their exact e_i relative to the row maximum; the rest of the row was summed per part relative
                 * to the part's own maximum and is rescaled here. */
                double part = 0.0;
                for (int i = g.tid; i < total; i += g.n) {
                    const float e = exp_exact(scaled_arg(cbuf[i].v, row_max, r.inv_t));
                    cbuf[i].v     = e;
                    part += (double) e;
                }
                if (g.tid < n_parts) {
                    const unsigned long long *rec = &sh->stage[g.tid * st_w + 2];
                    part += ref_move(__uint_as_float((unsigned) (rec[0] >> 32)), row_max, r.inv_t) * __longlong_as_double((long long) rec[1]);
                }
                const double S = group_sum_d(g, gs, part);
                if (g.tid == 0) {
                    sh->wide_S = S;
                }
                rank_hi = __double2float_rn(1.0 / S);
                for (int i = g.tid; i < total; i += g.n) {
                    cbuf[i].v = __double2float_rn((double) cbuf[i].v / S); /* p_i as the reference normalises it */
                }
                g.sync();
            }
        }
    }
    if (!need_multipass) { /* in order, (value or p desc, id asc); top-k: and the weights of the softmax over the k kept logits (sampler.c:217-222) */
        const bool weigh = r.mode == M_TOPK && !r.select_only;
        if (n_rank <= kRankFew) {
            if (weigh) {
                rank_few<true>(cbuf, n_rank, r.kq, r.inv_t, sh->fsort, sh->fq);
            } else {
                rank_few<false>(cbuf, n_rank, r.kq, r.inv_t, sh->fsort, sh->fq);
            }
        } else {
            rank_in_bins(cbuf, n_rank, r.kq, tau_row, rank_hi, r.mode == M_TOPP, cbuf + kFinCap, reinterpret_cast<int *>(cbuf + 2 * kFinCap), sh->fsort);
            g.sync();
            if (weigh) {
                const float m = sh->fsort[0].v;
                for (int i = g.tid; i < r.kq; i += g.n) {
                    sh->fq[i] = exp_exact(scaled_arg(sh->fsort[i].v, m, r.inv_t));
                }
            }
        }
        g.sync();
    }
    if (!need_multipass && r.mode == M_TOPK) {
        PROF(11);
        const int k = r.k;
        if (r.select_only) {
            for (int i = g.tid; i < min(k, p.kept_cap); i += g.n) {
                kept_i[i] = sh->fsort[i].idx + p.vocab_offset;
                kept_v[i] = sh->fsort[i].v;
            }
            if (g.tid == 0) {
                p.kept_n[row] = k;
                p.tokens[row] = sh->fsort[0].idx + p.vocab_offset;
            }
            g.sync();
            return st;
        }
        if (g.warp == 0) { /* one draw */
            double    S;
            const int pick = draw_sorted(g.lane, sh->fq, k, u01, &S);
            if (g.lane == 0) {
                p.tokens[row] = sh->fsort[pick].idx + p.vocab_offset;
                gs->S         = S;
                if (p.kept_cap > 0) {
                    p.kept_n[row] = k;
                }
            }
        }
        if (p.kept_cap > 0) {
            g.sync();
            const double S = gs->S;
            for (int i = g.tid; i < min(k, p.kept_cap); i += g.n) {
                kept_i[i] = sh->fsort[i].idx + p.vocab_offset;
                kept_v[i] = __double2float_rn((double) sh->fq[i] / S);
            }
        }
        g.sync();
        return st;
    }
    if constexpr (!kFast) {
        if (!need_multipass) { /* top-p over a small nucleus (sampler.c:245-300) */
            const int kq = r.kq;
            /* The walks over the kq entries, one per lane of a warp. Their running sums are exact wherever no entry is smaller
             * than 2^-29, so the order of additions is not seen; one thread that adds them one by one, three times over,
             * took 4 us of a row's 15. */
            static_assert(kNucleusProbe <= 32, "an entry per lane");
            if (g.warp == 0) {
                const Pair e    = g.lane < kq ? sh->fsort[g.lane] : Pair{0.0f, 0};
                double     cum  = (double) e.v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double up = __shfl_up_sync(0xffffffffu, cum, o);
                    if (g.lane >= o) {
                        cum += up;
                    }
                }
                const float    p_floor = __shfl_sync(0xffffffffu, e.v, kq - 1); /* nothing outside fsort has a larger p */
                const unsigned reached = __ballot_sync(0xffffffffu, g.lane < kq && cum >= (double) r.top_p);
                const bool     all_in  = kq >= p.V && __shfl_sync(0xffffffffu, cum, kq - 1) >= 0.0; /* no numbers: nothing of this is in order */
                /* never reached top_p: the nucleus is the whole row, if all of it is here */
                const int      cut = reached != 0u ? __ffs(reached) : (all_in ? kq : -1);
                const float    p_cut = __shfl_sync(0xffffffffu, e.v, max(cut - 1, 0));
                const bool     ok    = cut > 0 && (reached == 0u || p_cut > p_floor || all_in);
                if (ok) {
                    if (g.lane == 0) {
                        atomicAdd(&p.wide_head->rows, 1ull); /* the row is not wide: said as early as it is known */
                    }
                    const double   N    = __shfl_sync(0xffffffffu, cum, cut - 1);
                    const double   u    = (double) u01 * N;
                    const unsigned over = __ballot_sync(0xffffffffu, g.lane < cut && u < cum);
                    const int      pick = over != 0u ? __ffs(over) - 1 : cut - 1;
                    if (g.lane == pick) {
                        p.tokens[row] = e.idx + p.vocab_offset;
                    }
                    if (p.kept_cap > 0) {
                        if (g.lane == 0) {
                            p.kept_n[row] = cut;
                        }
                        if (g.lane < min(cut, p.kept_cap)) {
                            kept_i[g.lane] = e.idx + p.vocab_offset;
                            kept_v[g.lane] = __double2float_rn((double) e.v / N);
                        }
                    }
                }
                if (g.lane == 0) {
                    gs->flag = ok ? 1 : 0;
                }
            }
            g.sync();
            if (gs->flag) {
                return st;
            }
        }
    }
    g.sync();
    if (g.tid == 0) {
        gs->blk_max = row_max;
        gs->blk_arg = row_arg;
    }
    g.sync();
    return st | ST_DEFERRED;
}

/* ------------------------------------------------------------------ kernel -- */

/*
 * A lower bound of the kq-th largest of the threads' keys (one each, two with `two`) that kq of them reach and few more: the keys
 * are counted in kKeyBins bins between the smallest and the largest, and where the bin that the kq-th falls into holds too many,
 * once more between that bin's ends. `bins` is zero when this is called. Bound by latency: two barriers, an atomic and a scan
 * (0.84 us of one row of 4096) where building the key bit by bit took a barrier for each of about ten bits (1.25 - 1.5 us).
 * Ordered lists per warp, and halving in all of them, took as long as this alone on an SM and 0.3 us longer with another thread
 * block beside it: every instruction of it is issued by all eight warps. All threads call.
 */
__device__ __forceinline__ unsigned kth_key(unsigned key0, unsigned key1, bool two, int kq, int *bins, uint2 *ends, int lane, int warp) {
    unsigned lo = __reduce_min_sync(0xffffffffu, two ? min(key0, key1) : key0), hi = __reduce_max_sync(0xffffffffu, two ? max(key0, key1) : key0);
    if (lane == 0) {
        ends[warp] = make_uint2(lo, hi);
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        const uint2 e = ends[w];
        lo            = min(lo, e.x);
        hi            = max(hi, e.y);
    }
    int need = kq; /* of the keys from lo to hi */
    for (;;) {
        const int shift = max(0, 32 - __clz(hi - lo) - 9); /* (hi - lo) >> shift < kKeyBins */
        static_assert(kKeyBins == 1 << 9 && kKeyBins == 16 * 32, "sixteen bins per lane");
        if (key0 - lo <= hi - lo) {
            atomicAdd(&bins[(key0 - lo) >> shift], 1);
        }
        if (two && key1 - lo <= hi - lo) {
            atomicAdd(&bins[(key1 - lo) >> shift], 1);
        }
        __syncthreads();
        int4 c[4]; /* the lane's bins */
        int  sum = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            c[i] = reinterpret_cast<const int4 *>(bins)[4 * lane + i];
            sum += (c[i].x + c[i].y) + (c[i].z + c[i].w);
        }
        int up = sum; /* keys in the lane's bins and above */
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int more = __shfl_down_sync(0xffffffffu, up, o);
            up += lane + o < 32 ? more : 0;
        }
        const int from = 31 - __clz(__ballot_sync(0xffffffffu, up >= need)); /* the last lane from which up enough are */
        /* in it: the last of its bins from which up enough are, and how many are from there up */
        int b = 0, n = up, above = up - sum;
#pragma unroll
        for (int i = 3; i >= 0; i--) {
            const int q[4] = {c[i].x, c[i].y, c[i].z, c[i].w};
#pragma unroll
            for (int j = 3; j >= 0; j--) {
                const bool before = above < need;
                above += q[j];
                if (before && above >= need) {
                    b = 4 * i + j;
                    n = above;
                }
            }
        }
        b = __shfl_sync(0xffffffffu, 16 * lane + b, from);
        n = __shfl_sync(0xffffffffu, n, from);
        const unsigned key = lo + ((unsigned) b << shift);
        if (n - need <= 4 + kq / 4 || shift == 0) {
            return key;
        }
        const int in = bins[b];
        __syncthreads(); /* every warp has read the bins */
        for (int i = (int) threadIdx.x; i < kKeyBins; i += kThreads) {
            bins[i] = 0;
        }
        __syncthreads();
        need -= n - in;
        lo = key;
        hi = min(hi, key + ((1u << shift) - 1u));
    }
}

/* The part's maximum, as its candidates are. */
__device__ __forceinline__ float part_top(const StreamShared *sh, bool cap_late) {
    unsigned long long b = 0ull;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        b = max(b, sh->best[w]);
    }
    const float top = key_to_float((unsigned) (b >> 32));
    return cap_late && top > -CUDART_INF_F ? soft_cap(top, sh->cap) : top;
}

/* The largest of the warps' references of a part. */
__device__ __forceinline__ float part_ref(const StreamShared *sh) {
    float m = -CUDART_INF_F;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        m = fmaxf(m, sh->wb_ref[w]);
    }
    return m;
}

/* Two floats at a time: the same operations, rounded the same, in half the instructions. */
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

/* The terms of a float4 (sum_term's, two at a time), added up as every place that forms them adds them up. */
__device__ __forceinline__ float sum_terms(const float4 &x, const SumScale &k, float ref) {
    const unsigned long long less = pack2(-ref, -ref), hi = pack2(k.hi, k.hi), lo = pack2(k.lo, k.lo);
    const unsigned long long a = add2(pack2(x.x, x.y), less), b = add2(pack2(x.z, x.w), less);
    float                    t0, t1, t2, t3;
    unpack2(fma2(a, lo, mul2(a, hi)), t0, t1);
    unpack2(fma2(b, lo, mul2(b, hi)), t2, t3);
    return __fadd_rn(__fadd_rn(exp2_fast(t0), exp2_fast(t1)), __fadd_rn(exp2_fast(t2), exp2_fast(t3)));
}

/*
 * A part whose candidates outran their list: its large values lie with a few threads (a row sorted along its ids, say),
 * so the thread maxima let too many through. The threshold becomes the part's kq-th largest value, or less where the
 * list has room for what reaches that: its key is built byte by byte from counts of the values that reach tau, read
 * again in the groups that do; then the candidates are taken once more. Only equal values outrun the list now. All
 * threads call; the caller's barrier follows. Out of line: rare, and in line its code cost every part of a row of a
 * slice 2 - 4 %.
 */
__device__ __noinline__ float raise_threshold(const SampleParams &p, StreamShared *sh, float tau) {
    __syncthreads(); /* the part's description is there */
    const PartAgain &a = sh->again;
    const int      tid = (int) threadIdx.x, lane = tid & 31, per_log = kNV4Log + a.gm_shift, n_grp = sh->n_grp;
    const int      n_full = min(p.slice, p.V), n_last = p.V - (p.n_slices - 1) * p.slice;
    const float   *src    = row_again(p, a.row);
    const SumScale ks     = sum_scale2(a.inv_t);
    int           *bins   = reinterpret_cast<int *>(sh->fin_q);
    unsigned       prefix = 0u;
    int            need   = a.kq;
    for (int level = 3;; level--) { /* the byte that is counted; -1: the candidates are taken */
        __syncthreads(); /* the counts, and before them the candidates, have been read */
        bins[tid] = 0;
        if (tid == 0) {
            sh->n_cand = 0;
        }
        __syncthreads();
        double fix = 0.0;
        for (int t = tid; t < n_grp << per_log; t += kThreads) {
            const int name = sh->grp[t >> per_log], f = t & ((1 << per_log) - 1), w = (name & 255) >> 5;
            const int s = ((name >> 8) << a.gm_shift) + f / kNV4, c = a.c0 + s, i4 = (name & 31) + 32 * (f % kNV4);
            const int n = c == p.n_slices - 1 ? n_last : n_full, nv4 = (n + 3) >> 2, L = share_len(nv4), w4 = min(w * L, nv4);
            if (s >= a.part_len || i4 >= min(L, nv4 - w4)) {
                continue;
            }
            float v[4];
            bool  any = false;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int e = 4 * (w4 + i4) + q, id = c * p.slice + e, off = 4 * i4 + q, bit = id_bit(s, w, off);
                v[q] = -CUDART_INF_F;
                if (e >= n) {
                    continue;
                }
                v[q] = src[id];
                if (a.pro) {
                    v[q] = prologue_one(v[q], id, sh->cap, sh->mrow);
                }
                if (a.pen && ((sh->id_bits[bit >> 5] >> (bit & 31)) & 1u) != 0u) {
                    const int       g   = a.long_ids ? s * kWarps + w : (s & 31) * kWarps + w;
                    const int       lo  = a.long_smem ? sh->rl_cnt[g] : a.long_off[g], hi = a.long_smem ? sh->rl_cnt[g + 1] : a.long_off[g + 1];
                    for (int i = lo; i < hi; i++) {
                        if ((int) (a.list[i] & 0x3ffu) == off && (a.long_ids || (int) (a.list[i] >> kTagAt) == s >> 5)) {
                            v[q] = penalise_rcp(v[q], (int) ((a.list[i] >> 10) & (a.long_ids ? 0x3fffffu : 0x7ffu)), a.rep_rcp, a.rep, a.freq, a.pres);
                        }
                    }
                }
                if (v[q] >= tau) {
                    const unsigned key = order_key(v[q]);
                    if (level < 0) {
                        const int pos = atomicAdd(&sh->n_cand, 1);
                        if (pos < kPartCand) {
                            sh->cand[pos].v   = v[q];
                            sh->cand[pos].idx = id;
                        }
                        any = true;
                    } else if (level == 3 || (key >> (8 * level + 8)) == (prefix >> (8 * level + 8))) {
                        atomicAdd(&bins[(key >> (8 * level)) & 255u], 1);
                    }
                }
            }
            if (a.sums && any) { /* as where the candidates are taken first */
                const float u  = s < kSliceRefs ? sh->ref_at[s][w] : p.segs[((size_t) a.row * (size_t) p.n_slices + (size_t) c) * kWarps + w].ref;
                const float u0 = u == -CUDART_INF_F ? 0.0f : u;
                double      now = -(double) sum_terms(make_float4(v[0], v[1], v[2], v[3]), ks, u0);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (!(v[q] >= tau)) {
                        now += (double) sum_term(v[q], ks, u0);
                    }
                }
                fix += now * ref_move(u, part_ref(sh), a.inv_t);
            }
        }
        if (level < 0) {
            if (a.sums) {
                fix = warp_sum_d(fix);
                if (lane == 0) {
                    sh->wb_sum[tid >> 5] = sh->wb_acc[tid >> 5] * ref_move(sh->wb_ref[tid >> 5], part_ref(sh), a.inv_t) + fix;
                }
            }
            return tau;
        }
        __syncthreads();
        const int b     = top_bin(bins, lane, need);
        int       above = 0;
        for (int i = b + 1 + lane; i < 256; i += 32) {
            above += bins[i];
        }
        need -= __reduce_add_sync(0xffffffffu, above);
        prefix |= (unsigned) b << (8 * level);
        if (level == 0 || a.kq - need + bins[b] <= kPartCand) { /* what has a larger key, and this byte's */
            tau   = fmaxf(tau, prefix <= order_key(-CUDART_INF_F) ? -CUDART_INF_F : key_to_float(prefix));
            level = 0;
        }
    }
}

/*
 * A top-k row that went through one thread block as a whole, finished by that thread block from its own candidates
 * (all threads call): put in order, the k best get their exact weights and the draw is made as in finish_row. No
 * candidate lies below lo. Where they outran their list, finish_raised raises the threshold first. What does not fit
 * then (more equal values than the list holds, fewer than k) is handed back with ST_RETRY. What is rare is called out of
 * line and from branches that are there anyway: code that every row jumps over costs rows of a slice 2 - 4 %, code that
 * is called for the first time in a while a microsecond (k = 100 on 256 x 128256: 36.6 us with all of this behind one call).
 */
__device__ __noinline__ void finish_raised(const SampleParams &p, StreamShared *sh, unsigned char *gmem, float lo, bool cap_late, int st_bits);
template <bool kRaise, class Again>
__device__ __forceinline__ void inline_finish_topk(const SampleParams &p, StreamShared *sh, unsigned char *gmem, int row, int total, int k, float lo, bool cap_late, float inv_t, int st_bits,
                                                   Again &&again) {
    const int tid = (int) threadIdx.x;
    const bool ok = total <= kPartCand && total >= k && k <= kFastKMax;
    if constexpr (kRaise) {
        if (!ok && total > kPartCand && lo > -CUDART_INF_F) { /* below -inf there is nothing to raise: fewer than kq threads met a finite value */
            again();
            finish_raised(p, sh, gmem, lo, cap_late, st_bits);
            return;
        }
    }
    if (ok) {
        if (total <= kRankFew) {
            rank_few<true>(sh->cand, total, k, inv_t, sh->fin_s, sh->fin_q);
        } else {
            Pair *srt = reinterpret_cast<Pair *>(gmem); /* the group maxima are done with */
            rank_in_bins(sh->cand, total, k, lo, part_top(sh, cap_late), false, srt, reinterpret_cast<int *>(srt + kPartCand), sh->fin_s);
            __syncthreads();
            const float m = sh->fin_s[0].v;
            for (int i = tid; i < k; i += kThreads) {
                sh->fin_q[i] = exp_exact(scaled_arg(sh->fin_s[i].v, m, inv_t));
            }
        }
        __syncthreads();
    }
    /* The draw, by a warp that has nothing to do at the next row's set-up: the others go there (its first barrier comes before
     * anything that is read here is written again). */
    if (tid >> 5 == kWarps - 1) {
        unsigned long long rng = sh->cur_rng; /* the sequence's word; this row starts cur_rr draws behind it */
        for (int i = 0; i < sh->cur_rr; i++) {
            (void) xorshift_next(rng);
        }
        const float u01 = unit_from(xorshift_next(rng));
        int         tok = -1;
        if (ok) {
            double S;
            tok = sh->fin_s[draw_sorted(tid & 31, sh->fin_q, k, u01, &S)].idx + p.vocab_offset;
        } else {
            st_bits |= ST_RETRY;
        }
        if ((tid & 31) == 0) {
            p.tokens[row] = tok;
            p.status[row] = st_bits;
            if (p.rng_out != nullptr && sh->cur_last) {
                p.rng_out[sh->cur_seq] = rng; /* the word after the sequence's last row */
            }
        }
    }
}

__device__ __noinline__ void finish_raised(const SampleParams &p, StreamShared *sh, unsigned char *gmem, float lo, bool cap_late, int st_bits) {
    const float tau = raise_threshold(p, sh, lo);
    __syncthreads();
    inline_finish_topk<false>(p, sh, gmem, sh->again.row, min(sh->n_cand, kPartCand + 1), sh->again.kq, tau, cap_late, sh->again.inv_t, st_bits, 0);
}

/*
 * A row's parameters cost up to two dependent memory round trips (slot -> parameters and history ids). Warp 0
 * fetches them for the NEXT row of the run with 4-byte asynchronous copies into shared memory, one step per
 * slice of the part in work, so that nothing waits for them when that row begins. The history ids are asked for
 * before the row's history length is known: the first kRowIds words of the session's history row (they exist,
 * whatever the length is), and the tokens fed before this row into a list of their own. `stage`: 0 nothing asked
 * yet, 1 the slot, 2 everything. Called by all lanes of warp 0.
 */
constexpr int kPrefetchDone = 2;
__device__ __forceinline__ void prefetch_step(const SampleParams &p, StreamShared *sh, int row, int lane, int &stage) {
    const int seq0 = p.rows_per_seq == 1 ? row : row / p.rows_per_seq;
    if (stage == 0) {
        if (lane == 0) {
            if (p.slot) {
                copy_word_async(&sh->raw_nxt.seq, &p.slot[seq0]);
            } else {
                sh->raw_nxt.seq = seq0;
            }
        }
        stage = 1;
        if (p.slot) {
            return; /* the slot must arrive first */
        }
    }
    async_copies_wait();
    __syncwarp();
    const int seq = *reinterpret_cast<volatile int *>(&sh->raw_nxt.seq);
    /* a lane per word: a branch per parameter was a kilobyte and a half of code on every launch's way to its first row
     * (run once, it costs its fetch: 64 x 151936 greedy 14.4 -> 14.1 us, one row of 128256 by temperature 13.1 -> 11.8 with its walk in one scan) */
    if (lane >= 1 && lane < kRawWords) {
        static_assert(offsetof(RawCfg, T) == 4 && offsetof(RawCfg, top_p) == 8 && offsetof(RawCfg, top_k) == 12 && offsetof(RawCfg, hist_len) == 16 && offsetof(RawCfg, rep) == 20 &&
                              offsetof(RawCfg, freq) == 24 && offsetof(RawCfg, pres) == 28 && offsetof(RawCfg, cap) == 32 && offsetof(RawCfg, rng) == 40,
                      "raw_word is in the order of the words");
        const unsigned *from = sh->raw_word[lane];
        unsigned       *to   = reinterpret_cast<unsigned *>(&sh->raw_nxt) + lane;
        if (from != nullptr) {
            copy_word_async(to, from + (lane < 10 ? (size_t) seq : 2 * (size_t) seq + (size_t) (lane - 10)));
        } else {
            *to = lane == 5 ? __float_as_uint(1.0f) : lane == 10 ? 1u : 0u;
        }
    }
    if (p.hist) {
        const int hs = (int) min((long long) kRowIds, p.hist_stride);
        const int *from = p.hist + (size_t) seq * (size_t) p.hist_stride;
        if (p.hist_quads) { /* rows of ids on the 16-byte grid */
            for (int t = 4 * lane; t < hs; t += 128) {
                copy_quad_async(&sh->nxt_ids[t], from + t);
            }
        } else {
            for (int t = lane; t < hs; t += 32) {
                copy_word_async(&sh->nxt_ids[t], from + t);
            }
        }
        /* what lies behind them is read where the row begins: L2 is asked for it */
        for (int t = kRowIds + 32 * lane; t < (int) min((long long) kRowIdsMax, p.hist_stride); t += 32 * 32) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(from + t));
        }
    }
    if (p.extra) {
        const int E = min(row - seq0 * p.rows_per_seq, kRowIds);
        for (int t = lane; t < E; t += 32) {
            copy_word_async(&sh->nxt_ext[t], &p.extra[(size_t) seq0 * (size_t) p.extra_stride + 1 + t]);
        }
    }
    stage = kPrefetchDone;
}

/* Which kinds of rows an instantiation of the stream kernel carries the code for: every one carries greedy rows;
 * K_SEL adds the candidate select of top-k rows, K_SUMS the sums of temperature and top-p rows (and top-p's select).
 * A launch whose caller vouched for its rows' kinds (finish_hint) runs the instantiation without the rest: less
 * code to fetch, fewer live registers in the slice loop; likewise a launch without histories runs one without the
 * penalties' code. A row of a kind that is not carried is streamed as a
 * greedy row and reported (ROW_INTERNAL) where the launch's rows are finished. */
constexpr int K_SEL = 1, K_SUMS = 2, K_PEN = 4, K_PLAIN = 8, K_SHORT = 16; /* K_PEN: the launch brings history ids or fed tokens (penalties) */
template <int kKinds>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) sample_stream_kernel(const __grid_constant__ SampleParams p) {
    /* K_PLAIN: rows on the 16-byte grid, no soft cap, mask or logits output; K_SHORT: no row with more ids than the
     * thread block counts by itself. The launch's host side has checked it, the code for the rest is left out. */
    constexpr bool kPlain  = (kKinds & K_PLAIN) != 0;
    const bool     aligned = kPlain || p.aligned != 0;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *ring    = smem_raw;
    StreamShared  *sh      = reinterpret_cast<StreamShared *>(smem_raw + (size_t) kWarps * kStages * kWarpStageBytes);
    unsigned char *gmem    = reinterpret_cast<unsigned char *>(sh + 1); /* what belongs to the part in work alone */
    float         *gmax    = reinterpret_cast<float *>(gmem); /* [kGroupSlots][kThreads] */
    unsigned      *sl_list = reinterpret_cast<unsigned *>(gmem + kGroupBytes); /* long histories: the part's entries of the row's prepared list, when they fit */

    Grp g;
    g.tid  = (int) threadIdx.x;
    g.lane = g.tid & 31;
    g.warp = g.tid >> 5;
    g.n    = kThreads;
    g.nw   = kWarps;
    g.bar  = 0;
    const int      tid = g.tid, lane = g.lane, warp = g.warp;

    /* every thread block takes a contiguous run of the (row, slice) items */
    int my_first, my_count;
    run_of_cta(p, (int) blockIdx.x, my_first, my_count);

    if (tid == 0) {
        for (int w = 0; w < kWarps; w++) {
            for (int s = 0; s < kStages; s++) {
                mbar_init_only(&sh->full[w][s], 1);
            }
        }
        mbar_init_fence();
    }
    if (tid >= 32 && tid < 32 + kRawWords) {
        sh->raw_word[tid - 32] = p.raw_word[tid - 32];
    }
    __syncthreads();
    /* Launched as a programmatic dependent of the kernel before it in the stream: the thread block may have
     * been placed while that kernel's last blocks were still at work. Everything it touches in global memory
     * waits here for that kernel to be complete and visible, so the stream's order is kept; what is saved is
     * the gap between two grids. The kernel behind this one may be placed likewise. */
    if (lane == 0 && aligned) {
        /* While it waits, the thread block asks L2 for what its ring will copy first (the warp's shares of the run's
         * first kStages items, two more of a long run whose rows are not summed: the ring is full long before the first row's parameters are there; in
         * runs of four or five items that delays what is wanted first, 64 x 151936 greedy 14.1 -> 14.8 us, in runs of sixteen
         * it is worth 0.7 of 30.5). Nothing is read: a line that the kernel before this one is still writing arrives in
         * L2 with its stores either way. Back to back this is worth 0.5 us per launch: the last thread blocks of the
         * grid before leave DRAM idle. */
        const int n_full_ = min(p.slice, p.V), n_last_ = p.V - (p.n_slices - 1) * p.slice;
        for (int jj = 0; jj < ((kKinds & K_SUMS) == 0 && my_count >= 12 ? kStages + 2 : min(kStages, my_count)); jj++) {
            const int item = my_first + jj, r_ = item / p.n_slices, c_ = item - r_ * p.n_slices;
            const int n_   = c_ == p.n_slices - 1 ? n_last_ : n_full_;
            const int nv4_ = (n_ + 3) >> 2, L_ = share_len(nv4_);
            const int lo_  = min(warp * L_, nv4_);
            const int b4_  = max(0, min(min(L_, nv4_ - lo_), (n_ >> 2) - lo_));
            if (b4_ > 0) {
                bulk_prefetch_l2(p.logits + (size_t) r_ * (size_t) p.row_stride + (size_t) c_ * (size_t) p.slice + 4 * lo_, (unsigned) b4_ * 16u);
            }
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if ((kKinds & K_SUMS) != 0 && tid == 0 && blockIdx.x == 0 && p.wide_head != nullptr) { /* the finishing kernel's count of rows begins at nothing */
        static_assert(offsetof(WideHead, gave_up) == 16, "the words in front of it are one of 16 bytes");
        *reinterpret_cast<int4 *>(p.wide_head) = make_int4(0, 0, 0, 0);
        p.wide_head->gave_up                   = 0;
        p.wide_head->waited                    = 0;
        p.wide_head->turn                      = 0;
    }
    asm volatile("griddepcontrol.launch_dependents;");
#ifdef GB_PROFILE
    if (tid == 0 && blockIdx.x < 1024) {
        for (int i = 1; i < 16; i++) {
            g_prof[blockIdx.x][i] = 0;
        }
    }
#endif
    PROF(0);

    /* ---- the warp's own ring: lane 0 asks for the warp's share of the item kStages ahead ---- */
    unsigned char *wring = ring + (size_t) warp * kStages * kWarpStageBytes;
    /* a row's slices have one of two shapes: the full one and the row's last one; what the warp owns of each */
    const int n_full = min(p.slice, p.V), n_last = p.V - (p.n_slices - 1) * p.slice;
    int       w4lo_f, mine4_f, w4lo_l, mine4_l;
    {
        const int nv4f = (n_full + 3) >> 2, Lf = share_len(nv4f);
        w4lo_f         = min(warp * Lf, nv4f);
        mine4_f        = min(Lf, nv4f - w4lo_f);
        const int nv4l = (n_last + 3) >> 2, Ll = share_len(nv4l);
        w4lo_l         = min(warp * Ll, nv4l);
        mine4_l        = min(Ll, nv4l - w4lo_l);
    }
    const int    bulk4_f = max(0, min(mine4_f, (n_full >> 2) - w4lo_f)); /* float4 of the share that a bulk copy brings */
    const int    bulk4_l = max(0, min(mine4_l, (n_last >> 2) - w4lo_l));
    const int    row_first = my_first / p.n_slices, c_first = my_first - row_first * p.n_slices;
    int          irow = row_first, ic = c_first, ijj = 0; /* the next item to request */
    const float *isrc = p.logits + (size_t) irow * (size_t) p.row_stride + (size_t) ic * (size_t) p.slice; /* ... and where its slice starts */
    auto issue_next = [&]() {
        const bool last  = ic == p.n_slices - 1;
        const int  b4    = last ? bulk4_l : bulk4_f;
        const int  stage = ijj % kStages;
        if (b4 > 0) {
            mbar_expect_tx(&sh->full[warp][stage], (unsigned) b4 * 16u);
            bulk_g2s(wring + (size_t) stage * kWarpStageBytes, isrc + 4 * (last ? w4lo_l : w4lo_f), (unsigned) b4 * 16u, &sh->full[warp][stage]);
        } else {
            /* Every item moves its stage's barrier on by one phase, also one of which the warp owns nothing: the waits
             * below go by the item's number. A share can be empty in one of the two slice shapes alone (V = 18436:
             * the last warp owns no float4 of a full slice and 191 of the row's last one). */
            mbar_arrive(&sh->full[warp][stage]);
        }
        ijj++;
        ic++;
        isrc += p.slice;
        if (last) {
            ic = 0;
            isrc += p.row_stride - (long long) p.n_slices * p.slice; /* on to the next row */
        }
    };
    /* Rows off the 16-byte grid: the same ring, filled by all lanes with 4-byte asynchronous copies, a group per item. With
     * plain loads of the share in hand and nothing ahead every slice paid its own round trip to memory. */
    auto issue_words = [&]() {
        const bool last = ic == p.n_slices - 1;
        const int  lo   = 4 * (last ? w4lo_l : w4lo_f), m = 4 * (last ? mine4_l : mine4_f), n_ = last ? n_last : n_full;
        float     *dst  = reinterpret_cast<float *>(wring + (size_t) (ijj % kStages) * kWarpStageBytes);
#pragma unroll 8
        for (int i = lane; i < m; i += 32) {
            if (lo + i < n_) {
                copy_word_async(dst + i, isrc + lo + i);
            } else {
                dst[i] = -CUDART_INF_F;
            }
        }
        async_copies_commit();
        ijj++;
        ic++;
        isrc += p.slice;
        if (last) {
            ic = 0;
            isrc += p.row_stride - (long long) p.n_slices * p.slice;
        }
    };
    for (int jj = 0; jj < min(kStages, my_count); jj++) {
        if (!aligned) {
            issue_words();
        } else if (lane == 0) {
            issue_next();
        }
    }

    CYC_INIT();
    int j         = 0;
    int ring_dead = -1; /* the item at which a copy of this warp failed to arrive in time (-1: none) */
    int pf        = 0; /* warp 0: how far the parameters of the row that begins next have been fetched */
    for (int row = row_first, c0 = c_first; j < my_count; row++, c0 = 0) {
        const int  part_len   = min(p.n_slices - c0, my_count - j);
        const bool final_part = j + part_len == my_count;
        /* the table in which a row's ids are counted, the counts of their groups and the marks of changed values: cleared while
         * the row's parameters are on their way, or the row before is drawn from */
        constexpr int kPerT = (kKinds & K_SHORT) != 0 ? 1 : kRowIdsMax / kThreads, kIdSlots = 2 * kRowIds * kPerT; /* ids of a thread */
        int          *id_key = reinterpret_cast<int *>(gmem), *id_cnt = id_key + kIdSlots, *id_n = reinterpret_cast<int *>(sh->grp);
        if ((kKinds & K_PEN) != 0) {
#pragma unroll
            for (int i = 0; i < kGroupBytes / 16; i += kThreads) {
                reinterpret_cast<int4 *>(gmem)[i + tid] = make_int4(0, 0, 0, 0);
            }
            id_n[tid] = 0;
            static_assert(kRowIds == kThreads, "a group's count per thread");
            for (int i = tid; i < kIdBits / 128; i += kThreads) {
                reinterpret_cast<uint4 *>(sh->id_bits)[i] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        CYC(6);
        if (warp == 0) { /* what has not been fetched while the previous part streamed (first part, short parts) */
            while (pf < kPrefetchDone) {
                prefetch_step(p, sh, row, lane, pf);
            }
            async_copies_wait();
            pf = 0;
        }
        __syncthreads();
        PROF_ONCE(1);
        int   mode, kq, n_ids, id[kPerT];
        float inv_t, rep, freq, pres;
        bool  pen_on, pro_on, pro_part, cap_late;
        {
            const RawCfg raw = sh->raw_nxt;
            const RowCfg r   = row_config(p, row, raw, false); /* what the finisher needs more of is derived again when the row is complete */
            mode   = (int) r.mode;
            kq     = r.kq;
            inv_t  = r.inv_t;
            n_ids  = r.H + r.E;
            pen_on = (kKinds & K_PEN) != 0 && r.pen_on && n_ids > 0;
            rep    = r.rep;
            freq   = r.freq;
            pres   = r.pres;
            pro_on = !kPlain && (r.cap > 0.0f || r.mrow != nullptr); /* something happens to a logit before the penalties ... */
            /* ... and it has to while the part streams. The soft cap is monotone: a top-k row that brings no ids is
             * selected from its uncapped logits, and only what is read again is capped: a tanhf, a division and a
             * call per logit less. 48 rows of 262144 columns, half of them masked, top-k 64: 104.6 us a step with every
             * logit capped and 93.8 with these, when they came in (48 since). */
            cap_late = !kPlain && (kKinds & K_SEL) != 0 && r.cap > 0.0f && r.cap < 1e38f && mode == M_TOPK && kq <= kFastKMax && !pen_on && p.out_logits == nullptr;
            pro_part = !kPlain && ((r.cap > 0.0f && !cap_late) || r.mrow != nullptr);
            if (tid == 0) { /* read again by the warps only if pro_on; the barriers of the part set-up lie between */
                sh->cap      = r.cap;
                sh->mrow     = r.mrow;
                sh->cur_rng  = raw.rng;
                sh->cur_seq  = r.seq;
                sh->cur_last = r.rr == p.rows_per_seq - 1 ? 1 : 0;
                sh->cur_rr   = r.rr;
            }
            /* the thread's ids that fall into the part, or -1 */
            const int at0 = c0 * p.slice, at_n = min(part_len * p.slice, p.V - at0);
#pragma unroll
            for (int q = 0; q < kPerT; q++) {
                const int t = tid + q * kThreads;
                id[q]       = -1;
                if (pen_on && t < n_ids && n_ids <= kRowIds * kPerT) {
                    const int at = (q == 0 ? (t < r.H ? sh->nxt_ids[t] : sh->nxt_ext[t - r.H]) : t < r.H ? r.hrow[t] : r.erow[1 + t - r.H]) - p.vocab_offset - at0;
                    id[q]        = at >= 0 && at < at_n ? at : -1;
                }
            }
        }
        /* the kind the row is streamed as */
        const int   smode   = ((kKinds & K_SUMS) == 0 && (mode == M_TEMP || mode == M_TOPP)) || ((kKinds & K_SEL) == 0 && mode == M_TOPK) ? (int) M_ARGMAX : mode;
        const bool  sel     = (kKinds & K_SEL) != 0 && (smode == M_TOPK || ((kKinds & K_SUMS) != 0 && smode == M_TOPP)) && kq > 0 && kq <= kFastKMax;
        const bool  sums    = (kKinds & K_SUMS) != 0 && (smode == M_TEMP || (smode == M_TOPP && sel));
        const bool  long_ids = (kKinds & K_SHORT) == 0 && n_ids > kRowIdsMax;

        const int  *long_off  = (kKinds & K_SHORT) == 0 && long_ids ? p.pre_off + (size_t) row * (size_t) (p.n_slices * kWarps + 1) + c0 * kWarps : nullptr;
        bool        long_smem = true; /* a long list's part lies in shared memory like a short one's */

        unsigned *id_list = (kKinds & K_SHORT) != 0 ? sh->rl_id : sl_list;

        /* ---- part set-up ---- */
        if (tid == 0) {
            sh->st     = 0;
            sh->n_grp  = 0;
            sh->n_cand = 0;
            sh->max_cnt = 1;
        }
        if (sel) {
            reinterpret_cast<int2 *>(sh->key_bins)[tid] = make_int2(0, 0);
            static_assert(kKeyBins == 2 * kThreads, "two bins per thread");
        }
        if (pen_on && !long_ids) {
            /* The distinct ids that fall into the part, with their counts: an open-addressing table in the group maxima's memory (free
             * between two parts), one id per thread at a time; the thread whose id opened a slot speaks for that id. The ids
             * are then grouped by the (slice, warp) share of the part that they fall into, so that a warp looks at
             * its own share's run alone (most shares hold none): kRowIds groups, slice c of the part and slice
             * c + 32 share one and tell their ids apart by a tag. Bound by latency, of shared-memory atomics and four
             * barriers: 64 ids of a row take 0.55 us, 2.2 with eight integer divisions (150 cycles each) per thread and
             * a table cleared between barriers; 1024 ids 3, where a kernel ahead of the launch took 50 us for 4096 rows
             * (4096 x 128256 with 1024 ids 453 -> 397 us, 8 x 50257 with 500 ids 25.2 -> 19.8). */
            int      grp[kPerT], place[kPerT];
            unsigned entry[kPerT];
            int      slot[kPerT]; /* -1: the thread does not speak for the id */
            /* Where the penalty does not ask how often an id occurs and a bit per column fits, whoever sets an id's bit speaks
             * for it; else the ids are counted in an open-addressing table. */
            const bool by_bit = freq == 0.0f && part_len * p.slice <= kGroupBytes * 8;
#pragma unroll
            for (int q = 0; q < kPerT; q++) {
                slot[q] = -1;
                if (id[q] >= 0) {
                    if (by_bit) {
                        const unsigned bit = 1u << (id[q] & 31);
                        slot[q]            = (atomicOr(reinterpret_cast<unsigned *>(gmem) + (id[q] >> 5), bit) & bit) == 0u ? 0 : -1;
                    } else {
                        unsigned h = ((unsigned) id[q] * 2654435761u) >> (32 - ((kKinds & K_SHORT) != 0 ? 9 : 11));
                        static_assert(kIdSlots == 1 << ((kKinds & K_SHORT) != 0 ? 9 : 11), "the bits that the hash keeps");
                        for (int probe = 0; probe < kIdSlots; probe++) { /* at most half of the slots are ever taken */
                            const int old = atomicCAS(&id_key[h], 0, id[q] + 1);
                            if (old == 0 || old == id[q] + 1) {
                                atomicAdd(&id_cnt[h], 1);
                                slot[q] = old == 0 ? (int) h : -1;
                                break;
                            }
                            h = (h + 1) & (kIdSlots - 1);
                        }
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < kPerT; q++) {
                if (slot[q] >= 0) {
                    const int  c = quotient(id[q], p.slice, p.slice_rcp), local = id[q] - c * p.slice;
                    const bool last = c0 + c == p.n_slices - 1;
                    const int  L = share_len(((last ? n_last : n_full) + 3) >> 2), w = quotient(local >> 2, L, last ? p.share_rcp_last : p.share_rcp); /* L float4 per warp */
                    grp[q]   = (c & 31) * kWarps + w;
                    entry[q] = (unsigned) (local - 4 * w * L) | ((unsigned) (c >> 5) << kTagAt);
                    place[q] = atomicAdd(&id_n[grp[q]], 1);
                }
            }
            __syncthreads();
            if (warp == 0) { /* running sums over the kRowIds counters, eight per lane */
                static_assert(kRowIds == 8 * 32, "eight per lane");
                const int4 a = reinterpret_cast<const int4 *>(id_n)[2 * lane], b = reinterpret_cast<const int4 *>(id_n)[2 * lane + 1];
                const int  s0 = a.x, s1 = s0 + a.y, s2 = s1 + a.z, s3 = s2 + a.w, s4 = s3 + b.x, s5 = s4 + b.y, s6 = s5 + b.z, s7 = s6 + b.w;
                int        before = s7;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int o = __shfl_up_sync(0xffffffffu, before, d);
                    if (lane >= d) {
                        before += o;
                    }
                }
                if (lane == 31) {
                    sh->rl_cnt[kRowIds] = before;
                }
                before -= s7;
                reinterpret_cast<int4 *>(sh->rl_cnt)[2 * lane]     = make_int4(before, before + s0, before + s1, before + s2);
                reinterpret_cast<int4 *>(sh->rl_cnt)[2 * lane + 1] = make_int4(before + s3, before + s4, before + s5, before + s6);
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kPerT; q++) {
                if (slot[q] >= 0) {
                    id_list[sh->rl_cnt[grp[q]] + place[q]] = entry[q] | ((by_bit ? 1u : (unsigned) id_cnt[slot[q]]) << 10);
                }
            }
        } else if (pen_on) {
            /* long histories: a kernel that ran before this one left the row's distinct ids with their counts in
             * global memory, grouped by share. The part copies where its shares' runs start, and the entries
             * themselves when there are at most kListSmem of them: the slices then read them from shared memory
             * instead of paying a round trip to L2 each. */
            if (part_len * kWarps <= kRowIds) {
                for (int i = tid; i <= part_len * kWarps; i += kThreads) {
                    sh->rl_cnt[i] = long_off[i] - long_off[0];
                }
            }
            const int e_lo = long_off[0], e_n = long_off[part_len * kWarps] - e_lo;
            if (e_n <= kListSmem) {
                const unsigned *src = p.pre_list + (size_t) row * (size_t) p.row_cap + e_lo;
                for (int i = tid; i < e_n; i += kThreads) {
                    sl_list[i] = src[i];
                }
            }
            long_smem = part_len * kWarps <= kRowIds && e_n <= kListSmem;
        }
        __syncthreads();

        PROF_ONCE(3);
        CYC(5);
        const double rep_rcp = pen_on ? 1.0 / (double) rep : 1.0;
        /* the entries of the ids that fall into warp w's share of the part's slice s_: an entry that belongs to
         * another slice of the same group has another tag */
        auto ids_of = [&](int s_, int w, const unsigned *&ent, int &lo, int &hi, unsigned &tag) {
            if (!long_ids) {
                const int grp = (s_ & 31) * kWarps + w;
                ent           = id_list;
                lo            = sh->rl_cnt[grp];
                hi            = sh->rl_cnt[grp + 1];
                tag           = (unsigned) s_ >> 5;
            } else {
                const int grp = s_ * kWarps + w;
                ent           = long_smem ? sl_list : p.pre_list + (size_t) row * (size_t) p.row_cap;
                lo            = long_smem ? sh->rl_cnt[grp] : long_off[grp];
                hi            = long_smem ? sh->rl_cnt[grp + 1] : long_off[grp + 1];
                tag           = 0u;
            }
        };
        const unsigned cnt_mask = long_ids ? 0x3fffffu : 0x7ffu; /* above the offset's ten bits; entries of ids counted here carry a tag on top */
        unsigned       run_key = 0u; /* greedy: this warp's maximum of the part so far (key) and its first id */
        int            run_arg = 0x7fffffff;
        float          top0 = -CUDART_INF_F, top1 = -CUDART_INF_F; /* others: the thread's maxima over every other one of its float4 */
        float          ref  = -CUDART_INF_F; /* top-p: what the warp's sum is relative to */
        double         acc  = 0.0;     /* top-p: the thread's sum over the part */
        int            wst  = 0, most = 0; /* most: how often the most frequent id occurs */
        const SumScale ks   = sum_scale2(inv_t);
        int            gm_shift = 0; /* slices that share one slot of the group maxima: 2^gm_shift */
        while (((part_len - 1) >> gm_shift) >= kGroupSlots) {
            gm_shift++;
        }

        const bool masked = !kPlain && pro_part && sh->mrow != nullptr;
        ShareMask  words{};
        if (masked) {
            words = share_mask(sh->mrow, p.V, lane, c0 * p.slice + 4 * (c0 == p.n_slices - 1 ? w4lo_l : w4lo_f));
        }

        /* ---- the part's slices, every warp on its own ---- */
        for (int s = 0; s < part_len; s++, j++) {
            const int      stage  = j % kStages;
            const unsigned parity = (unsigned) (j / kStages) & 1u;
            const int      c      = c0 + s, s0 = c * p.slice;
            const bool     last_c = c == p.n_slices - 1;
            const int      n = last_c ? n_last : n_full, nv4 = (n + 3) >> 2, body = n & ~3;
            const int      w4lo = last_c ? w4lo_l : w4lo_f, mine4 = last_c ? mine4_l : mine4_f;
            float         *sl   = reinterpret_cast<float *>(wring + (size_t) stage * kWarpStageBytes); /* local index = slice index - 4 * w4lo */
            const float   *grow = p.logits + (size_t) row * (size_t) p.row_stride + s0;
            bool           wrote = !aligned; /* the warp wrote into its stage with ordinary stores */
            if (warp == 0 && !final_part && pf < kPrefetchDone) {
                prefetch_step(p, sh, row + 1, lane, pf); /* one step per slice: the step before has long arrived */
            }
            CYC(4);
            /* ---- 1. the warp's share of the slice is in its stage; the slice's tail is padded with -inf ---- */
            if (aligned) {
                if (ring_dead >= 0) {
                    wst |= ST_LOAD_TIMEOUT; /* every row the warp still touches is reported as not loaded */
                } else if (!mbar_wait_bounded(&sh->full[warp][stage], parity)) {
                    wst |= ST_LOAD_TIMEOUT;
                    ring_dead = j; /* the warp asks for no further copy and waits for none; see the kernel's end */
                }
                if (nv4 * 4 > body && w4lo + mine4 == nv4 && mine4 > 0) {
                    wrote = true;
                    if (lane < 4) {
                        const int i      = body + lane; /* the last float4 is not part of the bulk copy */
                        sl[i - 4 * w4lo] = i < n ? grow[i] : -CUDART_INF_F;
                    }
                }
            } else {
                async_copies_wait_but(j + 1 < my_count ? 1 : 0); /* the next item's group may be on its way */
            }
            __syncwarp();
            CYC(0);

            /* ---- 1b. soft cap and mask, in place ---- */
            if (pro_part) {
                wrote = true;
                prologue_share(sl, lane, mine4, 4 * w4lo, n, s0, cap_late ? 0.0f : sh->cap, masked, words);
                if (masked && s + 1 < part_len) {
                    words = share_mask(sh->mrow, p.V, lane, s0 + p.slice + 4 * (c + 1 == p.n_slices - 1 ? w4lo_l : w4lo_f));
                }
            }

            /* ---- 2. penalties on the share ---- */
            if (pen_on) {
                bool touched = false; /* most shares hold none of the row's ids: those need no fence before the refill */
                const unsigned *ent;
                int             lo, hi;
                unsigned        tag;
                ids_of(s, warp, ent, lo, hi, tag);
                for (int e = lo + lane; e < hi; e += 32) {
                    const unsigned en = ent[e];
                    if (long_ids || (en >> kTagAt) == tag) {
                        most    = max(most, (int) ((en >> 10) & cnt_mask));
                        float *q = sl + (en & 0x3ffu);
                        *q       = penalise_rcp(*q, (int) ((en >> 10) & cnt_mask), rep_rcp, rep, freq, pres);
                        touched  = true;
                        if (sel) {
                            const int bit = id_bit(s, warp, (int) (en & 0x3ffu));
                            atomicOr(&sh->id_bits[bit >> 5], 1u << (bit & 31));
                        }
                    }
                }
                wrote |= __any_sync(0xffffffffu, touched); /* also orders the stores before the loads below */
            }
            if (!kPlain && p.out_logits != nullptr) {
                float *orow = p.out_logits + (size_t) row * (size_t) p.V + s0;
                for (int i = 4 * w4lo + lane; i < min(4 * (w4lo + mine4), n); i += 32) {
                    orow[i] = sl[i - 4 * w4lo];
                }
            }

            /* ---- 3. the share in registers; what a thread does not own reads as -inf ---- */
            const float4 *s4 = reinterpret_cast<const float4 *>(sl) + lane;
            /* the share has been read: the stage is free again and the warp refills it itself */
            auto refill = [&]() {
                __syncwarp();
                if (!aligned) {
                    if (j + kStages < my_count) {
                        issue_words();
                    }
                } else if (lane == 0 && j + kStages < my_count && ring_dead < 0) {
                    if (wrote) { /* ordinary stores of this warp come before the copy engine's */
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    }
                    issue_next();
                }
            };
            auto note_maxima = [&](int s_, float m0, float m1) {
                top0          = fmaxf(top0, m0);
                top1          = fmaxf(top1, m1);
                float      *q = &gmax[(s_ >> gm_shift) * kThreads + tid];
                const float m = fmaxf(m0, m1);
                *q            = (s_ & ((1 << gm_shift) - 1)) == 0 ? m : fmaxf(*q, m);
            };
            if (smode == M_ARGMAX) {
                float4 x[kNV4];
                float  bv = -CUDART_INF_F;
#pragma unroll
                for (int i = 0; i < kNV4; i++) {
                    x[i] = lane + 32 * i < mine4 ? s4[32 * i] : make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
                    bv   = max3(max3(bv, x[i].x, x[i].y), x[i].z, x[i].w);
                }
                const unsigned bkey = order_key(bv);
                const bool     own  = lane < mine4;
                const unsigned wkey = __reduce_max_sync(0xffffffffu, own ? bkey : 0u);
                if (wkey > run_key) { /* rare: the warp's running maximum moves; its first id in this slice */
                    const float wmax = key_to_float(wkey);
                    int         best = 0x7fffffff;
                    if (own && bkey == wkey) {
#pragma unroll
                        for (int i = kNV4 - 1; i >= 0; i--) {
                            const int b = 4 * (w4lo + lane + 32 * i);
                            if (x[i].w == wmax) best = b + 3;
                            if (x[i].z == wmax) best = b + 2;
                            if (x[i].y == wmax) best = b + 1;
                            if (x[i].x == wmax) best = b;
                        }
                    }
                    best    = __reduce_min_sync(0xffffffffu, best);
                    run_key = wkey;
                    run_arg = s0 + best;
                }
                refill();
            } else if (!sums) {
                /* top-k: the largest value of the thread's floats is all that the select asks of a slice */
                float m0 = -CUDART_INF_F, m1 = -CUDART_INF_F;
                if (mine4 == 32 * kNV4) {
#pragma unroll
                    for (int i = 0; i < kNV4; i++) {
                        const float4 x = s4[32 * i];
                        float       &m = (i & 1) == 0 ? m0 : m1;
                        m              = max3(max3(m, x.x, x.y), x.z, x.w);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < kNV4; i++) {
                        if (lane + 32 * i < mine4) {
                            const float4 x = s4[32 * i];
                            float       &m = (i & 1) == 0 ? m0 : m1;
                            m              = max3(max3(m, x.x, x.y), x.z, x.w);
                        }
                    }
                }
                refill();
                note_maxima(s, m0, m1);
            } else if constexpr ((kKinds & K_SUMS) != 0) {
                float4 x[kNV4];
                float  m0 = -CUDART_INF_F, m1 = -CUDART_INF_F;
                if (mine4 == 32 * kNV4) {
#pragma unroll
                    for (int i = 0; i < kNV4; i++) {
                        x[i] = s4[32 * i];
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < kNV4; i++) {
                        x[i] = lane + 32 * i < mine4 ? s4[32 * i] : make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
                    }
                }
#pragma unroll
                for (int i = 0; i < kNV4; i++) {
                    float &m = (i & 1) == 0 ? m0 : m1;
                    m        = max3(max3(m, x[i].x, x[i].y), x[i].z, x[i].w);
                }
                refill();
                /* A temperature row's share is summed relative to its own maximum, a top-p row's relative to a value that the
                 * warp's maximum may leave behind by 2^60: the row's largest values are candidates, which leave the
                 * sum again. Where it has gone further, what was summed so far is too little for its factor's last bits
                 * to count. */
                const float m = fmaxf(m0, m1);
                float       from;
                if (smode == M_TEMP) {
                    from = key_to_float(__reduce_max_sync(0xffffffffu, order_key(m)));
                } else {
                    if (__any_sync(0xffffffffu, m > ref && !(__fmul_rn(__fsub_rn(m, ref), ks.hi) <= 60.0f))) {
                        const float now = key_to_float(__reduce_max_sync(0xffffffffu, order_key(m)));
                        acc *= (double) sum_term(ref, ks, now);
                        ref = now;
                    }
                    from = ref;
                }
                const float from0 = from == -CUDART_INF_F ? 0.0f : from; /* nothing but -inf so far: its terms are 0 */
                double      sum   = 0.0;
#pragma unroll
                for (int i = 0; i < kNV4; i++) {
                    sum += (double) sum_terms(x[i], ks, from0);
                }
                if (smode == M_TOPP) {
                    acc += sum;
                    if (lane == 0) {
                        if (s < kSliceRefs) {
                            sh->ref_at[s][warp] = from;
                        } else { /* parts of more slices keep the rest where a temperature row's sums would lie */
                            p.segs[((size_t) row * (size_t) p.n_slices + (size_t) c) * kWarps + warp].ref = from;
                        }
                    }
                    note_maxima(s, m0, m1);
                } else {
                    /* The warp's sum in fixed point: a lane's is at most 32, in steps of 2^-57 its double loses nothing that
                     * a double of the total would hold. Three integer reductions instead of five rounds of double
                     * additions between lanes. A lane whose sum is NaN adds what no sum of lanes comes to. */
                    const long long q   = __double2ll_rn(sum * 0x1p57);
                    const unsigned  lo  = __reduce_add_sync(0xffffffffu, (unsigned) q & 0x1fffffu);
                    const unsigned  mid = __reduce_add_sync(0xffffffffu, (unsigned) (q >> 21) & 0x1fffffu);
                    const unsigned  hi  = __reduce_add_sync(0xffffffffu, sum <= 32.0 ? (unsigned) (q >> 42) : 1u << 26);
                    top0                = fmaxf(top0, m);
                    if (lane == 0) {
                        SegRec sr;
                        sr.ref = from;
                        sr.pad = 0.0f;
                        sr.sum = hi < (1u << 26) ? (double) hi * 0x1p-15 + ((double) mid * 0x1p-36 + (double) lo * 0x1p-57) : CUDART_NAN;
                        p.segs[((size_t) row * (size_t) p.n_slices + (size_t) c) * kWarps + warp] = sr;
                    }
                }
            }
            CYC(2);
        }

        PROF(2);
        /* ---- the part is through ---- */
        wst = __reduce_or_sync(0xffffffffu, (unsigned) wst);
        if (pen_on && sel && freq < 0.0f) {
            most = __reduce_max_sync(0xffffffffu, most);
            if (lane == 0) {
                atomicMax(&sh->max_cnt, most);
            }
        }
        if (smode != M_ARGMAX) {
            run_key = __reduce_max_sync(0xffffffffu, order_key(fmaxf(top0, top1)));
        }
        if ((kKinds & K_SUMS) != 0 && smode == M_TOPP && sums) {
            acc = warp_sum_d(acc);
        }
        if (lane == 0) {
            sh->best[warp]   = ((unsigned long long) run_key << 32) | (unsigned long long) (0xffffffffu - (unsigned) run_arg);
            sh->wb_ref[warp] = ref;
            if (wst != 0) {
                atomicOr(&sh->st, wst);
            }
        }
        float tau  = CUDART_INF_F;
        bool  over = false;
        if (sel) {
            /*
             * The threshold: the kq-th largest (or one a little below) of the 256 thread maxima, a lower bound of the
             * part's kq-th largest value that lies close to it (k of 256 threads hold about k + k^2 / 512 of the
             * values above it; beyond k = 128 the 512 half maxima are asked).
             * Against capturing candidates above a rising threshold while the part streams (465 instead of about 100
             * instructions per warp and slice, two barriers and shared-memory atomics inside the part): 256 x 128256
             * top-k 40 with penalties 33.2 -> 32.2 us, 4096 x 128256 top-k 50 549 -> 541 us, 256 x 262144 top-p
             * 97.0 -> 85.2 us with the sums' new form, 48 x 262144 soft-capped top-k 64 116 -> 104 us a step.
             */
            const bool two  = kq > kThreads / 2;
            float      sel0 = two ? top0 : fmaxf(top0, top1), sel1 = top1;
            if (cap_late) { /* as the values they belong to will be once they are read again */
                sel0 = sel0 == -CUDART_INF_F ? sel0 : soft_cap(sel0, sh->cap);
                if (two) {
                    sel1 = sel1 == -CUDART_INF_F ? sel1 : soft_cap(sel1, sh->cap);
                }
            }
            const unsigned tkey = kth_key(order_key(sel0), order_key(sel1), two, kq, sh->key_bins, sh->key_ends, lane, warp);
            tau = tkey <= order_key(-CUDART_INF_F) ? -CUDART_INF_F : key_to_float(tkey); /* fewer than kq of them: everything passes */
            float tau_grp = tau;
            if (cap_late && tau > -CUDART_INF_F) {
                /* The place of the uncapped row below which no capped value reaches tau. tanhf, the division and the product
                 * are good to 2^-21 together, so such a value's true tanh(x / c) is at least y; the margins are four times
                 * that and cover atanhf, the last two what falls below the smallest normal float. */
                const float c = sh->cap, y0 = __fdiv_rn(tau, c), y = y0 - fabsf(y0) * 0x1p-19f;
                const float t = y > -1.0f ? c * atanhf(y) : -CUDART_INF_F;
                tau_grp       = t - fabsf(t) * 0x1p-20f - c * 0x1p-140f - 0x1p-120f;
            }
            /* the thread's groups that reach it: listed by the warp, a place in the list for all of the warp's at once */
            const int slots = ((part_len - 1) >> gm_shift) + 1;
            unsigned  hits  = 0u; /* of the thread's slots */
            if (fmaxf(top0, top1) >= tau_grp) {
#pragma unroll 4
                for (int i = 0; i < slots; i++) {
                    hits |= gmax[i * kThreads + tid] >= tau_grp ? 1u << i : 0u;
                }
            }
            const int hits_w = __reduce_add_sync(0xffffffffu, __popc(hits));
            int       at     = lane == 0 && hits_w > 0 ? atomicAdd(&sh->n_grp, hits_w) : 0;
            at               = __shfl_sync(0xffffffffu, at, 0);
            for (unsigned any; (any = __ballot_sync(0xffffffffu, hits != 0u)) != 0u; at += __popc(any)) {
                if (hits != 0u) {
                    sh->grp[at + __popc(any & ((1u << lane) - 1u))] = (unsigned short) (((__ffs(hits) - 1) << 8) | tid);
                    hits &= hits - 1u;
                }
            }
            __syncthreads();
            /* their float4, read again (L2 holds them), changed as they were while the part streamed */
            const bool rewritten = !kPlain && p.out_logits != nullptr, src_al = kPlain || again_aligned(p);
            const bool bits_say  = part_len <= 4 && freq == 0.0f; /* every value has a bit of its own and its penalty does not ask how often */
            /* no value below tau_raw reaches tau with the penalties that raise it most (a repetition penalty below 1, negative
             * ones); the margins are eight times what the roundings of a penalised value add up to */
            float tau_raw = tau;
            if (pen_on && !(rep >= 1.0f && freq >= 0.0f && pres >= 0.0f)) {
                const float f = (float) (freq < 0.0f ? sh->max_cnt : 1) * freq, y = tau + f + pres - (fabsf(tau) + fabsf(f) + fabsf(pres)) * 0x1p-20f;
                const float x = y > 0.0f ? y * rep : __fdiv_rn(y, rep);
                tau_raw       = fminf(tau, x - fabsf(x) * 0x1p-20f);
            }
            /* a candidate at least in each: more groups than candidates fit need no look (uncapped values may fall short) */
            over = sh->n_grp > kPartCand && !(cap_late && tau > -CUDART_INF_F);
            const int per_log = kNV4Log + gm_shift, n_again = over ? 0 : sh->n_grp << per_log;
            double    fix     = 0.0;
            /* the float4 that item t of the groups names: slice of the part, warp, index in the share, where in the slice; whether there is one */
            auto named = [&](int t, int &s, int &w, int &i4, int &e0, int &n) {
                const int name = t < n_again ? sh->grp[t >> per_log] : 0, f = t & ((1 << per_log) - 1);
                s              = ((name >> 8) << gm_shift) + f / kNV4;
                w              = (name & 255) >> 5;
                i4             = (name & 31) + 32 * (f % kNV4);
                n              = c0 + s == p.n_slices - 1 ? n_last : n_full;
                const int nv4 = (n + 3) >> 2, L = share_len(nv4), w4 = min(w * L, nv4);
                e0 = 4 * (w4 + i4);
                return t < n_again && s < part_len && i4 < min(L, nv4 - w4);
            };
            const float *src_row = kPlain ? p.logits + (size_t) row * (size_t) p.row_stride : row_again(p, row);
            auto         fetched = [&](int t) {
                float4 v = make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
                int    s, w, i4, e0, n;
                if (named(t, s, w, i4, e0, n)) {
                    const float *src = src_row + (c0 + s) * p.slice + e0;
                    if (src_al && e0 + 4 <= n) {
                        v = *reinterpret_cast<const float4 *>(src);
                    } else {
                        v.x = e0 + 0 < n ? src[0] : -CUDART_INF_F;
                        v.y = e0 + 1 < n ? src[1] : -CUDART_INF_F;
                        v.z = e0 + 2 < n ? src[2] : -CUDART_INF_F;
                        v.w = e0 + 3 < n ? src[3] : -CUDART_INF_F;
                    }
                }
                return v;
            };
            float4 ahead{};
#pragma unroll 1
            for (int t0 = 32 * warp; t0 < n_again; t0 += kThreads) { /* whole warps: ids are looked up by all lanes together */
                const bool   first = ((t0 / kThreads) & 1) == 0; /* two of a lane's float4 on their way at a time */
                const float4 got   = first ? fetched(t0 + lane) : ahead;
                if (first) {
                    ahead = fetched(t0 + kThreads + lane);
                }
                float      v[4] = {got.x, got.y, got.z, got.w};
                int        s, w, i4, e0, n;
                const bool own = named(t0 + lane, s, w, i4, e0, n);
                const int  c = c0 + s, id0 = c * p.slice + e0;
                if (pro_on && !rewritten && own) {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (e0 + q < n) {
                            v[q] = prologue_one(v[q], id0 + q, cap_late ? 0.0f : sh->cap, sh->mrow);
                        }
                    }
                }
                if (pen_on && !rewritten) {
                    /* Which of the four an id has changed (a bit each, which may be another slice's where the part is long).
                     * Where the bits are the value's own and the penalty does not ask how often the id occurs, that is
                     * all there is to know. Else the ids are looked up, the warp's lanes going through the share's
                     * list together, for values that can reach the threshold (a sum wants all four of a candidate's
                     * float4). Against every float4 going through its share's list by itself, us: 1000 rows of 4096
                     * columns, top-k 40, rep 1.1: 64 ids 45.1 -> 39.8, 256 ids 63.2 -> 44.9, 1000 ids 132 -> 64.7;
                     * 256 x 128256 with 64 ids 32.2 -> 31.2; 4096 x 128256 with 1024 ids, top-k 50: 539 -> 509. */
                    const int bit   = id_bit(s, w, 4 * i4);
                    unsigned  mark  = own ? (sh->id_bits[bit >> 5] >> (bit & 31)) & 15u : 0u;
                    int       cnt[4] = {1, 1, 1, 1};
                    if (!bits_say) {
                        unsigned reach = 0u, found = 0u;
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            reach |= v[q] < tau_raw ? 0u : 1u << q;
                        }
                        mark = (kKinds & K_SUMS) != 0 && sums ? (reach != 0u ? mark : 0u) : mark & reach;
                        for (unsigned ask = __ballot_sync(0xffffffffu, mark != 0u); ask != 0u; ask &= ask - 1u) {
                            const int       from = __ffs(ask) - 1, i4_ = __shfl_sync(0xffffffffu, i4, from);
                            const unsigned *ent;
                            int             lo, hi;
                            unsigned        tag;
                            ids_of(__shfl_sync(0xffffffffu, s, from), __shfl_sync(0xffffffffu, w, from), ent, lo, hi, tag);
                            for (int base = lo; base < hi; base += 32) {
                                const unsigned en = base + lane < hi ? ent[base + lane] : 0u;
                                for (unsigned hit = __ballot_sync(0xffffffffu, base + lane < hi && (int) ((en & 0x3ffu) >> 2) == i4_ && (long_ids || (en >> kTagAt) == tag)); hit != 0u; hit &= hit - 1u) {
                                    const unsigned eh = __shfl_sync(0xffffffffu, en, __ffs(hit) - 1);
                                    if (lane == from) {
                                        found |= 1u << (eh & 3u);
#pragma unroll
                                        for (int q = 0; q < 4; q++) {
                                            cnt[q] = (int) (eh & 3u) == q ? (int) ((eh >> 10) & cnt_mask) : cnt[q];
                                        }
                                    }
                                }
                            }
                        }
                        mark = found;
                    }
                    if (mark != 0u) {
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if ((mark >> q) & 1u) {
                                v[q] = penalise_rcp(v[q], cnt[q], rep_rcp, rep, freq, pres);
                            }
                        }
                    }
                }
                unsigned hit[4], found = 0u; /* which lanes' values are candidates */
                bool     any = false;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const bool cand = own && v[q] >= tau_grp && e0 + q < n; /* tau itself, but for values that are capped below */
                    hit[q]          = __ballot_sync(0xffffffffu, cand);
                    found += __popc(hit[q]);
                    any |= cand;
                }
                if (found != 0u) {
                    int pos = lane == 0 ? atomicAdd(&sh->n_cand, (int) found) : 0;
                    pos     = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int at = pos + __popc(hit[q] & ((1u << lane) - 1u));
                        if (((hit[q] >> lane) & 1u) != 0u && at < kPartCand) {
                            sh->cand[at].v   = v[q];
                            sh->cand[at].idx = id0 + q;
                        }
                        pos += __popc(hit[q]);
                    }
                }
                if ((kKinds & K_SUMS) != 0 && sums && any) {
                    /* a candidate's weight is evaluated exactly where the row is finished: it leaves the sum, as the
                     * term of its float4 entered it, and what shares its float4 comes back one by one */
                    const float u  = s < kSliceRefs ? sh->ref_at[s][w] : p.segs[((size_t) row * (size_t) p.n_slices + (size_t) c) * kWarps + w].ref;
                    const float u0 = u == -CUDART_INF_F ? 0.0f : u;
                    double      now = -(double) sum_terms(make_float4(v[0], v[1], v[2], v[3]), ks, u0);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (!(v[q] >= tau)) {
                            now += (double) sum_term(v[q], ks, u0);
                        }
                    }
                    fix += now * ref_move(u, part_ref(sh), inv_t);
                }
            }
            if ((kKinds & K_SUMS) != 0 && sums) {
                fix = warp_sum_d(fix);
                if (lane == 0) { /* with the warp's own sum: each warp moves its own */
                    sh->wb_acc[warp] = acc;
                    sh->wb_sum[warp] = acc * ref_move(ref, part_ref(sh), inv_t) + fix;
                }
            }
        }
        __syncthreads();
        auto part_again = [&]() { /* raise_threshold is called next; its arguments lie here and not in a stack frame */
            if (tid != 0) {
                return;
            }
            constexpr bool kPen = (kKinds & K_PEN) != 0, kLong = kPen && (kKinds & K_SHORT) == 0, kSums = (kKinds & K_SUMS) != 0;
            const bool     done = !kPlain && p.out_logits != nullptr;
            PartAgain     &again = sh->again;
            again.row       = row;
            again.c0        = c0;
            again.part_len  = part_len;
            again.gm_shift  = gm_shift;
            again.kq        = kq;
            again.pro       = !kPlain && pro_on && !done;
            again.sums      = kSums && sums;
            again.inv_t     = inv_t;
            again.pen       = kPen && pen_on && !done;
            again.rep       = kPen ? rep : 1.0f;
            again.freq      = kPen ? freq : 0.0f;
            again.pres      = kPen ? pres : 0.0f;
            again.rep_rcp   = kPen ? rep_rcp : 1.0;
            again.long_ids  = kLong && long_ids;
            again.long_off  = kLong ? long_off : nullptr;
            again.long_smem = !kLong || long_smem;
            again.list      = !kLong || !long_ids || long_smem ? id_list : p.pre_list + (size_t) row * (size_t) p.row_cap;
        };
        int       n_cand = over ? kPartCand + 1 : min(sh->n_cand, kPartCand + 1); /* more than kPartCand: the list ran over */
        if (!kPlain && cap_late && n_cand <= kPartCand) {
            /* One candidate per thread, where every value that was read again took a tanhf and a division. What falls short of
             * tau now is no more than a candidate too many. */
            for (int i = tid; i < n_cand; i += kThreads) {
                sh->cand[i].v = prologue_one(sh->cand[i].v, sh->cand[i].idx, sh->cap, sh->mrow); /* the mask again: the cap of -inf is not -inf */
            }
            __syncthreads();
        }
        /* Rows are finished here in launches of greedy and top-k rows alone: the instantiations with sums carry none of it (with it, and
         * the code behind it, a launch of one temperature row of 128256 takes 9.1 us and not 8.3) */
        if constexpr ((kKinds & (K_SEL | K_SUMS)) == K_SEL) {
            if ((p.flags & F_INLINE_TOPK) != 0u && mode != M_ARGMAX) {
                /* whole rows, top-k: finished here, nothing goes to global scratch (every row of such a launch is one
                 * part); a row of another kind is reported as the small finishing kernel would */
                if (mode == M_TOPK) {
                    inline_finish_topk<true>(p, sh, gmem, row, n_cand, kq, tau, cap_late, inv_t, sh->st, part_again);
                } else {
                    if (tid == 0) {
                        p.tokens[row] = -1;
                        p.status[row] = sh->st | ST_INTERNAL;
                    }
                    __syncthreads();
                }
                CYC(6);
                continue;
            }
        }
        if (sel && n_cand > kPartCand && tau > -CUDART_INF_F) {
            part_again();
            tau = raise_threshold(p, sh, tau);
            __syncthreads();
            n_cand = min(sh->n_cand, kPartCand + 1);
        }
        const int held = sel ? min(n_cand, kPartCand) : 0;
        int       part_idx = 0, n_parts = 1; /* which part of the row this is, of how many */
        if (p.map.mode == RUN_PARTS) {
            n_parts  = p.map.P;
            part_idx = (int) blockIdx.x - row * n_parts;
        } else if (p.map.mode == RUN_ITEMS) {
            const int b_first = cta_of_item(p, row * p.n_slices);
            part_idx          = (int) blockIdx.x - b_first;
            n_parts           = cta_of_item(p, row * p.n_slices + p.n_slices - 1) - b_first + 1;
        }
        int own_arg = 0, own_st = 0; /* what the first thread writes as the part's record */
        if (tid == 0) {
            unsigned long long bw = 0ull;
#pragma unroll
            for (int w = 0; w < kWarps; w++) {
                bw = max(bw, sh->best[w]);
            }
            float  bref = -CUDART_INF_F;
            double bsum = 0.0;
            if ((kKinds & K_SUMS) != 0 && smode == M_TOPP && sums) {
                bref = part_ref(sh);
#pragma unroll
                for (int w = 0; w < kWarps; w++) {
                    bsum += sh->wb_sum[w];
                }
                bsum = bsum < 0.0 ? 0.0 : bsum; /* a NaN stays one: the walk ends on the row's last id, as the reference's does */
                p.wide_head->any = p.launch; /* the finishing kernel's blocks without a row of their own wait for wide ones */
            }
            int4           h, h2;
            h.x  = __float_as_int((unsigned) (bw >> 32) == 0u ? -CUDART_INF_F : part_top(sh, cap_late));
            h.y  = (int) (0xffffffffu - (unsigned) (bw & 0xffffffffull));
            h.z  = sel ? n_cand : 0;
            h.w  = sh->st;
            h2.x = __float_as_int(sel ? tau : -CUDART_INF_F);
            h2.y = __float_as_int(bref);
            h2.z = __double2loint(bsum);
            h2.w = __double2hiint(bsum);
            int4 *rec = part_rec(p, row, part_idx);
            rec[0]    = h; /* the record lies in front of the part's candidates */
            rec[1]    = h2;
            own_arg = h.y;
            own_st  = h.w;
        }
        if ((kKinds & K_SUMS) == 0 && (p.flags & (F_GREEDY_ONLY | F_INLINE_TOPK)) != 0u && warp == 0) { /* in a launch that finishes its top-k rows here, the greedy ones are finished here as well */
            /* The caller said that every row is greedy: no finishing kernel follows. A row that went through
             * this thread block as a whole is known here. A row cut into parts is finished by whichever of its
             * parts arrives last: every part publishes its record, then counts itself in; the one that finds
             * all the others counted reads their records and puts the counter back to zero for the next launch.
             * Nobody waits for anybody. A row that is not greedy after all is reported. Bound by three round trips to L2: the
             * records are read by a lane each (one thread, one after the other: one row of
             * 151936 in 19 parts, with its call, 14.8 us; 13.2). */
            int  best_arg = __shfl_sync(0xffffffffu, own_arg, 0), stq = __shfl_sync(0xffffffffu, own_st, 0);
            bool mine     = n_parts == 1;
            if (!mine) {
                int before = 0;
                if (lane == 0) {
                    __threadfence();
                    before = atomicAdd(&p.arrive[row], 1);
                }
                if (__shfl_sync(0xffffffffu, before, 0) == n_parts - 1) {
                    __threadfence();
                    unsigned key = 0u;
                    int      arg = 0x7fffffff, st = 0;
                    for (int q = lane; q < n_parts; q += 32) {
                        const int4     o = __ldcg(part_rec(p, row, q));
                        const unsigned k = order_key(__int_as_float(o.x));
                        if (k > key || (k == key && o.y < arg)) {
                            key = k;
                            arg = o.y;
                        }
                        st |= o.w;
                    }
                    const unsigned top = __reduce_max_sync(0xffffffffu, key);
                    best_arg           = __reduce_min_sync(0xffffffffu, key == top ? arg : 0x7fffffff);
                    stq |= __reduce_or_sync(0xffffffffu, st);
                    if (lane == 0) {
                        p.arrive[row] = 0;
                    }
                    mine = true;
                }
            }
            if (mine && lane == 0) {
                if (mode == M_ARGMAX) {
                    p.tokens[row] = best_arg + p.vocab_offset;
                } else { /* only with F_GREEDY_ONLY: the other flag's rows of other kinds never come here */
                    p.tokens[row] = -1;
                    stq |= ST_INTERNAL;
                }
                if (p.kept_cap > 0) {
                    p.kept_n[row] = 0;
                }
                p.status[row] = stq;
                if (p.rng_out != nullptr && sh->cur_last) {
                    p.rng_out[sh->cur_seq] = sh->cur_rng; /* greedy rows draw nothing (sampler.c:106-112) */
                }
            }
        }
        {
            unsigned long long *dst = reinterpret_cast<unsigned long long *>(part_rec(p, row, part_idx)) + 4;
            for (int f = tid; f < held; f += kThreads) {
                dst[f] = *reinterpret_cast<const unsigned long long *>(&sh->cand[f]);
            }
        }
        __syncthreads(); /* the lists are free for the next part */
        CYC(6);
    }
    if (ring_dead >= 0 && aligned) {
        /* copies that were asked for before the warp gave up (the item it gave up on and the one behind it) may
         * still be on their way into this thread block's shared memory: one more bounded wait for each before the
         * thread block may end */
        for (int jj = ring_dead; jj < min(ring_dead + kStages, my_count); jj++) {
            (void) mbar_wait_bounded(&sh->full[warp][jj % kStages], (unsigned) (jj / kStages) & 1u);
        }
    }
    CYC_DONE();
    PROF(4);
}

/* ----------------------------------------------------------- finishing kernel -- */

/*
 * Run behind the stream kernel, one thread block per row at a time (rows blockIdx.x, blockIdx.x + gridDim.x, ...):
 * it merges the records that the row's parts left and finishes the row. finish_rows_kernel<false> carries the
 * code for every kind of row: greedy, top-k, temperature (segment walks), top-p (nucleus sums), wide nuclei, which
 * thread blocks without a row of their own help with, and the multi-pass path over a private copy of the row (a copy per
 * row, or a pool that the thread blocks claim slots of). finish_rows_kernel<true> carries greedy and top-k (k <= 256) alone: a tenth of the code, 7 - 8 us
 * less per launch; it is launched instead when the caller vouched for such rows, and reports any other row as
 * ROW_INTERNAL. Both write the row's status and, behind a sequence's last row, its generator.
 */
/*
 * A row that the candidates could not serve, all threads of its thread block: a wide nucleus becomes everybody's, any
 * other row takes the multi-pass path over a private copy. Out of line, and it asks for the row's parameters again; what the
 * functions behind it need of them lies in shared memory. Handed on by reference, the parameters and the group had lain in
 * the kernel's stack frame, and the out-of-line functions had spilled around them: a frame of 464 bytes, 96 now and
 * no spills; 1000 wide rows of 8192 212 -> 194 us, 24 of 100003 among 96 rows 80 -> 75.
 * Narrow launches did not change: for those the frame alone costs nothing that was measured.
 */
__device__ __noinline__ void deferred_row(const SampleParams &p, FinishShared *sh, unsigned char *cmem, int row, int st) {
    const Grp    g  = whole_block();
    const RawCfg rc = raw_config(p, row, true);
    const RowCfg r  = finish_config(p, row, rc);
    const float bm = sh->gs.blk_max;
    const int   ba = sh->gs.blk_arg;
    if (g.tid == 0) {
        /* claim a row copy: bounded search, the holders always make progress; with a copy per row there is nothing to claim */
        int got = p.n_rows <= p.pool_slots ? row : -1;
        for (long long t = 0; t < (1ll << 24) && got < 0; t++) {
            const int c = (int) ((blockIdx.x + t) % (unsigned) p.pool_slots);
            if (atomicCAS(&p.pool[c], 0, 1) == 0) {
                got = c;
            }
        }
        __threadfence();
        sh->slot = got;
    }
    __syncthreads();
    const int    slot = sh->slot;
    const double S0   = sh->wide_S;
    if (slot >= 0 && r.mode == M_TOPP && S0 > 0.0 && S0 < CUDART_INF && p.V <= kWidePiecesMax * kWidePiece) {
        wide_open(p, &sh->gs, reinterpret_cast<WideShared *>(cmem), slot, row, st, bm, ba, S0, sh->save); /* done by whoever completes it */
        return;
    }
    if (g.tid == 0 && r.mode == M_TOPP) {
        atomicAdd(&p.wide_head->rows, 1ull);
    }
    if (slot < 0) {
        st |= ST_INTERNAL;
    } else {
        WideShared *ws = reinterpret_cast<WideShared *>(cmem);
        if (g.tid == 0) {
            ws->cfg = r;
        }
        __syncthreads();
        st |= multipass_row(p, &sh->gs, &ws->cfg, bm, ba, cmem, offsetof(WideShared, cfg), slot, sh->save);
        __syncthreads();
        if (g.tid == 0 && p.n_rows > p.pool_slots) {
            __threadfence();
            atomicExch(&p.pool[slot], 0);
        }
    }
    if (g.tid == 0) {
        row_epilogue(p, r, row, st, rc.rng);
    }
    __syncthreads();
}

template <bool kFast>
__global__ void __launch_bounds__(kThreads, 2) finish_rows_kernel(const __grid_constant__ SampleParams p) {
    extern __shared__ __align__(128) unsigned char fsmem[];
    FinishShared  *sh   = reinterpret_cast<FinishShared *>(fsmem);
    unsigned char *cmem = reinterpret_cast<unsigned char *>(sh + 1);

    Grp g;
    g.tid  = (int) threadIdx.x;
    g.lane = g.tid & 31;
    g.warp = g.tid >> 5;
    g.n    = kThreads;
    g.nw   = kWarps;
    g.bar  = 0;
    /* The first row's parameters are inputs of the launch, written before the stream kernel began: they may be
     * read while that kernel's last thread blocks are still at work. Everything it wrote waits for the line below. */
    const RunMap &m        = p.map;
    auto          parts_of = [&](int row) { /* over how many thread blocks the row was spread */
        const int i = row * p.n_slices;
        return m.mode == RUN_ROWS ? 1 : m.mode == RUN_PARTS ? m.P : run_of(i + p.n_slices - 1, m.q, m.r) - run_of(i, m.q, m.r) + 1;
    };
    const bool owns    = (int) blockIdx.x < p.n_rows;
    int        n_parts = owns ? parts_of((int) blockIdx.x) : 0;
    if (owns) {
        const RawCfg rc = raw_config(p, (int) blockIdx.x, true);
        const RowCfg r  = finish_config(p, (int) blockIdx.x, rc);
        if (g.tid == 0) {
            sh->cfg  = r;
            sh->rng0 = rc.rng;
        }
        __syncthreads();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory"); /* the records of the kernel before this one are complete and visible */
    asm volatile("griddepcontrol.launch_dependents;");
    PROF(kFast ? 5 : 7);
    /* the launch has top-p rows: the stream kernel has said so; wanted when the block's own rows are done */
    const bool any = !kFast && *reinterpret_cast<volatile const unsigned *>(&p.wide_head->any) == p.launch;
    if (g.tid == 0 && owns) {
        not_wide<kFast>(p, sh);
    }
    for (int row = (int) blockIdx.x; row < p.n_rows; row += (int) gridDim.x) {
        const bool first = row == (int) blockIdx.x, temp = sh->cfg.mode == M_TEMP; /* the row's, or the one's before it */
        if (!first) {
            n_parts = parts_of(row);
        }
        PROF(8);
        int st = finish_row<kFast>(g, p, sh, row, n_parts, first, temp, cmem);
        PROF(13);
        if (st & ST_DEFERRED) {
            if constexpr (kFast) {
                /* This kernel does not carry the code for the row. A top-k row whose candidates did not fit (many
                 * equal values at the top) is the caller's to launch again without the hint; any other kind of
                 * row the caller said would not come. */
                st = (st & ~ST_DEFERRED) | (sh->cfg.mode == M_TOPK ? ST_RETRY : ST_INTERNAL);
                if (g.tid == 0) {
                    p.tokens[row] = -1;
                }
            } else {
                deferred_row(p, sh, cmem, row, st & ~ST_DEFERRED);
                continue;
            }
        }
        if (g.tid == 0) {
            row_epilogue(p, sh->cfg, row, st, sh->rng0);
        }
        __syncthreads();
    }
    if constexpr (!kFast) {
        /* Else there is nothing to help with, and the blocks that have no row end where they begin. (They watched three
         * microseconds for a top-p row to be named: a matmul on another stream took 16.6 us next to launches of one temperature
         * row without such blocks, 22.7 with them, and 19.7 since they end at once.) */
        if (any) {
            int opened = 0;
            if (g.tid == 0) {
                if ((int) blockIdx.x == p.n_rows) { /* one of them says so: a count cost narrow launches 0.1 - 0.2 us */
                    p.wide_head->waited = 1;
                }
                opened = wide_wait(p, 0u);
            }
            if (__syncthreads_or(opened) != 0) {
                wide_help(p, &sh->gs, reinterpret_cast<WideShared *>(cmem), opened, sh->save);
            }
        }
    }
    PROF(kFast ? 6 : 7);
}

/* ------------------------------------------------ long histories, prepared -- */

/* Which (slice, warp) share a column lies in, and where in it. */
__device__ __forceinline__ int share_of(const SampleParams &p, int id, int &off) {
    const int c = id / p.slice, local = id - c * p.slice;
    const int L = share_len((min(p.slice, p.V - c * p.slice) + 3) >> 2);
    const int w = (local >> 2) / L;
    off         = local - 4 * w * L;
    return c * kWarps + w;
}

/* One thread block per row whose history (plus fed tokens) is longer than the stream kernel counts
 * by itself: the row's distinct ids with their counts, grouped by the (slice, warp) share they fall into.
 * pre_off[row][g] .. pre_off[row][g + 1] is share g's run in pre_list[row]; an entry is
 * (offset in the share) | (count << 10). Shorter rows are left to the stream kernel. A thread keeps its kPer ids in
 * registers: they are on their way while the table is cleared, and the thread whose id opened a slot of the table writes
 * that id's entry, at the place in its share's run that counting the share gave it. */
constexpr int kIdThreads = 1024, kPer = 8; /* 8192 ids at most: id_slots */
__global__ void __launch_bounds__(kIdThreads) row_ids_kernel(const __grid_constant__ SampleParams p) {
    extern __shared__ __align__(16) int row_ids_smem[];
    int *tkey = row_ids_smem;          /* open-addressing table: the id ... */
    int *tcnt = tkey + p.id_slots;     /* ... and how often it occurs */
    int *bcnt = tcnt + p.id_slots;     /* entry g + 1: distinct ids in share g; after the scan, entry g: ids in the shares before */

    /* the stream kernel behind this one may start now: it copies logits and sets itself up while the
     * lists are made, and waits for them where it first needs one */
    asm volatile("griddepcontrol.launch_dependents;");
    const int n_shares = p.n_slices * kWarps;
    const int row  = (int) blockIdx.x, tid = (int) threadIdx.x;
    const int seq0 = p.rows_per_seq == 1 ? row : row / p.rows_per_seq;
    const int seq  = p.slot ? p.slot[seq0] : seq0;
    const int H    = p.hist ? (int) min((long long) max(p.hist_len[seq], 0), p.hist_stride) : 0;
    const int E    = p.extra ? row - seq0 * p.rows_per_seq : 0;
    if (H + E <= kRowIdsMax) {
        return;
    }
    const int *hrow = p.hist ? p.hist + (size_t) seq * (size_t) p.hist_stride : nullptr;
    const int *erow = p.extra ? p.extra + (size_t) seq0 * (size_t) p.extra_stride : nullptr;
    int id[kPer];
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        const int j = tid + q * kIdThreads;
        id[q]       = j < H + E ? (j < H ? hrow[j] : erow[1 + j - H]) - p.vocab_offset : -1;
    }
    for (int i = tid; i < p.id_slots / 4; i += kIdThreads) {
        reinterpret_cast<int4 *>(tkey)[i] = make_int4(-1, -1, -1, -1);
        reinterpret_cast<int4 *>(tcnt)[i] = make_int4(0, 0, 0, 0);
    }
    for (int i = tid; i <= n_shares; i += kIdThreads) {
        bcnt[i] = 0;
    }
    __syncthreads();
    const unsigned smask = (unsigned) p.id_slots - 1u;
    int            slot[kPer], share[kPer], place[kPer];
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        slot[q] = -1;
        if (id[q] >= 0 && id[q] < p.V) {
            unsigned hsh = ((unsigned) id[q] * 2654435761u) & smask;
            for (int probe = 0; probe < p.id_slots; probe++) { /* at most half of the slots are ever taken */
                const int old = atomicCAS(&tkey[hsh], -1, id[q]);
                if (old == -1 || old == id[q]) {
                    atomicAdd(&tcnt[hsh], 1);
                    slot[q] = old == -1 ? (int) hsh : -1;
                    break;
                }
                hsh = (hsh + 1u) & smask;
            }
        }
        if (slot[q] >= 0) {
            int off;
            share[q] = share_of(p, id[q], off);
            place[q] = atomicAdd(&bcnt[share[q] + 1], 1);
            id[q]    = off;
        }
    }
    __syncthreads();
    if (tid < 32) {
        int *off   = p.pre_off + (size_t) row * (size_t) (n_shares + 1);
        int  carry = 0;
        for (int base = 0; base <= n_shares; base += 32) {
            const int i    = base + tid;
            int       incl = i <= n_shares ? bcnt[i] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, d);
                if (tid >= d) {
                    incl += up;
                }
            }
            if (i <= n_shares) {
                bcnt[i] = carry + incl;
                off[i]  = carry + incl;
            }
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
    unsigned *list = p.pre_list + (size_t) row * (size_t) p.row_cap;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        if (slot[q] >= 0) {
            list[bcnt[share[q]] + place[q]] = (unsigned) id[q] | ((unsigned) tcnt[slot[q]] << 10);
        }
    }
}


/* ----------------------------------------------------------------- launchers -- */

#ifdef GB_PROFILE
extern "C" int geist_b200_debug_mp(long long *out) { return (int) cudaMemcpyFromSymbol(out, g_mp, sizeof(long long) * 1024 * 24); }
extern "C" int geist_b200_debug_prof(long long *out) { return (int) cudaMemcpyFromSymbol(out, g_prof, sizeof(long long) * 1024 * 16); }
#ifdef GB_PROFILE_CYC
extern "C" int geist_b200_debug_cyc(long long *out) { return (int) cudaMemcpyFromSymbol(out, g_cyc, sizeof(long long) * 1024 * kWarps * 8); }
#endif
#endif

size_t sample_stream_smem(int n_slices, int long_ids) {
    size_t b = (size_t) kWarps * kStages * kWarpStageBytes + sizeof(StreamShared) + (size_t) kGroupBytes;
    if (long_ids) {
        b += (size_t) kListSmem * 4;
    }
    return b;
}

static cudaError_t ensure_attributes(size_t smem_bytes) {
    static int  configured_smem[64] = {0};
    int         dev                 = 0;
    cudaError_t e                   = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    if (dev < 0 || dev >= 64) {
        return cudaErrorInvalidDevice;
    }
    if ((int) smem_bytes > configured_smem[dev]) {
        /* two thread blocks per SM need nearly all of its shared memory: ask for the largest carve-out */
#define GB_STREAM_ALL(X)                                                                                                                     \
    X(K_SEL | K_SUMS | K_PEN) X(K_SEL | K_PEN) X(K_PEN) X(K_SEL | K_SUMS | K_PEN | K_SHORT) X(K_SEL | K_PEN | K_SHORT) X(K_PEN | K_SHORT)      \
    X(K_SEL | K_SUMS | K_SHORT) X(K_SEL | K_SHORT) X(K_SHORT)                                                                                  \
    X(K_PLAIN | K_SEL | K_SUMS | K_PEN) X(K_PLAIN | K_SEL | K_PEN) X(K_PLAIN | K_PEN)                                                         \
    X(K_PLAIN | K_SEL | K_SUMS | K_PEN | K_SHORT) X(K_PLAIN | K_SEL | K_PEN | K_SHORT) X(K_PLAIN | K_PEN | K_SHORT)                            \
    X(K_PLAIN | K_SEL | K_SUMS | K_SHORT) X(K_PLAIN | K_SEL | K_SHORT) X(K_PLAIN | K_SHORT)
#define GB_STREAM_PTR(K) reinterpret_cast<const void *>(sample_stream_kernel<(K)>),
        const void *kernels[] = {GB_STREAM_ALL(GB_STREAM_PTR)};
#undef GB_STREAM_PTR
        for (const void *k : kernels) {
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem_bytes);
            if (e == cudaSuccess) {
                e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int) cudaSharedmemCarveoutMaxShared);
            }
            if (e != cudaSuccess) {
                return e;
            }
        }
        configured_smem[dev] = (int) smem_bytes;
    }
    return cudaSuccess;
}

/* Thread blocks of the stream kernel that one SM of the current device holds at this much shared memory. */
cudaError_t sample_stream_ctas_per_sm(size_t smem_bytes, int *out) {
    cudaError_t e = ensure_attributes(smem_bytes);
    if (e != cudaSuccess) {
        return e;
    }
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, sample_stream_kernel<K_SEL | K_SUMS | K_PEN>, kThreads, smem_bytes);
}

static cudaError_t ensure_row_ids_attributes(size_t smem_bytes) {
    static int  configured_smem[64] = {0};
    int         dev                 = 0;
    cudaError_t e                   = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    if (dev < 0 || dev >= 64) {
        return cudaErrorInvalidDevice;
    }
    if (smem_bytes > 48 * 1024 && (int) smem_bytes > configured_smem[dev]) {
        e = cudaFuncSetAttribute(row_ids_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem_bytes);
        if (e != cudaSuccess) {
            return e;
        }
        configured_smem[dev] = (int) smem_bytes;
    }
    return cudaSuccess;
}

size_t finish_rows_smem(bool fast) { return sizeof(FinishShared) + (size_t) (fast ? kFinBytes : kFinGeneralBytes); }

static cudaError_t ensure_finish_attributes() {
    static int  configured[64] = {0};
    int         dev            = 0;
    cudaError_t e              = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    if (dev < 0 || dev >= 64) {
        return cudaErrorInvalidDevice;
    }
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(finish_rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) finish_rows_smem(true));
        if (e == cudaSuccess) {
            e = cudaFuncSetAttribute(finish_rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) finish_rows_smem(false));
        }
        if (e != cudaSuccess) {
            return e;
        }
        configured[dev] = 1;
    }
    return cudaSuccess;
}

/* Thread blocks of the finishing kernel that the current device holds at once. */
cudaError_t finish_rows_max_ctas(int sms, int *out) {
    cudaError_t e = ensure_finish_attributes();
    if (e != cudaSuccess) {
        return e;
    }
    int per_sm = 0;
    e          = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, finish_rows_kernel<false>, kThreads, finish_rows_smem(false));
    *out       = per_sm * sms;
    return e;
}

cudaError_t launch_sample_stream(const SampleParams &p, int grid, size_t smem_bytes, int finish_grid, cudaStream_t stream) {
    cudaError_t e = ensure_attributes(smem_bytes);
    if (e == cudaSuccess) {
        e = ensure_finish_attributes();
    }
    if (e != cudaSuccess) {
        return e;
    }
    if (p.id_slots > 0) { /* rows may bring more ids than the stream kernel counts by itself: prepare their lists first */
        const size_t ids_smem = ((size_t) p.id_slots * 2 + (size_t) p.bucket_cap) * sizeof(int);
        e                     = ensure_row_ids_attributes(ids_smem);
        if (e != cudaSuccess) {
            return e;
        }
        row_ids_kernel<<<dim3((unsigned) p.n_rows), dim3(kIdThreads), ids_smem, stream>>>(p);
        e = cudaGetLastError();
        if (e != cudaSuccess) {
            return e;
        }
    }
    /* Programmatic dependent launch, both kernels: the thread blocks are placed while the kernel before them
     * in the stream drains, and wait (griddepcontrol.wait) until that kernel is complete and visible before they
     * touch global memory. No thread block of the stream kernel or of the small finishing kernel ever waits for another one of
     * its grid. Those of the general finishing kernel do, where a launch has wide top-p rows: for pieces of such a row that
     * have been dealt out, and every one of those lies with a thread block that is running (a block takes pieces for the
     * warps it has); and, before they end, a bounded while for rows to help with. So neither grid needs co-residency. */
    cudaLaunchConfig_t  cfg{};
    cudaLaunchAttribute attr[1];
    cfg.gridDim          = dim3((unsigned) grid);
    cfg.blockDim         = dim3(kThreads);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream           = stream;
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs                                          = attr;
    cfg.numAttrs                                       = 1;
    /* the instantiation that carries no more than the kinds of rows the caller vouched for, and the penalties' code
     * only where the launch brings ids */
    const bool pen   = p.hist != nullptr || p.extra != nullptr;
    const int  kinds = (p.flags & F_SELECT_ONLY) != 0u ? (K_SEL | K_SUMS) : (p.flags & F_GREEDY_ONLY) != 0u ? 0 : (p.flags & F_FAST_ONLY) != 0u ? K_SEL : (K_SEL | K_SUMS);
    const bool plain     = p.aligned != 0 && p.softcap == nullptr && p.mask == nullptr && p.out_logits == nullptr;
    const bool short_ids = !pen || p.many_ids == 0; /* no row brings more ids than a thread block has threads */
#define GB_STREAM_CASE(K)                                                  \
    case (K):                                                              \
        e = cudaLaunchKernelEx(&cfg, sample_stream_kernel<(K)>, p);        \
        break;
    switch (kinds | (pen ? K_PEN : 0) | (plain ? K_PLAIN : 0) | (short_ids ? K_SHORT : 0)) {
        GB_STREAM_ALL(GB_STREAM_CASE)
    default:
        e = cudaErrorInvalidValue;
        break;
    }
#undef GB_STREAM_CASE
    if (e != cudaSuccess) {
        return e;
    }
    cfg.gridDim          = dim3((unsigned) finish_grid);
    cfg.dynamicSmemBytes = finish_rows_smem((p.flags & F_FAST_ONLY) != 0u);
    if ((p.flags & (F_GREEDY_ONLY | F_INLINE_TOPK)) != 0u) {
        return cudaSuccess; /* the stream kernel writes the tokens itself */
    }
    /* one finishing kernel per launch: the small one when the caller vouched for greedy / top-k rows, else the
     * general one (it finishes every kind of row; a third kernel in the chain of dependent launches cost 7 - 8 us
     * even when it had no row to take, as much as the general kernel costs more than the small one) */
    if ((p.flags & F_FAST_ONLY) != 0u) {
        return cudaLaunchKernelEx(&cfg, finish_rows_kernel<true>, p);
    }
    return cudaLaunchKernelEx(&cfg, finish_rows_kernel<false>, p);
}

} /* namespace gb */
