/*
 * sampler_wide.cuh — top-p rows whose nucleus is wide, part of finish_rows_kernel<false> (included by
 * sampler_stream.cu behind the helpers it uses).
 *
 * Such a row is worked on by every thread block of the finishing kernel that has nothing else to do. It is cut into
 * pieces of kWidePiece columns, dealt out one by one to warps, which share nothing but counters while they work:
 *
 *   pass 1  e_i = expf((x_i - max) / T), correctly rounded, kept in the row's scratch; their sum per piece in double; and
 *           a histogram of their mass over kWideBins bins of their bits, in whole units of S0 / 2^30 (S0: the row's sum
 *           as the stream kernel formed it).
 *   pass 2  starts when every piece is through pass 1: S is known, and from the histogram the bins in which the walk
 *           reaches top_p and in which the draw will fall, with a margin for the units' rounding. p_i = (float)(e_i / S);
 *           what lies above a window is summed in units of 2^-62, what lies in it is listed (a few entries, or a few hundred).
 *   end     the thread block that completes pass 2 walks the two lists exactly, in (p desc, id asc) order, and has the
 *           token. Whatever the lists do not decide (more entries than they hold, a crossing outside its window, equal
 *           probabilities at a window's edge) goes to multipass_row, one thread block for the row. Rows with thousands of
 *           equal values are where that happens: the lists outrun their room, and equal masses round to units alike, so
 *           that the window misses its target by more than the margin allows for. The two passes are lost then: 256 rows
 *           of 128256 that end in 10^5 equal values 8.1 -> 8.6 ms. Logits that were 16 bits wide do not come near it.
 *
 * Nobody waits for a thread block that has not begun: the block that owns the row takes pieces like any other, and once
 * they are all dealt out, every piece lies with a block that runs. A wait that runs out all the same leaves the row to the
 * blocks that are still at it. Sums do not depend on who took which piece, nor does the order of the lists matter.
 *
 * Pass 1 is bound by the issue of its instructions at the finishing kernel's 16 warps per SM: 25 SM cycles per 32 values,
 * where its double arithmetic takes 6 and its conversions 8; a launch's first piece waits for the code as well, 4 us. 256
 * rows of 128256 columns, top-p 0.95 (98 of them wide): 428 us with a thread block and a dozen sweeps per row, 135 - 139
 * now; 24 wide rows of 100003 among 96: 402 -> 69. Of the 98 rows' 77 us from the first row opened to the last token pass 1 takes 38,
 * what is added up and waited for between the passes 4, the windows 3, pass 2 12; 16 are the last row's end and uneven work.
 * Pieces of 512 for a warp: when they came in (the 24 rows took 93 us) pieces of
 * 1024 took 99, and pieces of 2048 for a thread block, a barrier each, 204 us on the 105.
 */
#pragma once

#include "sampler_wide_math.cuh"

namespace gb {

constexpr int kWideRank = 512;  /* lists up to here are walked by ranking */
constexpr int kWideIds  = 1024; /* ids of a row that a thread block keeps at hand; more are read from memory for every piece */

/* What the wide row that a slot (row copy) holds is. */
struct __align__(16) WideCtl {
    int    rem1, rem2;    /* pieces not yet dealt out of pass 1 and pass 2; rem1 at most 0: no row to help with */
    int    done1, done2;  /* pieces through pass 1; pieces whose thread block of pass 1 has left pass 2 */
    int    n_cut, n_pick; /* entries of the two lists */
    int    row, st;
    float  row_max;
    int    row_arg;
    double S0;
    unsigned long long above_cut, above_pick; /* of p, above the two windows (wide_mass): whole numbers, so in any order */
    int                n_above;               /* entries above the window of the crossing */
    int                pad[3];
};
static_assert(sizeof(WideCtl) == 4 * kWideCtlInts, "a slot's words");

/* What a piece adds up to. */
struct WidePart {
    double sum; /* of e */
};
static_assert(sizeof(WidePart) == kWidePartBytes, "the host sizes the parts");

/* A thread block's memory while it works on wide rows (the merged candidates' memory). */
struct __align__(16) WideShared {
    unsigned           hist[kWideBins];
    float              x[kWarps][2][kWidePiece];    /* every warp's pieces: the one in work and the next on its way */
    unsigned           cnt[kWarps][kWidePiece / 2]; /* how often an id of the warp's piece occurs, 16 bits each; zero between pieces */
    int                ids[kWideIds];
    unsigned           wsum[kWarps], open[2 * kWarps];
    int                win[4]; /* the crossing's window, lowest and highest bin; the draw's */
    int                next, slot, mine;
    int                best_rank;
    unsigned long long best, best_mass;
    RowCfg             cfg; /* the row's, for the functions that finish it */
};

__device__ __forceinline__ int ld_volatile(const int *q) { return *reinterpret_cast<const volatile int *>(q); }

/* Bins of a row's histogram: the bits of e from the floor up to 1, in at most kWideBins equal steps of a power of two.
 * Entries with p < (1 - top_p) / V add up to less than 1 - top_p, so the walk crosses above half of that. */
struct WideBins {
    unsigned k_floor;
    int      shift;
    float    unit; /* 2^30 / S0 */
    __device__ __forceinline__ WideBins(double S0, float top_p, int V) {
        const float f       = __double2float_rn(0.5 * (1.0 - (double) top_p) / (double) V * S0);
        k_floor             = f > 0.0f && f < 1.0f ? __float_as_uint(f) : 1u;
        const unsigned span = __float_as_uint(1.0f) - k_floor;
        shift               = max(0, 32 - __clz(span) - kWideBinsLog);
        unit                = __double2float_rn(0x1p30 / S0);
    }
    __device__ __forceinline__ unsigned bin(unsigned k) const { return (k - k_floor) >> shift; } /* kWideBins and more: below the floor */
    __device__ __forceinline__ unsigned edge(int b) const { return k_floor + ((unsigned) b << shift); } /* lowest bits of bin b */
};

/* Where one of the two walks ends. */
struct WideHit {
    bool               found;
    unsigned long long word; /* (bits of p, id) as composite() packs them */
    double             mass; /* of everything up to and with it */
    long long          rank; /* its place, from 1, in its list */
};

/* The first of the n listed entries, in (p desc, id asc) order, at which base + running mass reaches (inclusive) or
 * exceeds the target. Masses are added in units of 2^-62 (wide_mass), so the order of the list does not matter. All threads call. */
__device__ WideHit wide_walk(const Grp &g, GroupShared *gs, WideShared *ws, const Pair *list, int n, long long base, double target, bool inclusive, int idx_bits) {
    WideHit out;
    if (n <= kWideRank) {
        unsigned long long *word = reinterpret_cast<unsigned long long *>(&ws->x[0][0][0]), *mass = word + kWideRank;
        static_assert(sizeof(ws->x) >= 2 * kWideRank * 8, "the list fits");
        g.sync();
        for (int i = g.tid; i < n; i += g.n) {
            const unsigned long long w  = __ldcg(reinterpret_cast<const unsigned long long *>(list + i)); /* p, then the id */
            const float              pv = __uint_as_float((unsigned) w);
            word[i]                     = composite(__float_as_uint(pv), (int) (w >> 32), idx_bits);
            mass[i]                     = (unsigned long long) wide_mass(pv);
        }
        if (g.tid == 0) {
            ws->best = 0ull;
        }
        g.sync();
        unsigned long long mine = 0ull, my_sum[kWideRank / kThreads];
        int                my_rank[kWideRank / kThreads];
#pragma unroll
        for (int q = 0; q < kWideRank / kThreads; q++) {
            const int i = g.tid + q * kThreads;
            my_sum[q]   = 0ull;
            my_rank[q]  = 0;
            if (i < n) {
                const unsigned long long me = word[i];
#pragma unroll 4
                for (int j = 0; j < n; j++) {
                    const bool up = word[j] >= me;
                    my_sum[q] += up ? mass[j] : 0ull;
                    my_rank[q] += up ? 1 : 0;
                }
                const double at = mass_value(base + (long long) my_sum[q]);
                if (inclusive ? at >= target : at > target) {
                    mine = max(mine, me);
                }
            }
        }
        if (mine != 0ull) {
            atomicMax(&ws->best, mine);
        }
        g.sync();
        out.word = ws->best;
#pragma unroll
        for (int q = 0; q < kWideRank / kThreads; q++) {
            const int i = g.tid + q * kThreads;
            if (i < n && word[i] == out.word) {
                ws->best_mass = my_sum[q];
                ws->best_rank = my_rank[q];
            }
        }
        g.sync();
        out.found = out.word != 0ull;
        out.mass  = mass_value(base + (long long) ws->best_mass);
        out.rank  = (long long) ws->best_rank;
        g.sync();
        return out;
    }
    /* long lists (many equal values): byte by byte as the multi-pass path walks its own */
    auto     sweep = [&](auto &&f) { list_sweep(g, list, n, f); };
    auto     keyf  = [](float pv) { return __float_as_uint(pv); };
    auto     massf = [](float pv, int) { return (double) pv; };
    double  *hm    = reinterpret_cast<double *>(&ws->x[0][0][0]);
    int     *hc    = reinterpret_cast<int *>(hm + kWarps * 256);
    static_assert(sizeof(ws->x) >= (size_t) kWarps * 256 * 12, "a byte histogram per warp fits");
    const double   rest = target - mass_value(base);
    const RadixOut ro   = radix_mass(g, gs, hm, hc, kWarps, 0x1p62, sweep, rest, inclusive, keyf, massf);
    out.found           = ro.found;
    out.word            = ro.found ? resolve_ties(g, gs, sweep, idx_bits, ro, rest, inclusive, keyf, massf) : 0ull;
    long long m = 0, c = 0;
    sweep([&](float pv, int i) {
        if (composite(__float_as_uint(pv), i, idx_bits) >= out.word) {
            m += wide_mass(pv);
            c++;
        }
    });
    out.mass = mass_value(base + group_sum_ll(g, gs, m));
    out.rank = group_sum_ll(g, gs, c);
    return out;
}

/* The same for at most 32 entries, by one warp: an entry per lane, each met with all others. The windows are a bin or two of
 * thousands, most lists hold less than ten: a row's end, 10 us by all threads with their barriers, takes a warp 4. (Bins instead
 * of one against all in wide_walk: 13 us.) */
__device__ __forceinline__ WideHit wide_walk_few(int lane, const Pair *list, int n, long long base, double target, bool inclusive, int idx_bits) {
    const unsigned long long e  = lane < n ? __ldcg(reinterpret_cast<const unsigned long long *>(list + lane)) : 0ull; /* p, then the id */
    const unsigned long long me = lane < n ? composite((unsigned) e, (int) (e >> 32), idx_bits) : 0ull;
    const long long          m  = lane < n ? wide_mass(__uint_as_float((unsigned) e)) : 0;
    long long                to = 0; /* of the entries up to the lane's */
    int                      rank = 0;
#pragma unroll 4
    for (int j = 0; j < n; j++) {
        const bool      up = __shfl_sync(0xffffffffu, me, j) >= me;
        const long long mj = __shfl_sync(0xffffffffu, m, j);
        to += up ? mj : 0;
        rank += up ? 1 : 0;
    }
    const double             at = mass_value(base + to);
    unsigned long long best = lane < n && (inclusive ? at >= target : at > target) ? me : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    }
    const int from = __ffs(__ballot_sync(0xffffffffu, lane < n && me == best)) - 1;
    WideHit   out;
    out.found = best != 0ull;
    out.word  = best;
    out.mass  = mass_value(base + __shfl_sync(0xffffffffu, to, max(from, 0)));
    out.rank  = (long long) __shfl_sync(0xffffffffu, rank, max(from, 0));
    return out;
}

/* Takes a piece of a row of which *rem were left: its number, -1 when there was none. Called by a whole warp; the answer
 * takes a round trip, so a warp asks a piece ahead (lane 0 holds what came back). */
__device__ __forceinline__ int wide_ask(int *rem, int lane) { return lane == 0 ? atomicSub(rem, 1) : 0; }
__device__ __forceinline__ int wide_got(int left, int pieces) {
    const int l = __shfl_sync(0xffffffffu, left, 0);
    return l > 0 ? pieces - l : -1;
}

/* The last of a row's thread blocks: the two walks, the token, and the slot made ready for its next row. `listed`: the block
 * took part in pass 2, so that is through; one that had given up waiting for pass 1 does not know its windows, and nobody
 * need have made the lists. */
__device__ __noinline__ void wide_finish(const SampleParams &p, GroupShared *gs, WideShared *ws, int slot, bool listed, double S, unsigned long long rng0, void *save_mem) {
    const Grp       g      = whole_block();
    const RowCfg    r      = ws->cfg;
    WideCtl        *ctl    = p.wide_ctl + slot;
    const int       V      = p.V, idx_bits = 32 - __clz(max(V - 1, 1));
    const Pair     *list   = p.gen_list + (size_t) slot * (size_t) p.gen_list_cap;
    const int       half   = p.gen_list_cap / 2;
    const WideBins  bins(__ldcg(&ctl->S0), r.top_p, V);
    const int       n_cut = __ldcg(&ctl->n_cut), n_pick = __ldcg(&ctl->n_pick);
    const bool      few   = listed && n_cut <= 32 && n_pick <= 32; /* nearly always: one warp finishes the row */
    const int       w0 = ws->win[0], w1 = ws->win[1], w2 = ws->win[2], w3 = ws->win[3];
    uint4          *gh    = reinterpret_cast<uint4 *>(p.wide_hist + (size_t) slot * kWideBins);
    auto            clear = [&](int from, int step) { /* for the slot's next row */
        for (int i = from; i < kWideBins / 4; i += step) {
            gh[i] = make_uint4(0u, 0u, 0u, 0u);
        }
    };
    const long long a_cut = (long long) __ldcg(&ctl->above_cut), a_pick = (long long) __ldcg(&ctl->above_pick), above = __ldcg(&ctl->n_above);
    WideHit   cut{}, pick{};
    bool      ok = listed && n_cut <= half && n_pick <= half && n_cut > 0 && mass_value(a_cut) < (double) r.top_p;
    /* p of the nearest entries outside a window: an entry of the window that shares it cannot be placed */
    const WideQuotient quot(S);
    auto p_at   = [&](unsigned k) { return quot(__uint_as_float(k)); };
    auto inside = [&](unsigned long long word, int lo, int hi) {
        const float pv = __uint_as_float((unsigned) (word >> idx_bits));
        return pv > 0.0f && (hi >= kWideBins - 1 || pv < p_at(bins.edge(hi + 1))) && pv > p_at(bins.edge(lo) - 1u);
    };
    auto drawn = [&](unsigned long long rng) { return (double) unit_from(xorshift_next(rng)) * cut.mass; };
    if (few) {
        if (g.warp != 0) {
            clear(g.tid - 32, kThreads - 32);
        } else {
            if (ok) {
                cut = wide_walk_few(g.lane, list, n_cut, a_cut, (double) r.top_p, true, idx_bits);
                ok  = cut.found && inside(cut.word, w0, w1);
            }
            if (ok) {
                const double u = drawn(r.rng);
                ok             = mass_value(a_pick) <= u;
                if (ok) {
                    pick = wide_walk_few(g.lane, list + half, n_pick, a_pick, u, false, idx_bits);
                    ok   = pick.found && inside(pick.word, w2, w3);
                }
            }
        }
        ok = __syncthreads_or(g.warp == 0 && ok) != 0; /* the first thread holds what there is to write */
    } else {
        if (ok) {
            cut = wide_walk(g, gs, ws, list, n_cut, a_cut, (double) r.top_p, true, idx_bits);
            ok  = cut.found && inside(cut.word, w0, w1);
        }
        if (ok) {
            const double u = drawn(r.rng);
            ok             = mass_value(a_pick) <= u;
            if (ok) {
                pick = wide_walk(g, gs, ws, list + half, n_pick, a_pick, u, false, idx_bits);
                ok   = pick.found && inside(pick.word, w2, w3);
            }
        }
    }
    int st = __ldcg(&ctl->st);
    if (ok) {
        if (g.tid == 0) {
            const unsigned long long id_mask = (1ull << idx_bits) - 1ull;
            const unsigned long long word    = max(pick.word, cut.word); /* the draw does not leave the nucleus (sampler.c:292) */
            p.tokens[r.row]                  = min((int) (id_mask - (word & id_mask)), V - 1) + p.vocab_offset;
            if (p.kept_cap > 0) {
                p.kept_n[r.row] = (int) (above + cut.rank);
            }
            atomicAdd(&p.wide_head->by_lists, 1);
            atomicMax(&p.wide_head->longest, max(n_cut, n_pick));
        }
        st |= ST_SLOW_PATH | (p.kept_cap > 0 ? (int) ST_KEPT_PARTIAL : 0);
    } else {
        st |= multipass_row(p, gs, &ws->cfg, __ldcg(&ctl->row_max), __ldcg(&ctl->row_arg), ws, (int) offsetof(WideShared, cfg), slot, save_mem);
    }
    if (!few) {
        clear(g.tid, g.n);
    }
    __threadfence();
    g.sync();
    if (g.tid == 0) { /* the row's status comes behind all that is done to its slot */
        if (p.n_rows > p.pool_slots) {
            atomicExch(&p.pool[slot], 0);
            __threadfence();
        }
        row_epilogue(p, r, r.row, st, rng0);
    }
    g.sync();
}

/* Works on the row of a slot. `first`: the first of the n_first pieces that the thread block has been dealt already, one for each
 * of its first warps (all threads call). */
__device__ __noinline__ void wide_join(const SampleParams &p, GroupShared *gs, WideShared *ws, int slot, int first, int n_first, void *save_mem) {
    const Grp       g       = whole_block();
    WideCtl        *ctl     = p.wide_ctl + slot;
    const int       V       = p.V, pieces = (V + kWidePiece - 1) / kWidePiece;
    int             left    = wide_ask(&ctl->rem1, g.lane);
    const int       row     = __ldcg(&ctl->row);
    const float     row_max = __ldcg(&ctl->row_max);
    const double    S0      = __ldcg(&ctl->S0);
    for (int i = g.tid; i < kWideBins / 4; i += g.n) {
        reinterpret_cast<uint4 *>(ws->hist)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    for (int i = g.tid; i < kWarps * kWidePiece / 8; i += g.n) {
        reinterpret_cast<uint4 *>(ws->cnt)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (g.tid == 0) {
        ws->mine = 0;
    }
    const RawCfg rc = raw_config(p, row, true);
    RowCfg       r  = row_config(p, row, rc, true);
    if (p.out_logits != nullptr) { /* read back as it is sampled from (row_again) */
        r.cap    = 0.0f;
        r.mrow   = nullptr;
        r.pen_on = false;
    }
    if (g.tid == 0) {
        ws->cfg = r; /* here, not where the row is finished: nothing of it need be kept in registers until then */
    }
    const WideBins bins(S0, r.top_p, V);
    const float   *src    = row_again(p, row);
    const bool     src_al = again_aligned(p);
    float         *gr     = p.gen_rows + (size_t) slot * (size_t) p.gen_stride;
    WidePart      *parts  = p.wide_part + (size_t) slot * (size_t) pieces;
    const double   t32    = exp2((double) g.lane * 0x1p-5);
    const int      n_ids  = r.pen_on ? r.H + r.E : 0;
    const bool     pro    = r.cap > 0.0f || r.mrow != nullptr;
    for (int j = g.tid; j < min(n_ids, kWideIds); j += g.n) {
        ws->ids[j] = hist_id(r, j, p.vocab_offset);
    }
    g.sync();
    /* ---- pass 1 ---- */
    constexpr int kPer = 8, kSteps = kWidePiece / (32 * kPer); /* eight values of a lane at a time: as many independent chains */
    auto column = [&](int step, int q) { return step * (32 * kPer) + (q >> 2) * 128 + 4 * g.lane + (q & 3); }; /* inside the piece */
    /* A piece on its way into one of the warp's two buffers. What bounds the passes is the bytes on their way: with eight
     * values per lane in registers and none ahead 16 KB per SM, 3.5 TB/s with nothing else done. */
    auto fetch = [&](const float *from, bool al, int end, int pc, int to, float pad) {
        const int    s0  = pc * kWidePiece, n = min(kWidePiece, end - s0);
        float       *buf = ws->x[g.warp][to];
        const float *at  = from + s0;
        if (al) {
#pragma unroll
            for (int i = 4 * g.lane; i < kWidePiece; i += 128) {
                if (i + 4 <= n) {
                    copy_quad_async(buf + i, at + i);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        buf[i + q] = i + q < n ? at[i + q] : pad;
                    }
                }
            }
        } else {
#pragma unroll 4
            for (int i = g.lane; i < kWidePiece; i += 32) {
                if (i < n) {
                    copy_word_async(buf + i, at + i);
                } else {
                    buf[i] = pad;
                }
            }
        }
        async_copies_commit();
    };
    auto take_values = [&](int from, int step, float (&e)[kPer]) {
#pragma unroll
        for (int h = 0; h < kPer; h += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(&ws->x[g.warp][from][column(step, h)]);
            e[h] = v.x, e[h + 1] = v.y, e[h + 2] = v.z, e[h + 3] = v.w;
        }
    };
    auto one_behind = [&](bool more) { /* the piece in work has arrived; the next may be on its way */
        async_copies_wait_but(more ? 1 : 0);
        __syncwarp();
    };
    int       mine  = 0;
    int       piece = g.warp < n_first ? first + g.warp : -1;
    unsigned *cnt   = ws->cnt[g.warp];
    if (piece < 0) {
        piece = wide_got(left, pieces);
        left  = piece >= 0 ? wide_ask(&ctl->rem1, g.lane) : 0;
    }
    if (piece >= 0) {
        fetch(src, src_al, V, piece, 0, -CUDART_INF_F);
    }
    for (int in = 0; piece >= 0; in ^= 1) {
        const int s0   = piece * kWidePiece;
        const int next = wide_got(left, pieces);
        if (next >= 0) {
            left = wide_ask(&ctl->rem1, g.lane);
            fetch(src, src_al, V, next, in ^ 1, -CUDART_INF_F);
        }
        if (n_ids > 0) { /* how often each id of the piece occurs */
            for (int j = g.lane; j < n_ids; j += 32) {
                const int li = (j < kWideIds ? ws->ids[j] : hist_id(r, j, p.vocab_offset)) - s0;
                if (li >= 0 && li < kWidePiece && li + s0 < V) {
                    atomicAdd(&cnt[li >> 1], 1u << (16 * (li & 1)));
                }
            }
            __syncwarp();
        }
        one_behind(next >= 0);
        double sum = 0.0;
#pragma unroll 1
        for (int step = 0; step < kSteps; step++) {
            float e[kPer];
            take_values(in, step, e);
            if (pro || n_ids > 0) {
#pragma unroll
                for (int h = 0; h < kPer; h += 4) {
                    const int      c     = s0 + column(step, h);
                    uint2         &cw    = *reinterpret_cast<uint2 *>(cnt + (column(step, h) >> 1));
                    const unsigned c4[4] = {cw.x & 0xffffu, cw.x >> 16, cw.y & 0xffffu, cw.y >> 16};
                    if (pro) {
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if (c + q < V) {
                                e[h + q] = prologue_one(e[h + q], c + q, r.cap, r.mrow);
                            }
                        }
                    }
                    if ((cw.x | cw.y) != 0u) {
                        cw = make_uint2(0u, 0u);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if (c4[q] != 0u) {
                                e[h + q] = penalise(e[h + q], (int) c4[q], r.rep, r.freq, r.pres);
                            }
                        }
                    }
                }
                __syncwarp();
            }
#pragma unroll
            for (int q = 0; q < kPer; q++) {
                e[q] = wide_exp(scaled_arg(e[q], row_max, r.inv_t), t32);
            }
#pragma unroll
            for (int h = 0; h < kPer; h += 4) {
                const int c = s0 + column(step, h);
                sum += ((double) e[h] + (double) e[h + 1]) + ((double) e[h + 2] + (double) e[h + 3]);
                if (c + 4 <= p.gen_stride) {
                    *reinterpret_cast<float4 *>(gr + c) = make_float4(e[h], e[h + 1], e[h + 2], e[h + 3]);
                }
            }
#pragma unroll
            for (int q = 0; q < kPer; q++) {
                const unsigned b = bins.bin(__float_as_uint(e[q])), m = __float2uint_rn(e[q] * bins.unit);
                if (b < (unsigned) kWideBins) {
                    atomicAdd(&ws->hist[b], m);
                }
            }
        }
        sum = warp_sum_d(sum);
        if (g.lane == 0) {
            parts[piece].sum = sum;
        }
        mine++;
        piece = next;
        __syncwarp(); /* the buffer is free */
    }
    if (g.lane == 0 && mine > 0) {
        atomicAdd(&ws->mine, mine);
    }
    g.sync();
    unsigned *gh = p.wide_hist + (size_t) slot * kWideBins;
    for (int i = g.tid; i < kWideBins; i += g.n) {
        const unsigned v = ws->hist[i];
        if (v != 0u) {
            atomicAdd(&gh[i], v);
        }
    }
    __threadfence();
    g.sync();
    if (g.tid == 0) {
        atomicAdd(&ctl->done1, ws->mine);
        /* every piece lies with a thread block that runs: the wait ends */
        const unsigned long long t0 = global_ns();
        bool                     in = true;
        while (ld_volatile(&ctl->done1) < pieces && in) {
            __nanosleep(50);
            in = global_ns() - t0 < p.wide_wait_ns;
        }
        __threadfence();
        ws->next = in ? 1 : 0;
    }
    g.sync();
    /* A row's last thread block finishes it, whoever that is: each was dealt a piece of pass 1 at least, and counts its own
     * once more when it is through here. The slot is then free for another row. */
    auto leave = [&](bool listed, double S) {
        __threadfence();
        g.sync();
        if (g.tid == 0) {
            ws->next = atomicAdd(&ctl->done2, ws->mine) + ws->mine == pieces ? 1 : 0;
            __threadfence();
        }
        g.sync();
        if (ws->next != 0) {
            wide_finish(p, gs, ws, slot, listed, S, rc.rng, save_mem);
        }
    };
    if (ws->next == 0) { /* gave up: its pieces of pass 1 are done all the same, so the row goes on without the block */
        if (g.tid == 0) {
            atomicAdd(&p.wide_head->gave_up, 1);
        }
        leave(false, 1.0);
        return;
    }
    left = wide_ask(&ctl->rem2, g.lane);
    /* ---- S, and the two windows ---- */
    constexpr int kOwn = kWideBins / kThreads;
    unsigned      h[kOwn], run = 0u; /* thread t holds kOwn bins, the highest with thread 0 */
    const int     b0 = kWideBins - kOwn * (g.tid + 1);
#pragma unroll
    for (int q = 0; q < kOwn / 4; q++) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(gh + b0) + q);
        h[4 * q] = v.x, h[4 * q + 1] = v.y, h[4 * q + 2] = v.z, h[4 * q + 3] = v.w;
    }
    double S = 0.0;
    for (int t = g.tid; t < pieces; t += g.n) {
        S += __ldcg(&parts[t].sum);
    }
    S = group_sum_d(g, gs, S);
    const WideQuotient quot(S);
    {
#pragma unroll
        for (int q = 0; q < kOwn; q++) {
            run += h[q];
        }
        unsigned incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned up = __shfl_up_sync(0xffffffffu, incl, o);
            if (g.lane >= o) {
                incl += up;
            }
        }
        if (g.lane == 31) {
            ws->wsum[g.warp] = incl;
        }
        if (g.tid < 4) {
            ws->win[g.tid] = 0;
        }
        g.sync();
        unsigned before = incl - run;
        for (int w = 0; w < g.warp; w++) {
            before += ws->wsum[w];
        }
        /* Units that reach a target, less and more the margin (the units' rounding moves the sum of n entries by 0.29
         * sqrt(n), rms): the highest bin up to which the target can be reached, and the one up to which it surely is. */
        unsigned long long rng    = r.rng;
        const double       u01    = (double) unit_from(xorshift_next(rng));
        const double       margin = 1024.0 + (double) (V >> 8);
        const double       t_cut  = (double) r.top_p * S * (double) bins.unit;
        auto place = [&](int which, double target) { /* the highest bin b so that the units in bins >= b reach the target */
            const unsigned t = __double2uint_ru(fmax(target, 1e-3)); /* units are whole */
            if (before < t && before + run >= t) {
                unsigned acc = before;
                int      b   = b0;
#pragma unroll
                for (int q = kOwn - 1; q >= 0; q--) {
                    const bool below = acc < t;
                    acc += h[q];
                    b = below && acc >= t ? b0 + q : b;
                }
                ws->win[which] = b;
            }
        };
        place(1, t_cut - margin);
        place(0, t_cut + margin);
        g.sync();
        /* the draw's target lies between u and u times what the crossing entry can add at most */
        const double p_one = (double) __uint_as_float(bins.edge(ws->win[1] + 1)) * (double) bins.unit;
        place(3, u01 * t_cut - margin);
        place(2, u01 * (t_cut + p_one) + margin);
        g.sync();
        if (g.tid == 0) {
            ws->win[2] = max(ws->win[2], ws->win[0]);
        }
        g.sync();
    }
    /* ---- pass 2 ---- */
    const unsigned c_lo = bins.edge(ws->win[0]), c_hi = ws->win[1] >= kWideBins - 1 ? 0xffffffffu : bins.edge(ws->win[1] + 1);
    const unsigned k_lo = bins.edge(ws->win[2]), k_hi = ws->win[3] >= kWideBins - 1 ? 0xffffffffu : bins.edge(ws->win[3] + 1);
    const int      half = p.gen_list_cap / 2;
    Pair          *list = p.gen_list + (size_t) slot * (size_t) p.gen_list_cap;
    /* A lane that finds a list full counts nothing more in it: its count is beyond its room already, which is all that is
     * asked of it then. (Counted on, 10^5 equal values of a row queued for one word: 256 rows of 128256 that end in equal
     * values took 12.6 ms, 8.1 on the multi-pass path alone.) */
    bool           full_cut = false, full_pick = false;
    auto           note = [&](bool &full, int *count, Pair *to, float pv, int id) {
        if (!full) {
            const int pos = atomicAdd(count, 1);
            if (pos < half) {
                to[pos].v   = pv;
                to[pos].idx = id;
            } else {
                full = true;
            }
        }
    };
    piece = wide_got(left, pieces);
    left  = piece >= 0 ? wide_ask(&ctl->rem2, g.lane) : 0;
    if (piece >= 0) {
        fetch(gr, true, (int) p.gen_stride, piece, 0, 0.0f);
    }
    long long a_cut = 0, a_pick = 0;
    int       above = 0;
    for (int in = 0; piece >= 0; in ^= 1) {
        const int s0   = piece * kWidePiece;
        const int next = wide_got(left, pieces);
        if (next >= 0) {
            left = wide_ask(&ctl->rem2, g.lane);
            fetch(gr, true, (int) p.gen_stride, next, in ^ 1, 0.0f);
        }
        one_behind(next >= 0);
#pragma unroll 1
        for (int step = 0; step < kSteps; step++) {
            float    e[kPer];
            unsigned listed = 0u; /* which of the lane's values lie in a window */
            bool     unsure = false; /* one of them wants the division */
            take_values(in, step, e);
#pragma unroll
            for (int q = 0; q < kPer; q++) {
                const unsigned k = __float_as_uint(e[q]);
                if (__any_sync(0xffffffffu, k >= c_lo)) { /* most of a row lies below the nucleus; the draw's window lies no lower */
                    const long long m = __float2ll_rz(quot.quick(e[q], unsure));
                    if (k >= c_hi) {
                        a_cut += m;
                        above++;
                    }
                    if (k >= k_hi) {
                        a_pick += m;
                    }
                    listed |= (k - c_lo < c_hi - c_lo || k - k_lo < k_hi - k_lo) ? 1u << q : 0u;
                }
            }
            if (unsure) { /* masses are whole numbers: what went in comes out again */
#pragma unroll
                for (int q = 0; q < kPer; q++) {
                    const unsigned  k = __float_as_uint(e[q]);
                    const long long m = wide_mass(quot.divide(e[q])) - __float2ll_rz(quot.quick(e[q], unsure));
                    a_cut += k >= c_hi ? m : 0;
                    a_pick += k >= k_hi ? m : 0;
                }
            }
            if (listed != 0u) {
#pragma unroll
                for (int q = 0; q < kPer; q++) {
                    if ((listed >> q) & 1u) {
                        const unsigned k  = __float_as_uint(e[q]);
                        const float    pv = quot(e[q]);
                        const int      id = s0 + column(step, q);
                        if (k - c_lo < c_hi - c_lo) {
                            note(full_cut, &ctl->n_cut, list, pv, id);
                        }
                        if (k - k_lo < k_hi - k_lo) {
                            note(full_pick, &ctl->n_pick, list + half, pv, id);
                        }
                    }
                }
            }
        }
        piece = next;
        __syncwarp();
    }
    a_cut  = warp_sum_ll(a_cut);
    a_pick = warp_sum_ll(a_pick);
    above  = __reduce_add_sync(0xffffffffu, above);
    if (g.lane == 0 && (a_cut | a_pick) != 0) { /* what lies above has a mass */
        atomicAdd(&ctl->above_cut, (unsigned long long) a_cut);
        atomicAdd(&ctl->above_pick, (unsigned long long) a_pick);
        atomicAdd(&ctl->n_above, above);
    }
    leave(true, S);
}

/* Opens the row in a slot that the thread block has claimed, for everybody; the block then works on it itself. */
__device__ __forceinline__ void wide_open(const SampleParams &p, GroupShared *gs, WideShared *ws, int slot, int row, int st, float row_max, int row_arg, double S0, void *save_mem) {
    WideCtl  *ctl    = p.wide_ctl + slot;
    const int pieces = (p.V + kWidePiece - 1) / kWidePiece, own = min(pieces, kWarps);
    if (threadIdx.x == 0) {
        ctl->done1       = 0;
        ctl->done2       = 0;
        ctl->n_cut       = 0;
        ctl->n_pick      = 0;
        ctl->row         = row;
        ctl->st          = st;
        ctl->row_max     = row_max;
        ctl->row_arg     = row_arg;
        ctl->S0          = S0;
        ctl->above_cut   = 0ull;
        ctl->above_pick  = 0ull;
        ctl->n_above     = 0;
        ctl->rem2        = pieces;
        __threadfence();
        atomicExch(&ctl->rem1, pieces - own); /* the first are the block's own */
    }
    __syncthreads();
    if (threadIdx.x == 32) {
        __threadfence();
        atomicAdd(&p.wide_head->rows, (1ull << 32) + 1ull);
    }
    wide_join(p, gs, ws, slot, 0, own, save_mem);
    __syncthreads();
}

/* A thread block that has no rows of its own left helps with wide ones, as long as there can be any: it waits for rows
 * that have not been decided on, but no longer than kWideHelpNs. How many rows have been opened, 0 where those are no more
 * than `looked` and there is nothing to wait for. One thread. */
constexpr unsigned long long kWideHelpNs = 50000ull, kWideDecideNs = 4000ull; /* rows that go the same way are decided on within 3 us */
__device__ __forceinline__ int wide_wait(const SampleParams &p, unsigned looked) {
    const unsigned long long t0 = global_ns();
    unsigned long long       seen = 0ull; /* when a row was first there to help with */
    for (;;) {
        const unsigned long long rows = *reinterpret_cast<volatile unsigned long long *>(&p.wide_head->rows), now = global_ns();
        const bool               decided = (int) (unsigned) rows >= p.n_rows;
        if ((unsigned) (rows >> 32) > looked) {
            /* who looks for the first time waits a little for the others, so that all of them can be shared out */
            seen = seen == 0ull ? now : seen;
            if (decided || looked > 0u || now - seen > kWideDecideNs) {
                return (int) (rows >> 32);
            }
        } else if (decided || now - t0 > kWideHelpNs) {
            return 0;
        }
        __nanosleep(40);
    }
}
/* `opened`: what the first thread's wait has said. */
__device__ __noinline__ void wide_help(const SampleParams &p, GroupShared *gs, WideShared *ws, int opened, void *save_mem) {
    const Grp          g      = whole_block();
    const int          pieces = (p.V + kWidePiece - 1) / kWidePiece;
    unsigned           looked = 0u; /* rows that had been opened when the slots were last looked through in vain */
    for (;;) {
        if (g.tid == 0) {
            ws->next = opened > 0 ? opened : wide_wait(p, looked);
            __threadfence();
        }
        g.sync();
        const int rows_seen = ws->next;
        opened              = 0;
        if (rows_seen == 0) {
            return;
        }
        /* Of the rows that have more than half as much left to do as the one with the most, the blocks take up one each in turn, in
         * the order in which they come: a block stays for both passes. Each going to the nearest row left some with two blocks next
         * to others with nine (256 flat rows, 98 of them wide, 163 us; 152 so). */
        constexpr int kLook = 2 * kThreads; /* slots that are looked at: more than a device holds thread blocks */
        int           rem[2], most = 0;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = g.tid + h * kThreads;
            rem[h]      = i < p.pool_slots ? ld_volatile(&p.wide_ctl[i].rem1) : 0;
            most        = max(most, rem[h]);
        }
        most = __reduce_max_sync(0xffffffffu, most);
        if (g.lane == 0) {
            ws->wsum[g.warp] = (unsigned) most;
        }
        g.sync();
        for (int w = 0; w < kWarps; w++) {
            most = max(most, (int) ws->wsum[w]);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const unsigned open = __ballot_sync(0xffffffffu, rem[h] > max(kWarps / 2, most / 2));
            if (g.lane == 0) {
                ws->open[h * kWarps + g.warp] = open;
            }
        }
        g.sync();
        if (g.tid == 0) {
            int rows = 0, found = -1;
            for (int w = 0; w < kLook / 32; w++) {
                rows += __popc(ws->open[w]);
            }
            int k = rows > 0 ? (int) ((unsigned) atomicAdd(&p.wide_head->turn, 1) % (unsigned) rows) : -1;
            for (int w = 0; w < kLook / 32 && k >= 0; w++) {
                const int c = __popc(ws->open[w]);
                if (k < c) {
                    unsigned bits = ws->open[w];
                    for (int i = 0; i < k; i++) {
                        bits &= bits - 1u;
                    }
                    found = 32 * w + __ffs(bits) - 1;
                }
                k -= c;
            }
            ws->slot = found;
        }
        g.sync();
        const int slot = ws->slot;
        if (g.tid == 0) {
            /* a piece for every warp: with one for the block a row that is opened first was taken up by all of them */
            const int left = slot < 0 ? 0 : atomicSub(&p.wide_ctl[slot].rem1, kWarps);
            ws->next       = left > 0 ? pieces - left : -1;
            __threadfence();
        }
        g.sync();
        const int piece = ws->next;
        g.sync();
        if (piece >= 0) {
            wide_join(p, gs, ws, slot, piece, min(kWarps, pieces - piece), save_mem);
            g.sync();
        } else if (slot < 0) {
            looked = (unsigned) rows_seen;
        }
    }
}

} /* namespace gb */
