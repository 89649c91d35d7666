// ladder.cuh -- the ladder reader of the input-plane gather, one warp per
// ladder on row bitboards.
//
// Reference semantics: FastBoard::saving_size (FastBoard.cpp:1273-1292),
// kill_or_connect / self_atari (:1342-1470), is_suicide (:191-240),
// minimum_elib_count (:2429-2442), after_liberties_color (:2511-2528),
// check_winning_ladder (:2530-2564), check_losing_ladder (:2647-2837).  The
// reference keeps incremental string records (parents, liberty counts, stone
// rings); here a board is two colour masks held by a warp, lane y holding
// row y (bit x = point y*19+x; lanes 19..31 hold zeros), and every string,
// liberty count and capture comes from shifts, shuffles and warp votes.  The
// reference's liberty counts are exact, and the two places where it depends
// on the order of a string's liberties (which liberty the attacker tries
// first; the two branches of an even choice) give the same answer in either
// order, so this restatement agrees point for point; the oracle checks it
// against the reference's planes.
//
// Every function here is called by all 32 lanes of a warp with the same
// (warp-uniform) arguments and returns the same value on every lane.
//
// What bounds it is one warp's latency: a step of a ladder looks at the
// strings around two liberties and an escape, each found by a flood of
// dependent shuffles.  They are flooded side by side, each once (the hunted
// string is carried along), and every question -- captures, suicide, self-
// atari, liberties after a move -- is answered from those masks: 1,000 boards,
// both plane sets, 301 us against 595 with a flood per question and neighbour;
// 8,192 boards 1.79 against 6.5 ms.  Tried and slower: a kernel of one-warp
// CTAs for the candidates (330 us), lines shared between the CTA's warps at
// even choices (347), floods started from the gathered board's strings (357).
//
// check_losing_ladder recurses on even choices (both ataris tried, result
// OR-ed, at most 5 levels of branching); here that is a depth-first search
// with an explicit stack of at most 6 pending lines, stopping at the first
// losing line.
#pragma once
#include "lg_common.cuh"

namespace lg {
namespace lad {

constexpr unsigned kAll = 0xffffffffu;
constexpr uint32_t kRowBits = (1u << kBoard) - 1;

// this lane's row of black (c[0]) and white (c[1]) stones
struct Board {
    uint32_t c[2];
};

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ uint32_t row_mask() { return lane_id() < kBoard ? kRowBits : 0u; }
__device__ __forceinline__ uint32_t point_mask(int p) {
    return lane_id() == p / kBoard ? 1u << (p % kBoard) : 0u;
}
__device__ __forceinline__ uint32_t row_of(uint32_t m, int y) { return __shfl_sync(kAll, m, y); }
__device__ __forceinline__ bool test(uint32_t m, int p) {
    return (row_of(m, p / kBoard) >> (p % kBoard)) & 1u;
}
__device__ __forceinline__ bool any(uint32_t m) { return __any_sync(kAll, m != 0u); }
__device__ __forceinline__ int popc(uint32_t m) {
    return (int)__reduce_add_sync(kAll, (unsigned)__popc(m));
}
// lowest set point of m, or -1
__device__ __forceinline__ int first_point(uint32_t m) {
    const unsigned rows = __ballot_sync(kAll, m != 0u);
    if (!rows) return -1;
    const int y = __ffs(rows) - 1;
    return y * kBoard + __ffs(row_of(m, y)) - 1;
}

__device__ __forceinline__ uint32_t stones(const Board &b, int c) { return c ? b.c[1] : b.c[0]; }
__device__ __forceinline__ void set_stones(Board &b, int c, uint32_t v) {
    if (c) b.c[1] = v;
    else b.c[0] = v;
}
__device__ __forceinline__ uint32_t empties(const Board &b) { return row_mask() & ~(b.c[0] | b.c[1]); }

// the 4-neighbourhood of m (not m itself), on the board
__device__ __forceinline__ uint32_t dilate(uint32_t m) {
    uint32_t up = __shfl_up_sync(kAll, m, 1);
    const uint32_t dn = __shfl_down_sync(kAll, m, 1);
    if (lane_id() == 0) up = 0;
    return ((m << 1) | (m >> 1) | up | dn) & row_mask();
}

// seeds x (inside row r) grown along r towards higher bits: the carry of
// r + x runs from each seed through the set bits above it
__device__ __forceinline__ uint32_t run_up(uint32_t x, uint32_t r) { return (x | ((r + x) ^ r ^ x)) & r; }
// the runs of r that hold a seed of x
__device__ __forceinline__ uint32_t runs_of(uint32_t x, uint32_t r) {
    return run_up(x, r) | __brev(run_up(__brev(x), __brev(r)));
}

// N strings at once: each s[k], seeded inside colour-mask st[k], grown to the
// strings it touches.  Whole runs of a row at a time, then a step to the rows
// above and below; the floods share a step's latency (75 cycles of dependent
// shuffles, and a vote).
template <int N>
__device__ __forceinline__ void flood(uint32_t (&s)[N], const uint32_t (&st)[N]) {
    for (int it = 0; it < 400; ++it) {
        uint32_t changed = 0;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t t = runs_of(s[k], st[k]);
            uint32_t up = __shfl_up_sync(kAll, t, 1);
            const uint32_t dn = __shfl_down_sync(kAll, t, 1);
            if (lane_id() == 0) up = 0;
            s[k] = t | ((up | dn) & st[k]);
            changed |= s[k] ^ t;
        }
        if (!any(changed)) break;
    }
}

// The four neighbours of a point: colour (0, 1, 2 empty, 3 off the board),
// the strings through its stones (0 elsewhere) and their liberties.
struct Around {
    int v;
    int c[4];
    uint32_t s[4], l[4];
};

__device__ __forceinline__ void neighbour_colours(const Board &b, int v, int (&c)[4]) {
    const int y = v / kBoard, x = v - y * kBoard;
    const int yu = y > 0 ? y - 1 : y, yd = y < kBoard - 1 ? y + 1 : y;
    const uint32_t b0 = row_of(b.c[0], y), w0 = row_of(b.c[1], y);
    const uint32_t bu = row_of(b.c[0], yu), wu = row_of(b.c[1], yu);
    const uint32_t bd = row_of(b.c[0], yd), wd = row_of(b.c[1], yd);
    auto at = [](uint32_t bl, uint32_t wh, int i) { return (bl >> i & 1u) ? 0 : ((wh >> i & 1u) ? 1 : 2); };
    c[0] = x > 0 ? at(b0, w0, x - 1) : 3;
    c[1] = x < kBoard - 1 ? at(b0, w0, x + 1) : 3;
    c[2] = y > 0 ? at(bu, wu, x) : 3;
    c[3] = y < kBoard - 1 ? at(bd, wd, x) : 3;
}

__device__ __forceinline__ uint32_t neighbour_mask(int v, int k) {
    return point_mask(k == 0 ? v - 1 : (k == 1 ? v + 1 : (k == 2 ? v - kBoard : v + kBoard)));
}

// Around of N points at once.  known: a whole string of the board (or 0),
// taken as it is where a neighbour belongs to it.
template <int N>
__device__ __forceinline__ void look(const Board &b, const int (&v)[N], uint32_t known, Around (&a)[N]) {
    uint32_t s[4 * N], st[4 * N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        a[i].v = v[i];
        neighbour_colours(b, v[i], a[i].c);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int c = a[i].c[k], j = 4 * i + k;
            st[j] = c < 2 ? stones(b, c) : 0u;
            s[j] = c < 2 ? neighbour_mask(v[i], k) : 0u;
            if (any(s[j] & known)) s[j] = known;
        }
    }
    flood(s, st);
    const uint32_t e = empties(b);
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            a[i].s[k] = s[4 * i + k];
            a[i].l[k] = dilate(s[4 * i + k]) & e;
        }
}

__device__ __forceinline__ int empty_neighbours(const Around &a) {
    return (a.c[0] == 2) + (a.c[1] == 2) + (a.c[2] == 2) + (a.c[3] == 2);
}

// FastBoard::update_board_fast at a.v (a: taken on b): place, capture opponent
// strings without liberties, remove the new string if it has none.  The new
// string in own_out (0 if it was removed), its liberties in libs_out.
__device__ __forceinline__ void play(Board &b, int color, const Around &a, uint32_t &own_out, uint32_t &libs_out) {
    const uint32_t pt = point_mask(a.v);
    uint32_t own = pt, dead = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (a.c[k] == color) own |= a.s[k];
        if (a.c[k] == 1 - color && !any(a.l[k] & ~pt)) dead |= a.s[k];
    }
    set_stones(b, 1 - color, stones(b, 1 - color) & ~dead);
    set_stones(b, color, stones(b, color) | pt);
    uint32_t l = dilate(own) & empties(b);
    if (!any(l)) {
        set_stones(b, color, stones(b, color) & ~own);
        own = 0;
    }
    own_out = own;
    libs_out = l;
}

// FastBoard::after_liberties_color: liberties of the string formed by playing
// a.v, 0 for a suicide
__device__ __forceinline__ int after_libs(const Board &b, int color, const Around &a) {
    Board t = b;
    uint32_t own, l;
    play(t, color, a, own, l);
    return popc(l);
}

// FastBoard::minimum_elib_count: fewest liberties among the opponent strings
// next to the point itself (100 if none)
__device__ __forceinline__ int min_elib(const Around &a, int color) {
    int best = 100;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (a.c[k] == 1 - color) best = min(best, popc(a.l[k]));
    return best;
}

// FastBoard::self_atari (fewer than two empty neighbours, no capture, no
// connection to 3+ liberties, and v + empty neighbours + liberties of the own
// neighbour strings with 2+ liberties number at most two); with suicide,
// FastBoard::is_suicide (no empty neighbour, no own string next to it with
// another liberty, no opponent string in atari) counts too
__device__ __forceinline__ bool self_atari(const Around &a, int color, bool suicide) {
    const int ne = empty_neighbours(a);
    if (ne >= 2) return false;
    uint32_t set = point_mask(a.v);
    bool safe = false, escapes = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (a.c[k] == 2) set |= neighbour_mask(a.v, k);
        if (a.c[k] >= 2) continue;
        const int n = popc(a.l[k]);
        const bool own = a.c[k] == color;
        safe = safe || (own ? n >= 3 : n <= 1);
        escapes = escapes || (own ? n > 1 : n <= 1);
        if (own && n > 1) set |= a.l[k];
    }
    if (suicide && ne == 0 && !escapes) return true;
    return !safe && popc(set) <= 2;
}

// the own strings in atari next to a.v: exactly one, which cannot capture
// an attacker (check_losing_ladder's opening tests)
__device__ __forceinline__ bool lone_critical_string(const Board &b, int color, const Around &a) {
    const uint32_t opp = stones(b, 1 - color);
    uint32_t crit = 0;
    int ncrit = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (a.c[k] != color || any(crit & a.s[k]) || popc(a.l[k]) > 1) continue;
        ++ncrit;
        crit |= a.s[k];
    }
    if (ncrit != 1) return false;
    // any attacker string next to it in atari?  Three at a time, from three
    // points next to it (of one string, perhaps)
    uint32_t d = dilate(crit) & opp;
    const uint32_t e = empties(b);
    for (int it = 0; it < kPoints; ++it) {
        uint32_t s[3], st[3] = {opp, opp, opp};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int q = first_point(d);
            s[k] = q >= 0 ? point_mask(q) : 0u;
            d &= ~s[k];
        }
        if (!any(s[0])) break;
        flood(s, st);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int n = popc(dilate(s[k]) & e);
            if (n <= 1 && any(s[k])) return false;
            d &= ~s[k];
        }
    }
    return true;
}

struct Alt {
    Board b;
    int vtx, branching;
};

// FastBoard::check_losing_ladder(color, vtx): `color` (to move) saves its
// string in atari next to vtx by playing there; true if the attacker can
// keep it in atari until it dies.  Depth-first over the even choices.  The
// hunted string is carried from move to move, so a step floods only the
// other strings next to its two liberties and to the escape.
__device__ bool losing_ladder(const Board &start, int color, int vtx0) {
    Alt stack[6];
    int top = 0;
    stack[top].b = start;
    stack[top].vtx = vtx0;
    stack[top].branching = 0;
    ++top;
    while (top > 0) {
        --top;
        Board b = stack[top].b;
        const int vtx = stack[top].vtx, branching = stack[top].branching;
        if (branching > 5) continue;
        Around at[1];
        {
            const int v[1] = {vtx};
            look<1>(b, v, 0u, at);
        }
        const int elib = min_elib(at[0], color);
        if (elib == 0 || elib == 1 || !lone_critical_string(b, color, at[0])) continue;
        uint32_t own, l;
        play(b, color, at[0], own, l);
        for (int step = 0; step < 400; ++step) {
            const int nl = popc(l);
            if (nl <= 1) return true;  // the escape was a suicide, or a self-atari
            if (nl >= 3) break;        // escaped
            {
                // fewest liberties of the attacker's strings next to the escape
                // point, as they are after it
                const uint32_t e = empties(b), opp = stones(b, 1 - color);
                int best = 100;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t s = at[0].c[k] == 1 - color ? at[0].s[k] & opp : 0u;
                    const int n = popc(dilate(s) & e);
                    if (any(s)) best = min(best, n);
                }
                if (best == 1) break;  // counter-atari
            }
            const int lib0 = first_point(l);
            const int lib1 = first_point(l & ~point_mask(lib0));
            Around a[2];
            {
                const int v[2] = {lib0, lib1};
                look<2>(b, v, own, a);
            }
            if (empty_neighbours(a[0]) == 3 && empty_neighbours(a[1]) == 3) break;
            const bool s0 = self_atari(a[0], 1 - color, true), s1 = self_atari(a[1], 1 - color, true);
            if (s0 && s1) break;
            int first = s0 ? 1 : 0;  // the liberty that the attacker takes
            if (!s0 && !s1) {
                const int l0 = after_libs(b, color, a[0]), l1 = after_libs(b, color, a[1]);
                if (l0 == l1) {
                    // both ataris, each followed by the escape at the other
                    // liberty; lines at branching depth 6 fail at once, so a
                    // depth-5 branch is a failed line (and the stack holds at
                    // most one pending line per depth)
                    if (branching + 1 > 5) break;
                    uint32_t o, f;
                    stack[top].b = b;
                    play(stack[top].b, 1 - color, a[1], o, f);
                    stack[top].vtx = lib0;
                    stack[top].branching = branching + 1;
                    ++top;
                    stack[top].b = b;
                    play(stack[top].b, 1 - color, a[0], o, f);
                    stack[top].vtx = lib1;
                    stack[top].branching = branching + 1;
                    ++top;
                    break;
                }
                first = l0 > l1 ? 0 : 1;
            }
            uint32_t o, f;
            if (first)
                play(b, 1 - color, a[1], o, f);
            else
                play(b, 1 - color, a[0], o, f);
            // the string is back in atari: its one liberty is the next saving move
            l = dilate(own) & empties(b);
            if (popc(l) != 1) break;
            {
                const int v[1] = {first_point(l)};
                look<1>(b, v, own, at);
            }
            play(b, color, at[0], own, l);
        }
    }
    return false;
}

// FastBoard::check_winning_ladder(color, vtx)
__device__ bool winning_ladder(const Board &b, int color, int vtx) {
    Around at[1];
    {
        const int v[1] = {vtx};
        look<1>(b, v, 0u, at);
    }
    if (self_atari(at[0], color, false)) return false;
    Board t = b;
    uint32_t o, f;
    play(t, color, at[0], o, f);
    uint32_t done = 0;
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
        const int c = k == 0 ? at[0].c[0] : (k == 1 ? at[0].c[1] : (k == 2 ? at[0].c[2] : at[0].c[3]));
        const uint32_t s = k == 0 ? at[0].s[0] : (k == 1 ? at[0].s[1] : (k == 2 ? at[0].s[2] : at[0].s[3]));
        const uint32_t l = k == 0 ? at[0].l[0] : (k == 1 ? at[0].l[1] : (k == 2 ? at[0].l[2] : at[0].l[3]));
        if (c != 1 - color || any(s & done) || popc(l) != 2) continue;
        done |= s;
        const int esc = first_point(dilate(s) & empties(t));
        if (esc < 0) continue;
        int ec[4];
        neighbour_colours(t, esc, ec);
        if ((ec[0] == 2) + (ec[1] == 2) + (ec[2] == 2) + (ec[3] == 2) != 2) continue;
        if (losing_ladder(t, 1 - color, esc)) return true;
    }
    return false;
}

}  // namespace lad
}  // namespace lg
