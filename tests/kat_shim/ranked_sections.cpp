// SectionSet::put() against the marcher's insertion in its lane form (warp_put),
// on random sequences, for tests/test_ranked_sections_cpu.py.  Each "lane" is a
// loop iteration that only reads the old set, its own section and the masks that
// the ballots give, and writes the new set.
#include <cmath>
#include <cstring>
#include <random>

#include "../../differentiable_gaussian_mixture_renderer_b200/csrc/dgmr_sections.h"

namespace {

constexpr unsigned MAX = 16;
template <class T>
using Set = dgmr::SectionSet<MAX, T>;

unsigned below(int n) { return n >= 32 ? 0xffffffffu : (1u << n) - 1u; }
int top(unsigned m) { return 31 - __builtin_clz(m); }

// false: the case that the warp hands to merge_pieces
template <class T>
bool put_ranked(Set<T>& set, dgmr::Section<T> s)
{
    if (s.end <= set.lo || s.start >= set.hi)
        return true;
    s.start = dgmr::max_f(set.lo, s.start);
    s.end = dgmr::min_f(set.hi, s.end);
    const unsigned n = set.n;
    unsigned first = 0;
    while (first < n && !(set.e[first].end > s.start))
        ++first;
    if (first >= n) {
        set.put(s);
        return true;
    }
    unsigned last = first;
    while (last < n && !(set.e[last].end > s.end))
        ++last;
    if (last < n && set.e[last].start < s.end)
        ++last;
    bool odd = !(s.end > s.start) || s.delta_t != s.delta_t;
    for (unsigned i = first; i < last; ++i)
        odd = odd || !(set.e[i].end > set.e[i].start) || set.e[i].delta_t != set.e[i].delta_t;
    if (odd) {
        set.put_by_pieces(s);
        return false;
    }
    const Set<T> old = set;
    unsigned kept = 0;
    for (unsigned i = first; i < last; ++i)
        if (old.e[i].delta_t < s.delta_t)
            kept |= 1u << i;
    const bool run = last > first;
    const unsigned tail = run ? last - 1u : first;
    const dgmr::Section<T> f = old.e[first], l = old.e[tail];
    const bool left = run && !((kept >> first) & 1u) && f.start < s.start, right = run && !((kept >> tail) & 1u) && s.end < l.end;
    const T from = left && f.delta_t == s.delta_t ? f.start : s.start, to = right && l.delta_t == s.delta_t ? l.end : s.end;
    const unsigned n_left = left && f.delta_t != s.delta_t, n_right = right && l.delta_t != s.delta_t;
    const auto gap_start = [&](unsigned i) {
        const unsigned m = kept & below(int(i));
        return m ? old.e[top(m)].end : from;
    };
    unsigned gaps = 0;
    for (unsigned i = first; i < last; ++i)
        if (((kept >> i) & 1u) && old.e[i].start - gap_start(i) > T(0))
            gaps |= 1u << i;
    const T end_start = kept ? old.e[top(kept)].end : from;
    const unsigned n_end = to - end_start > T(0), base = first + n_left;
    const unsigned end_place = base + __builtin_popcount(gaps) + __builtin_popcount(kept), tail_place = end_place + n_end + n_right;
    const auto write = [&](unsigned at, const dgmr::Section<T>& q) {
        if (at < MAX)
            set.e[at] = q;
    };
    for (unsigned i = 0; i < n; ++i) {
        const unsigned place = base + __builtin_popcount(gaps & below(int(i) + 1)) + __builtin_popcount(kept & below(int(i)));
        if ((kept >> i) & 1u)
            write(place, old.e[i]);
        if ((gaps >> i) & 1u)
            write(place - 1u, { gap_start(i), old.e[i].start, s.delta_t });
        if (i >= last)
            write(tail_place + (i - last), old.e[i]);
    }
    if (n_left)
        write(first, { f.start, s.start, f.delta_t });
    if (n_right)
        write(end_place + n_end, { s.end, l.end, l.delta_t });
    if (n_end)
        write(end_place, { end_start, to, s.delta_t });
    set.n = tail_place + (n - last) < MAX ? tail_place + (n - last) : MAX;
    if (set.n == MAX)
        set.hi = dgmr::min_f(set.hi, set.e[MAX - 1].end);
    return true;
}

template <class T>
bool same_bits(T a, T b)
{
    return std::memcmp(&a, &b, sizeof(T)) == 0 || (a != a && b != b);
}

template <class T>
long check(unsigned seed, int trials, bool odd, long* puts, long* pieces)
{
    std::mt19937 rng(seed);
    long bad = 0;
    for (int trial = 0; trial < trials; ++trial) {
        Set<T> a, b;
        a.reset(T(rng() % 3) * T(0.5));
        b = a;
        const int n_put = 5 + int(rng() % 80);
        for (int k = 0; k < n_put; ++k) {
            T c = T(std::uniform_real_distribution<double>(0.0, 10.0)(rng));
            T w = T(0.02 + std::uniform_real_distribution<double>(0.0, 2.0)(rng));
            if (rng() % 2) {
                c = T(int(c * T(4))) / T(4);
                w = T(1 + rng() % 8) / T(4);
            }
            const T dt = (rng() % 3 == 0) ? T(1 + rng() % 4) / T(32) : w / T(31);
            dgmr::Section<T> s { c - w, c + w, dt };
            if (odd && rng() % 16 == 0)
                s.end = T(1) / T(0);
            if (odd && rng() % 16 == 0)
                s.end = s.start;
            if (odd && rng() % 32 == 0)
                s.delta_t = std::nan("");
            a.put(s);
            ++*puts;
            *pieces += !put_ranked(b, s);
            bool same = a.n == b.n && same_bits(a.hi, b.hi) && same_bits(a.lo, b.lo);
            for (unsigned i = 0; same && i < a.n; ++i)
                same = same_bits(a.e[i].start, b.e[i].start) && same_bits(a.e[i].end, b.e[i].end) && same_bits(a.e[i].delta_t, b.e[i].delta_t);
            if (!same) {
                ++bad;
                break;
            }
        }
    }
    return bad;
}

} // namespace

extern "C" long ranked_sections(int is_double, int odd, unsigned seed, int trials, long* puts, long* pieces)
{
    *puts = *pieces = 0;
    return is_double ? check<double>(seed, trials, odd, puts, pieces) : check<float>(seed, trials, odd, puts, pieces);
}
