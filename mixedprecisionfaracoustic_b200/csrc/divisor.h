// divisor.h - division by the grid spacing in two operations (host side).
#pragma once
#include <cmath>
#include <cstdint>
#include <initializer_list>
#include <limits>

namespace bpk {

// Division by a constant h > 0 in two operations: with inv = RN(1 / h) and
// lo = RN(1 / h - inv), a / h = fma(a, inv, RN(a lo)) (Brisebarre, Muller and
// Raina, IEEE Trans. Comput. 53(8), 2004).  Before its last rounding that is
// within 2^(1-2p) |a / h| of the quotient (p bits), so it can only round wrongly
// where a / h is that close to the midpoint m of two neighbours.  With integer
// significands A of a, B of h in [2^(p-1), 2^p) and m odd, that is
// |2^p A - m B| < 2 for A >= B, and |2^(p+1) A - m B| < 4 for A < B: for each
// of these few differences J (some more are tried, for what the bound's
// higher orders add) A is known modulo B, and the dividends so found are tried
// out.  Returns whether every one divides right.
template <class R>
bool const_divisor(R h, R inv, R* lo) {
    using u128 = unsigned __int128;
    constexpr int p = std::numeric_limits<R>::digits;
    const R r = std::fma(-h, inv, (R)1);            // exact
    *lo = r / h;
    int e = 0;
    const R f = std::frexp(h, &e);
    if (!(h > 0) || e < -20 || e > 20) return false;
    const uint64_t B = (uint64_t)std::ldexp(f, p);
    int s = 0;
    while (!((B >> s) & 1)) s++;
    // No J below is a multiple of 8.  That covers powers of two and every double
    // widened from a float (s >= 29), for which the search would otherwise take
    // steps of Bo <= 2^24 through 2^52 dividends.
    if (s > 2) return true;
    const uint64_t Bo = B >> s;
    const auto mul = [&](uint64_t x, uint64_t y) { return (uint64_t)((u128)x * y % Bo); };
    const auto wrong = [&](uint64_t A) {
        volatile R a = (R)A, t = a * *lo, q = std::fma((R)a, inv, (R)t), d = a / h;
        return q != d;
    };
    for (int E = p; E <= p + 1; E++) {
        uint64_t half = 1;                           // 2^-(E - s) modulo Bo
        for (int i = 0; i < E - s; i++) half = mul(half, (Bo + 1) / 2);
        for (int J = 1; J <= (E == p ? 3 : 6); J++) {
            if (J & ((1 << s) - 1)) continue;
            const uint64_t A0 = mul((uint64_t)(J >> s) % Bo, half);
            for (uint64_t a : {A0, Bo - A0})         // J and -J
                for (uint64_t A = a; A < (1ull << p); A += Bo)
                    if (A >= (1ull << (p - 1)) && wrong(A)) return false;
        }
    }
    return true;
}

}  // namespace bpk
