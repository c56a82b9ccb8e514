#include "plan.h"

#include "fft_device.cuh"

#include <algorithm>
#include <cmath>

namespace csipm {

namespace {

// n register radices of product r, descending and none above cap: the first
// as small as possible, then the second, ...
bool split_regs(int r, int n, int cap, int* out) {
    if (n == 0) return r == 1;
    for (int f = 2; f <= cap && f <= r; ++f) {
        if (!reg_radix(f) || r % f || !split_regs(r / f, n - 1, f, out + 1)) continue;
        out[0] = f;
        return true;
    }
    return false;
}

}  // namespace

bool make_fft_plan(int L, FftPlanDev* out, std::string* err) {
    FftPlanDev p{};
    p.L = L;
    if (L < 1) {
        if (err) *err = "FFT length must be positive";
        return false;
    }
    std::vector<int> primes;
    int r = L;
    for (int f = 2; r > 1; ++f) {
        if ((long long)f * f > r) f = r;   // what is left is prime
        for (; r % f == 0; r /= f)
            if (f > 7) primes.push_back(f);
    }
    int regs = L;
    for (int q : primes) regs /= q;
    int rad[FFT_MAX_STAGES];
    int n = 0;
    if (regs > 1) {
        for (n = 1; n <= FFT_MAX_STAGES && !split_regs(regs, n, 10, rad);) ++n;
    }
    if (n + (int)primes.size() > FFT_MAX_STAGES) {
        if (err) *err = "FFT length has too many prime factors";
        return false;
    }
    for (int s = 0; s < n; ++s) p.rad[p.nst++] = rad[s];
    for (int q : primes) p.rad[p.nst++] = q;
    if (p.nst == 0) p.rad[p.nst++] = 1;
    *out = p;
    return true;
}

void fill_stages(const FftPlanDev& pl, int Ltab, bool rev, FftStage* out) {
    int cs[FFT_MAX_STAGES], at = 0;
    for (int s = 0; s < pl.nst; ++s) {
        cs[s] = at;
        if (!reg_radix(pl.rad[s])) at += prime_table(pl.rad[s]);
    }
    int Ns = 1;
    for (int s = 0; s < pl.nst; ++s) {
        const int q = rev ? pl.nst - 1 - s : s;
        FftStage& o = out[s];
        o.R = (unsigned short)pl.rad[q];
        o.Ns = (unsigned short)Ns;
        o.m = (unsigned short)(pl.L / o.R);
        o.step = Ltab / (Ns * o.R);
        o.mag_ns = 0xffffffffu / (unsigned)Ns + 1u;
        o.mag_m = 0xffffffffu / (unsigned)o.m + 1u;
        o.cs = (unsigned short)cs[q];
        Ns *= o.R;
    }
}

int prime_table_size(const FftPlanDev& pl) {
    int n = 0;
    for (int s = 0; s < pl.nst; ++s)
        if (!reg_radix(pl.rad[s])) n += prime_table(pl.rad[s]);
    return n;
}

bool make_row_plan(int L, FftPlanDev* out, std::string* err) {
    FftPlanDev p;
    if (!make_fft_plan(L, &p, err)) return false;
    if (p.nst == 1 || !reg_radix(p.rad[0])) {
        if (p.nst >= FFT_MAX_STAGES) {
            if (err) *err = "FFT length has too many prime factors";
            return false;
        }
        for (int s = p.nst; s > 0; --s) p.rad[s] = p.rad[s - 1];
        p.rad[0] = 1;
        ++p.nst;
    }
    *out = p;
    return true;
}

bool make_fft_plan_ip(int L, FftPlanDev* out, std::string* err) {
    FftPlanDev p{};
    p.L = L;
    p.nst = 0;
    if (L < 1) {
        if (err) *err = "FFT length must be positive";
        return false;
    }
    int r = L;
    int twos = 0;
    while (r % 2 == 0) { r /= 2; ++twos; }
    auto push = [&](int radix) -> bool {
        if (p.nst >= FFT_MAX_STAGES) return false;
        p.rad[p.nst++] = radix;
        return true;
    };
    // 2^twos = 8^a * {1, 4*4 (for 2^4 -> 16 when rem 1), 4 (rem 2)} ; a lone 2 only for L=2
    int rem = twos % 3, a = twos / 3;
    if (rem == 1 && a >= 1) { a -= 1; rem = 4; }   // 8*2 -> 4*4
    for (int i = 0; i < a; ++i) if (!push(8)) goto too_many;
    if (rem == 1) { if (!push(2)) goto too_many; }
    else if (rem == 2) { if (!push(4)) goto too_many; }
    else if (rem == 4) { if (!push(4) || !push(4)) goto too_many; }
    for (int f : {5, 3, 7}) {
        while (r % f == 0) { if (!push(f)) goto too_many; r /= f; }
    }
    for (int f = 11; r > 1; f += 2) {
        while (r % f == 0) { if (!push(f)) goto too_many; r /= f; }
        if ((long long)f * f > r && r > 1) { if (!push(r)) goto too_many; r = 1; }
    }
    *out = p;
    return true;
too_many:
    if (err) *err = "FFT length has too many prime factors";
    return false;
}

bool plan_fits(const FftPlanDev& pl, int lines, int nthreads) {
    const long long total = (long long)lines * pl.L;
    for (int s = 0; s < pl.nst; ++s) {
        const int R = pl.rad[s];
        long long items;
        long long cap;
        switch (R) {
            case 2: cap = MaxItems<2>::v; break;
            case 3: cap = MaxItems<3>::v; break;
            case 4: cap = MaxItems<4>::v; break;
            case 5: cap = MaxItems<5>::v; break;
            case 7: cap = MaxItems<7>::v; break;
            case 8: cap = MaxItems<8>::v; break;
            default: cap = GENERIC_MAX_ITEMS; break;
        }
        if (R == 2 || R == 3 || R == 4 || R == 5 || R == 7 || R == 8)
            items = (total / R + nthreads - 1) / nthreads;
        else
            items = (total + nthreads - 1) / nthreads;
        if (items > cap) return false;
    }
    return true;
}

}  // namespace csipm
