// The checks of xmarch_check.cu at the splits of 256, 288, 432, 512 and 576 points, and the FP64 layout, in
// which the forward exchange takes the place of the inverse one, at every split.  Host code.
#include <algorithm>

#define main xmarch_check_main
#include "xmarch_check.cu"
#undef main

// FP64: both exchanges lie in front of the history and the table, which end the allocation
static void check_shared_exchange(int N1, int N2) {
    const int RW = 2, NT = xmarch_threads(N1, N2, RW);
    const long long ex = xmarch_exchange(N1, N2, RW, false), L1 = xmarch_l1(N1, N2), L2 = xmarch_l2(N1, N2);
    REQUIRE(NT % 32 == 0 && NT <= 256, "NT %d", NT);
    REQUIRE(xmarch_smem_elems(N1, N2, RW, false) == ex + (long long)N2 * NT + (long long)N1 * (N2 + 1), "size");
    long long in = -1, out = -1;  // the largest cells either exchange touches
    for (int t = 0; t < NT; ++t) {
        const XMRoles r = xmarch_roles(t, RW, N1, N2);
        for (int q = 0; q < N1; ++q) {
            if (r.act1) in = std::max(in, r.b1 * L1 + q * (N2 + 1) + r.n2);
            out = std::max(out, r.bfc * L2 + r.kb * (N1 + 1) + q);
        }
        for (int q = 0; q < N2; ++q) {
            in = std::max(in, r.b2 * L1 + r.k1 * (N2 + 1) + q);
            if (r.act2)
                for (int line = 0; line < 2; ++line) out = std::max(out, (6 * r.p2 + 2 * r.role + line) * L2 + q * (N1 + 1) + r.k1);
        }
    }
    REQUIRE(in < ex && out < ex, "exchange cells %lld, %lld of %lld", in, out, ex);
    std::printf("shared %dx%d: %lld elements\n", N1, N2, xmarch_smem_elems(N1, N2, RW, false));
}

int main() {
    const int splits[5][2] = {{16, 16}, {18, 16}, {27, 16}, {32, 16}, {36, 16}};
    for (auto& s : splits)
        for (int rw : {2, 4}) check_roles(s[0], s[1], rw);
    for (auto& s : splits) check_shared_exchange(s[0], s[1]);
    check_shared_exchange(24, 16);
    std::printf("OK\n");
    return 0;
}
