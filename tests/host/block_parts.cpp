// block_parts_complete (phg_mgplan.cpp) on the assembled block systems, forward
// and backward, and on systems with one entry that the composed block solver
// would drop or get wrong.  Prints one line per failure; exits 0 without any.
#include <algorithm>
#include <cstdio>

#include "phg_host.hpp"

using namespace phg;

static Csr with_entry(const Csr &a, int row, int col, double val) {   // added, or replaced where it is
    Csr b = a;
    const int *s = a.col.data() + a.ptr[row], *e = a.col.data() + a.ptr[row + 1];
    const int at = (int)(std::lower_bound(s, e, col) - a.col.data());
    if (at < a.ptr[row + 1] && a.col[at] == col) { b.val[at] = val; return b; }
    b.col.insert(b.col.begin() + at, col);
    b.val.insert(b.val.begin() + at, val);
    for (int r = row + 1; r <= b.n; ++r) ++b.ptr[r];
    return b;
}

int main() {
    int bad = 0;
    auto expect = [&](bool got, bool want, const char *what) {
        if (got != want) { printf("%s: %d\n", what, (int)got); ++bad; }
    };
    for (int level : {2, 3}) {
        Mesh m;
        std::string err;
        if (!generate_sphere(level, m, err)) return 2;
        SphereOps ops;
        assemble_sphere(m, ops);
        const Csr &M = ops.idt, &L = ops.lapl;
        const int n = M.n, i = n / 2, far = i > n / 4 ? 0 : n - 1;   // a column that row i has no entry in
        BaroclinParams c;
        c.tau = 1e-3; c.sigma = 0.05; c.mu = 6.77e-5; c.sigma1 = 0.05; c.mu1 = 6.77e-5; c.alpha = 0.3; c.theta = 0.5;
        for (bool backward : {false, true}) {
            c.backward = backward;
            Csr A, bcol[4];
            assemble_baroclin(m, c, A, bcol);
            expect(block_parts_complete(A, M, L), true, "assembled");
            expect(block_parts_complete(with_entry(A, i, far, 0.5), M, L), false, "w1 row off M's pattern");
            expect(block_parts_complete(with_entry(A, i, 2 * n + i, 0.5), M, L), false, "w1 row, u1 column");
            expect(block_parts_complete(with_entry(A, n + i, 2 * n + i, 0.5), M, L), false, "w2 row, u1 column");
            expect(block_parts_complete(with_entry(A, n + i, 3 * n + far, 0.5), M, L), false, "w2 row, u2 off pattern");
            expect(block_parts_complete(with_entry(A, 2 * n + i, n + i, 0.5), M, L), false, "u1 row, w2 column");
            expect(block_parts_complete(with_entry(A, 2 * n + i, i, 0.5), M, L), false, "u1 row, another coupling");
            expect(block_parts_complete(with_entry(A, 3 * n + i, 3 * n + i, 0.5), M, L), false, "u2 row, not -L");
            expect(block_parts_complete(with_entry(A, 3 * n + i, 2 * n + i, 0.5), M, L), false, "u2 row, u1 column");
        }
        expect(block_parts_complete(M, M, L), false, "not a block system");
    }
    if (!bad) printf("block parts checked\n");
    return bad != 0;
}
