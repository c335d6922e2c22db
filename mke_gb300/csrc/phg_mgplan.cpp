// phg_mgplan.cpp -- the multigrid V-cycle as products of composed operators.
//
// One damped-Jacobi sweep from zero, the coarse correction and one sweep after
// it are, on level l with A = A_l, S = omega D^-1, P and R = P^T,
//     r = b - A S b,  b_c = R r,  x = S b + P x_c,  x <- x + S (b - A x),
// which is the linear map
//     b_c = Q b,   x = T b + U x_c,
//     Q = R (I - A S),  T = S (2 I - A S),  U = (I - S A) P.
// Q, T and U are sparse (about 19, 7 and 7 entries a row), so a level costs
// one gather on the way down and one on the way up instead of five dependent
// phases; the small levels collapse into dense matrices B_k = T_k + U_k
// B_{k+1} Q_k.  For the finest level A U is kept beside U on one pattern, so
// that z = T b + U x_c and A z = A (T b) + (A U) x_c come from one gather.
// Everything is formed in FP64 from the assembled matrices.
#include <algorithm>
#include <cmath>

#include "phg_host.hpp"

namespace phg {

namespace {

// C = A B (sparse), columns ascending
Csr multiply(const Csr &A, const Csr &B) {
    Csr C;
    C.n = A.n;
    C.m = B.m;
    std::vector<std::vector<std::pair<int, double>>> rows(A.n);
#pragma omp parallel
    {
        std::vector<double> acc(B.m, 0.0);
        std::vector<int> at(B.m, -1), list;
#pragma omp for schedule(static)
        for (int i = 0; i < A.n; ++i) {
            list.clear();
            for (int q = A.ptr[i]; q < A.ptr[i + 1]; ++q) {
                const int k = A.col[q];
                const double a = A.val[q];
                for (int e = B.ptr[k]; e < B.ptr[k + 1]; ++e) {
                    const int j = B.col[e];
                    if (at[j] != i) { at[j] = i; acc[j] = 0.0; list.push_back(j); }
                    acc[j] += a * B.val[e];
                }
            }
            std::sort(list.begin(), list.end());
            rows[i].reserve(list.size());
            for (int j : list) rows[i].push_back({j, acc[j]});
        }
    }
    C.ptr.assign(A.n + 1, 0);
    for (int i = 0; i < A.n; ++i) C.ptr[i + 1] = C.ptr[i] + (int)rows[i].size();
    C.col.resize(C.ptr[A.n]);
    C.val.resize(C.ptr[A.n]);
#pragma omp parallel for schedule(static)
    for (int i = 0; i < A.n; ++i) {
        int e = C.ptr[i];
        for (auto &x : rows[i]) { C.col[e] = x.first; C.val[e] = x.second; ++e; }
    }
    return C;
}

// dense row-major C = A B, A sparse
std::vector<double> multiply(const Csr &A, const std::vector<double> &B, int m) {
    std::vector<double> C((size_t)A.n * m, 0.0);
#pragma omp parallel for schedule(static)
    for (int i = 0; i < A.n; ++i)
        for (int q = A.ptr[i]; q < A.ptr[i + 1]; ++q) {
            const double a = A.val[q];
            const double *b = &B[(size_t)A.col[q] * m];
            double *c = &C[(size_t)i * m];
            for (int j = 0; j < m; ++j) c[j] += a * b[j];
        }
    return C;
}

}  // namespace

Csr csr_multiply(const Csr &A, const Csr &B) { return multiply(A, B); }

bool block_parts_complete(const Csr &A, const Csr &M, const Csr &L) {
    const int n = M.n;
    if (A.n != 4 * n || L.n != n) return false;
    auto entry = [](const Csr &B, int i, int j, double *v) {
        const int *b = B.col.data() + B.ptr[i], *e = B.col.data() + B.ptr[i + 1];
        const int *at = std::lower_bound(b, e, j);
        if (at == e || *at != j) return false;
        *v = B.val[at - B.col.data()];
        return true;
    };
    bool complete = true;
#pragma omp parallel for schedule(static) reduction(&& : complete)
    for (int r = 0; r < A.n; ++r) {
        const int br = r / n, i = r % n;
        double scale = 0.0;
        int coupled = 0, own = 0;   // entries of a u row
        for (int q = A.ptr[r]; q < A.ptr[r + 1]; ++q) scale = std::max(scale, std::fabs(A.val[q]));
        for (int q = A.ptr[r]; q < A.ptr[r + 1]; ++q) {
            const int bc = A.col[q] / n, j = A.col[q] % n;
            double v = 0.0;
            bool ok;
            if (br < 2) {          // w rows: the w columns, and u2 in w2's
                ok = (bc < 2 || (br == 1 && bc == 3)) && entry(M, i, j, &v);
            } else if (bc < 2) {   // u rows: M in their layer's w columns, -L in their own
                ok = bc == br - 2 && entry(M, i, j, &v) && std::fabs(A.val[q] - v) <= 1e-13 * scale;
                ++coupled;
            } else {
                ok = bc == br && entry(L, i, j, &v) && std::fabs(A.val[q] + v) <= 1e-13 * scale;
                ++own;
            }
            complete = complete && ok;
        }
        if (br >= 2) complete = complete && coupled == M.ptr[i + 1] - M.ptr[i] && own == L.ptr[i + 1] - L.ptr[i];
    }
    return complete;
}

bool build_mg_plan(const Csr &fine, const MgHierarchy &h, double omega, MgPlan &p) {
    const int nlev = (int)h.A.size();
    p = MgPlan();
    if (nlev < 2) return false;
    p.lev.resize(nlev - 1);
    auto A = [&](int l) -> const Csr & { return l == 0 ? fine : h.A[l]; };
    for (int l = 0; l + 1 < nlev; ++l) {
        const Csr &a = A(l);
        std::vector<double> s(a.n, 0.0);   // omega D^-1
        for (int i = 0; i < a.n; ++i)
            for (int q = a.ptr[i]; q < a.ptr[i + 1]; ++q)
                if (a.col[q] == i) s[i] = omega / a.val[q];
        for (double v : s)
            if (!(v != 0.0) || !std::isfinite(v)) return false;
        Csr AS = a, SA = a;
        for (int i = 0; i < a.n; ++i)
            for (int q = a.ptr[i]; q < a.ptr[i + 1]; ++q) {
                const double id = a.col[q] == i ? 1.0 : 0.0;
                AS.val[q] = id - a.val[q] * s[a.col[q]];   // I - A S
                SA.val[q] = id - s[i] * a.val[q];          // I - S A
            }
        MgPlan::Level &L = p.lev[l];
        L.Q = multiply(h.R[l], AS);
        L.U = multiply(SA, h.P[l]);
        L.T = AS;
        for (int i = 0; i < a.n; ++i)
            for (int q = a.ptr[i]; q < a.ptr[i + 1]; ++q)
                L.T.val[q] = s[i] * ((a.col[q] == i ? 1.0 : 0.0) + AS.val[q]);
    }
    p.AU = multiply(fine, p.lev[0].U);
    // the small levels, dense
    const int last = nlev - 1;
    p.B.resize(nlev);
    p.B[last] = h.coarse_inv;
    p.first_dense = last;
    for (int k = last - 1; k >= 0 && A(k).n <= MG_DENSE_ROWS; --k) {
        const MgPlan::Level &L = p.lev[k];
        const int n = A(k).n, nc = A(k + 1).n;
        // B_{k+1} Q_k, then U_k times it, plus T_k
        std::vector<double> BQ((size_t)nc * n, 0.0);
        for (int i = 0; i < nc; ++i)
            for (int c = 0; c < nc; ++c) {
                const double b = p.B[k + 1][(size_t)i * nc + c];
                for (int q = L.Q.ptr[c]; q < L.Q.ptr[c + 1]; ++q) BQ[(size_t)i * n + L.Q.col[q]] += b * L.Q.val[q];
            }
        p.B[k] = multiply(L.U, BQ, n);
        for (int i = 0; i < n; ++i)
            for (int q = L.T.ptr[i]; q < L.T.ptr[i + 1]; ++q) p.B[k][(size_t)i * n + L.T.col[q]] += L.T.val[q];
        p.first_dense = k;
    }
    const int k = p.first_dense;
    if (k > 0 && A(k - 1).n <= MG_WIDE_ROWS) p.E = multiply(p.lev[k - 1].U, p.B[k], A(k).n);
    if (k == 0) p.AB = multiply(fine, p.B[0], fine.n);
    if (k == 1 && !p.E.empty()) p.AE = multiply(fine, p.E, A(1).n);
    return true;
}

}  // namespace phg
