// IncrementalCholesky.cpp — see include/deformation/IncrementalCholesky.h.
//
// Symbolic step: elimination tree and column counts of L from the upper
// triangle (Liu's tree via path compression-free ancestor walks, as in
// Davis' LDL).  Numeric step (per column k, "up-looking"): the nonzero
// pattern of row k of L is the union of the tree paths from every i with
// A(i, k) != 0, i < k, up to k; solving the triangular system along that
// pattern in topological order yields L(k, :) and D(k).  Constrained
// columns (Herholz et al. 2017, Eq. 14) get L(k, :) = 0 and D(k) = 1.
#include "../../include/deformation/IncrementalCholesky.h"

#include <algorithm>
#include <map>

#if defined(__x86_64__)
#include <immintrin.h>
#endif

namespace pbfdrop {

// The inner loops of the factorization and the solves, four values at a time
// where the processor has AVX2.  Every element takes one multiplication and
// one subtraction, each rounded (no fused operation), whatever the width: the
// same bits as the plain loops.  The factor's columns fill in runs (135 rows a
// column in 1.12 runs for a sphere of 2,562 vertices), so a run is one loop
// over consecutive memory where a walk over li_ gathered and scattered: the
// factorization with 585 handles 21 -> 4.8 ms, three axes' solve 2.9 -> 0.9 ms
// (one core), a frame with 262,144 particles, repeated from the same ones so
// that its handles settle, 11.0 -> 3.4 ms.
namespace {

// w[i] -= l[i] * y
void axpy_plain(double* w, const double* l, int n, double y)
{
    for (int i = 0; i < n; ++i) w[i] -= l[i] * y;
}

// w[4 i + a] -= l[i] * y[a]
void axpy4_plain(double* w, const double* l, int n, const double* y)
{
    for (int i = 0; i < n; ++i)
        for (int a = 0; a < 4; ++a) w[4 * i + a] -= l[i] * y[a];
}

// x[a] -= l[i] * w[4 i + a], i ascending
void dot4_plain(double* x, const double* l, int n, const double* w)
{
    for (int i = 0; i < n; ++i)
        for (int a = 0; a < 4; ++a) x[a] -= l[i] * w[4 * i + a];
}

#if defined(__x86_64__)
__attribute__((target("avx2"))) void axpy_avx2(double* w, const double* l, int n, double y)
{
    const __m256d y4 = _mm256_set1_pd(y);
    int i = 0;
    for (; i + 8 <= n; i += 8) {
        const __m256d a = _mm256_sub_pd(_mm256_loadu_pd(w + i), _mm256_mul_pd(_mm256_loadu_pd(l + i), y4));
        const __m256d b = _mm256_sub_pd(_mm256_loadu_pd(w + i + 4), _mm256_mul_pd(_mm256_loadu_pd(l + i + 4), y4));
        _mm256_storeu_pd(w + i, a);
        _mm256_storeu_pd(w + i + 4, b);
    }
    for (; i < n; ++i) w[i] -= l[i] * y;
}

__attribute__((target("avx2"))) void axpy4_avx2(double* w, const double* l, int n, const double* y)
{
    const __m256d y4 = _mm256_loadu_pd(y);
    for (int i = 0; i < n; ++i)
        _mm256_storeu_pd(w + 4 * i,
                         _mm256_sub_pd(_mm256_loadu_pd(w + 4 * i), _mm256_mul_pd(_mm256_set1_pd(l[i]), y4)));
}

__attribute__((target("avx2"))) void dot4_avx2(double* x, const double* l, int n, const double* w)
{
    __m256d x4 = _mm256_loadu_pd(x);
    for (int i = 0; i < n; ++i)
        x4 = _mm256_sub_pd(x4, _mm256_mul_pd(_mm256_set1_pd(l[i]), _mm256_loadu_pd(w + 4 * i)));
    _mm256_storeu_pd(x, x4);
}

const bool kAvx2 = __builtin_cpu_supports("avx2");
const auto axpy = kAvx2 ? axpy_avx2 : axpy_plain;
const auto axpy4 = kAvx2 ? axpy4_avx2 : axpy4_plain;
const auto dot4 = kAvx2 ? dot4_avx2 : dot4_plain;
#else
const auto axpy = axpy_plain;
const auto axpy4 = axpy4_plain;
const auto dot4 = dot4_plain;
#endif

}  // namespace

double SymCsc::at(int i, int j) const
{
    const auto b = rows.begin() + colptr[j], e = rows.begin() + colptr[j + 1];
    const auto it = std::lower_bound(b, e, i);
    return (it != e && *it == i) ? vals[it - rows.begin()] : 0.0;
}

SymCsc sym_from_triplets(int n, const std::vector<int>& r, const std::vector<int>& c, const std::vector<double>& v)
{
    std::vector<std::map<int, double>> cols(n);
    for (size_t t = 0; t < r.size(); ++t) cols[c[t]][r[t]] += v[t];
    SymCsc A;
    A.n = n;
    A.colptr.assign(n + 1, 0);
    for (int j = 0; j < n; ++j) {
        A.colptr[j + 1] = A.colptr[j] + (int)cols[j].size();
        for (const auto& kv : cols[j]) {
            A.rows.push_back(kv.first);
            A.vals.push_back(kv.second);
        }
    }
    return A;
}

void IncrementalCholesky::analyze(const SymCsc& A)
{
    n_ = A.n;
    ok_ = false;
    parent_.assign(n_, -1);
    std::vector<int> count(n_, 0), mark(n_, -1);
    for (int k = 0; k < n_; ++k) {
        mark[k] = k;
        for (int q = A.colptr[k]; q < A.colptr[k + 1] && A.rows[q] < k; ++q) {
            for (int j = A.rows[q]; mark[j] != k; j = parent_[j]) {
                if (parent_[j] == -1) parent_[j] = k;
                ++count[j];
                mark[j] = k;
            }
        }
    }
    lp_.assign(n_ + 1, 0);
    for (int j = 0; j < n_; ++j) lp_[j + 1] = lp_[j] + count[j];
    li_.assign(lp_[n_], 0);
    lx_.assign(lp_[n_], 0.0);
    d_.assign(n_, 0.0);
    std::vector<int> fill(n_, 0);
    std::fill(mark.begin(), mark.end(), -1);
    for (int k = 0; k < n_; ++k) {  // rows appended in increasing k: ascending per column
        mark[k] = k;
        for (int q = A.colptr[k]; q < A.colptr[k + 1] && A.rows[q] < k; ++q) {
            for (int j = A.rows[q]; mark[j] != k; j = parent_[j]) {
                li_[lp_[j] + fill[j]++] = k;
                mark[j] = k;
            }
        }
    }
    rp_.assign(n_ + 1, 0);
    runs_.clear();
    for (int j = 0; j < n_; ++j) {
        for (int p = lp_[j]; p < lp_[j + 1]; ++p) {
            if (p > lp_[j] && li_[p] == li_[p - 1] + 1)
                ++runs_.back().len;
            else
                runs_.push_back({li_[p], p, 1});
        }
        rp_[j + 1] = (int)runs_.size();
    }
    cursor_.assign(n_, 0);
    cons_.assign(n_, 0);
    work_.assign(n_, 0.0);
    stack_.assign(n_, 0);
    visit_.assign(n_, 0);
    stamp_ = 0;
    ok_ = n_ > 0;
}

void IncrementalCholesky::setConstrained(std::vector<char> constrained)
{
    cons_ = std::move(constrained);
    if ((int)cons_.size() != n_) cons_.assign(n_, 0);
}

void IncrementalCholesky::column(const SymCsc& A, int k)
{
    const int stamp = ++stamp_;
    visit_[k] = stamp;
    int top = n_;
    // scatter A^B(:, k) above the diagonal and collect the row-k pattern
    for (int q = A.colptr[k]; q < A.colptr[k + 1] && A.rows[q] < k; ++q) {
        const int i = A.rows[q];
        work_[i] += cons_[i] ? 0.0 : A.vals[q];
        int len = 0;
        for (int j = i; visit_[j] != stamp; j = parent_[j]) {
            stack_[len++] = j;
            visit_[j] = stamp;
        }
        while (len > 0) stack_[--top] = stack_[--len];
    }
    if (cons_[k]) {  // detached: L(k, :) = 0, D(k) = 1
        d_[k] = 1.0;
        for (int p = top; p < n_; ++p) {
            const int j = stack_[p];
            int r = cursor_[j];
            while (runs_[r].row + runs_[r].len <= k) ++r;
            cursor_[j] = r;
            lx_[runs_[r].at + (k - runs_[r].row)] = 0.0;
            work_[j] = 0.0;
        }
        return;
    }
    double dk = A.at(k, k);
    for (int p = top; p < n_; ++p) {
        const int j = stack_[p];
        const double y = work_[j];
        work_[j] = 0.0;
        // rows of column j above k, then L(k, j)'s place
        int r = cursor_[j];
        while (runs_[r].row + runs_[r].len <= k) ++r;
        cursor_[j] = r;
        if (y != 0.0) {  // (a detached column's is zero)
            for (int q = rp_[j]; q < r; ++q)
                axpy(work_.data() + runs_[q].row, lx_.data() + runs_[q].at, runs_[q].len, y);
            axpy(work_.data() + runs_[r].row, lx_.data() + runs_[r].at, k - runs_[r].row, y);
        }
        const int s = runs_[r].at + (k - runs_[r].row);
        const double l = d_[j] != 0.0 ? y / d_[j] : 0.0;
        dk -= l * y;
        lx_[s] = l;
    }
    d_[k] = dk;
}

void IncrementalCholesky::factorizeFull(const SymCsc& A)
{
    if (!ok_) return;
    std::fill(lx_.begin(), lx_.end(), 0.0);
    std::fill(work_.begin(), work_.end(), 0.0);
    std::copy(rp_.begin(), rp_.end() - 1, cursor_.begin());
    for (int k = 0; k < n_; ++k) column(A, k);
}

void IncrementalCholesky::updateColumns(const SymCsc& A, const std::vector<int>& changed)
{
    if (!ok_ || changed.empty()) return;
    // union of the tree paths from the changed columns to their roots
    const int stamp = ++stamp_;
    std::vector<int> cols;
    for (int c : changed)
        for (int j = c; j != -1 && visit_[j] != stamp; j = parent_[j]) {
            visit_[j] = stamp;
            cols.push_back(j);
        }
    std::sort(cols.begin(), cols.end());
    std::copy(rp_.begin(), rp_.end() - 1, cursor_.begin());
    for (int k : cols) column(A, k);
}

void IncrementalCholesky::solveInPlace(std::vector<double>& b) const
{
    for (int k = 0; k < n_; ++k) {  // L z = b
        const double bk = b[k];
        for (int q = rp_[k]; q < rp_[k + 1]; ++q)
            axpy(b.data() + runs_[q].row, lx_.data() + runs_[q].at, runs_[q].len, bk);
    }
    for (int k = 0; k < n_; ++k) b[k] /= d_[k];  // D y = z
    for (int k = n_ - 1; k >= 0; --k) {          // L^T x = y
        double x = b[k];
        for (int p = lp_[k]; p < lp_[k + 1]; ++p) x -= lx_[p] * b[li_[p]];
        b[k] = x;
    }
}

void IncrementalCholesky::solveInPlace(std::vector<double>& x, std::vector<double>& y, std::vector<double>& z) const
{
    std::vector<double> b(4 * (size_t)n_);
    for (int k = 0; k < n_; ++k) {
        b[4 * (size_t)k] = x[k];
        b[4 * (size_t)k + 1] = y[k];
        b[4 * (size_t)k + 2] = z[k];
    }
    for (int k = 0; k < n_; ++k) {
        double bk[4];
        std::copy_n(b.data() + 4 * (size_t)k, 4, bk);
        for (int q = rp_[k]; q < rp_[k + 1]; ++q)
            axpy4(b.data() + 4 * (size_t)runs_[q].row, lx_.data() + runs_[q].at, runs_[q].len, bk);
    }
    for (int k = 0; k < n_; ++k)
        for (int a = 0; a < 4; ++a) b[4 * (size_t)k + a] /= d_[k];
    for (int k = n_ - 1; k >= 0; --k)
        for (int q = rp_[k]; q < rp_[k + 1]; ++q)
            dot4(b.data() + 4 * (size_t)k, lx_.data() + runs_[q].at, runs_[q].len, b.data() + 4 * (size_t)runs_[q].row);
    for (int k = 0; k < n_; ++k) {
        x[k] = b[4 * (size_t)k];
        y[k] = b[4 * (size_t)k + 1];
        z[k] = b[4 * (size_t)k + 2];
    }
}

}  // namespace pbfdrop
