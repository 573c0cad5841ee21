// Small dense complex linear algebra on the host, in double: the k x k systems of the
// optimizers whose O(n m) and O(n m^2) work runs on the device (apo.cu, matrix.cu).  Matrices
// are row-major std::vector<std::complex<double>>.
#pragma once

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

namespace afc {
namespace dense {

using cd = std::complex<double>;

// Cholesky factorisation in place of the Hermitian positive definite k x k matrix a: its lower
// triangle becomes L with a = L L^H (the diagonal real).  False if a is not positive definite.
inline bool hpd_factor(std::vector<cd>& a, int k) {
    for (int j = 0; j < k; ++j) {
        double d = a[j * k + j].real();
        for (int p = 0; p < j; ++p) d -= std::norm(a[j * k + p]);
        if (!(d > 0.0)) return false;
        d = std::sqrt(d);
        a[j * k + j] = d;
        for (int i = j + 1; i < k; ++i) {
            cd s = a[i * k + j];
            for (int p = 0; p < j; ++p) s -= a[i * k + p] * std::conj(a[j * k + p]);
            a[i * k + j] = s / d;
        }
    }
    return true;
}

// Solve L L^H c = b in place for one right-hand side, L from hpd_factor.
inline void hpd_substitute(const std::vector<cd>& l, std::vector<cd>& b, int k) {
    for (int i = 0; i < k; ++i) {
        cd s = b[i];
        for (int p = 0; p < i; ++p) s -= l[i * k + p] * b[p];
        b[i] = s / l[i * k + i].real();
    }
    for (int i = k - 1; i >= 0; --i) {
        cd s = b[i];
        for (int p = i + 1; p < k; ++p) s -= std::conj(l[p * k + i]) * b[p];
        b[i] = s / l[i * k + i].real();
    }
}

// Solve the Hermitian positive definite system a c = b (k x k, a overwritten by its factor).
inline bool hpd_solve(std::vector<cd>& a, std::vector<cd>& b, int k) {
    if (!hpd_factor(a, k)) return false;
    hpd_substitute(a, b, k);
    return true;
}

// Inverse of the Hermitian positive definite k x k matrix a (overwritten by its factor) into
// inv, column by column.
inline bool hpd_inverse(std::vector<cd>& a, std::vector<cd>& inv, int k) {
    if (!hpd_factor(a, k)) return false;
    inv.assign(static_cast<size_t>(k) * k, cd(0.0, 0.0));
    std::vector<cd> col(k);
    for (int c = 0; c < k; ++c) {
        for (int i = 0; i < k; ++i) col[i] = cd(i == c ? 1.0 : 0.0, 0.0);
        hpd_substitute(a, col, k);
        for (int i = 0; i < k; ++i) inv[i * k + c] = col[i];
    }
    return true;
}

// Cyclic Jacobi eigendecomposition of the Hermitian k x k matrix a (row-major, destroyed; only
// its lower triangle and the real part of its diagonal are read, the upper triangle is taken as
// the conjugate of the lower).  Eigenvalues go to lam, unit eigenvectors to the columns of v.
//
// Pivot (p, q) with a_qp = |b| e^{-i phi} (so a_pq = |b| e^{i phi}) is annihilated by the
// unitary J with J_pp = J_qq = c, J_pq = s e^{i phi}, J_qp = -s e^{-i phi}, where t = s / c is
// the smaller root of t^2 + 2 theta t - 1 = 0, theta = (a_qq - a_pp) / (2 |b|): the real
// symmetric rotation after a diagonal phase change.
//
// The eigenpairs are then put in ascending order of eigenvalue (ties keep their order), and
// each eigenvector's phase is fixed: its first nonzero entry is real and positive.  Eigenvectors
// are defined only up to such a unit factor, and an order is a choice too, so both rules are
// part of what a caller gets.
inline void hermitian_eigen(std::vector<cd>& a, int k, std::vector<double>& lam,
                            std::vector<cd>& v) {
    for (int i = 0; i < k; ++i) {
        a[i * k + i] = cd(a[i * k + i].real(), 0.0);
        for (int j = i + 1; j < k; ++j) a[i * k + j] = std::conj(a[j * k + i]);
    }
    v.assign(static_cast<size_t>(k) * k, cd(0.0, 0.0));
    for (int i = 0; i < k; ++i) v[i * k + i] = 1.0;
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int i = 0; i < k; ++i)
            for (int j = 0; j < k; ++j) {
                const double x = std::norm(a[i * k + j]);
                tot += x;
                if (i != j) off += x;
            }
        if (off == 0.0 || off <= 1e-30 * tot) break;
        for (int p = 0; p < k; ++p)
            for (int q = p + 1; q < k; ++q) {
                const cd apq = a[p * k + q];
                const double b = std::abs(apq);
                if (b == 0.0) continue;
                const cd e = apq / b;  // e^{i phi}
                const double theta = (a[q * k + q].real() - a[p * k + p].real()) / (2.0 * b);
                const double t = (theta >= 0 ? 1.0 : -1.0) /
                                 (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
                const double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
                const cd se = s * e, sec = s * std::conj(e);
                for (int r = 0; r < k; ++r) {  // a J: columns p, q
                    const cd arp = a[r * k + p], arq = a[r * k + q];
                    a[r * k + p] = c * arp - sec * arq;
                    a[r * k + q] = se * arp + c * arq;
                }
                for (int r = 0; r < k; ++r) {  // J^H (a J): rows p, q
                    const cd apr = a[p * k + r], aqr = a[q * k + r];
                    a[p * k + r] = c * apr - se * aqr;
                    a[q * k + r] = sec * apr + c * aqr;
                }
                a[p * k + q] = a[q * k + p] = 0.0;
                a[p * k + p] = cd(a[p * k + p].real(), 0.0);
                a[q * k + q] = cd(a[q * k + q].real(), 0.0);
                for (int r = 0; r < k; ++r) {  // v J
                    const cd vrp = v[r * k + p], vrq = v[r * k + q];
                    v[r * k + p] = c * vrp - sec * vrq;
                    v[r * k + q] = se * vrp + c * vrq;
                }
            }
    }
    std::vector<int> order(k);
    for (int i = 0; i < k; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return a[x * k + x].real() < a[y * k + y].real();
    });
    lam.resize(k);
    std::vector<cd> vs(static_cast<size_t>(k) * k);
    for (int j = 0; j < k; ++j) {
        const int o = order[j];
        lam[j] = a[o * k + o].real();
        for (int r = 0; r < k; ++r) vs[r * k + j] = v[r * k + o];
    }
    v.swap(vs);
    for (int j = 0; j < k; ++j) {  // phase rule: the first nonzero entry real and positive
        int r0 = 0;
        while (r0 < k && v[r0 * k + j] == cd(0.0, 0.0)) ++r0;
        if (r0 == k) continue;
        const double mag = std::abs(v[r0 * k + j]);
        const cd ph = std::conj(v[r0 * k + j]) / mag;
        for (int r = 0; r < k; ++r) v[r * k + j] *= ph;
        v[r0 * k + j] = mag;
    }
}

// The unit eigenvector of the largest eigenvalue of the Hermitian k x k matrix a (row-major; read as by
// hermitian_eigen), for a caller that needs no other: Householder reflections to a tridiagonal
// matrix, made real by a diagonal of phases, implicit QR steps with Wilkinson's shift on that (Golub
// and Van Loan, Matrix Computations, 8.3), and the reflections on the one vector.  O(k^3) once
// instead of each of Jacobi's eight to ten sweeps: k = 31 takes 48 us on a Grace core (Jacobi 792),
// k = 64 0.31 ms (7.7).  Real and imaginary parts lie apart and the inner loops run along rows, without
// the NaN rules of std::complex products, so that they vectorise.
//
// Equal largest eigenvalues give the eigenvector that comes first, and the phase is hermitian_eigen's:
// the first nonzero entry real and positive, where an entry below 1e-14 counts as zero.
inline void principal_eigenvector(const std::vector<cd>& a, int k, std::vector<cd>& out) {
    const size_t kk = static_cast<size_t>(k) * k;
    std::vector<double> re(kk), im(kk), vr(kk), vi(kk), beta(k, 0.0), wr(k), wi(k), d(k), e(k, 0.0);
    std::vector<cd> sub(k, cd(0.0, 0.0));  // sub-diagonal
    for (int i = 0; i < k; ++i)
        for (int j = 0; j <= i; ++j) {
            const cd x = a[static_cast<size_t>(i) * k + j];
            re[i * k + j] = re[j * k + i] = x.real();
            im[i * k + j] = i == j ? 0.0 : x.imag();
            im[j * k + i] = i == j ? 0.0 : -x.imag();
        }
    // column p below the sub-diagonal to zero: I - beta v v^H on rows and columns p + 1 ..
    for (int p = 0; p + 1 < k; ++p) {
        const int f = p + 1;
        double tail = 0.0;
        for (int i = f + 1; i < k; ++i)
            tail += re[i * k + p] * re[i * k + p] + im[i * k + p] * im[i * k + p];
        const cd x0(re[f * k + p], im[f * k + p]);
        sub[p] = x0;
        if (tail == 0.0) continue;
        const double n0 = std::abs(x0), norm = std::sqrt(n0 * n0 + tail);
        const cd ph = n0 > 0.0 ? x0 / n0 : cd(1.0, 0.0);
        sub[p] = -ph * norm;
        double *hr = &vr[static_cast<size_t>(p) * k], *hi = &vi[static_cast<size_t>(p) * k];
        const cd v0 = ph * (n0 + norm);
        hr[f] = v0.real();
        hi[f] = v0.imag();
        for (int i = f + 1; i < k; ++i) {
            hr[i] = re[i * k + p];
            hi[i] = im[i * k + p];
        }
        const double b = beta[p] = 2.0 / ((n0 + norm) * (n0 + norm) + tail);
        for (int i = f; i < k; ++i) wr[i] = wi[i] = 0.0;
        for (int j = f; j < k; ++j) {  // w = beta a v, by the rows of a (the conjugates of its columns)
            const double *ar = &re[static_cast<size_t>(j) * k], *ai = &im[static_cast<size_t>(j) * k];
            const double xr = b * hr[j], xi = b * hi[j];
            for (int i = f; i < k; ++i) {
                wr[i] += ar[i] * xr + ai[i] * xi;
                wi[i] += ar[i] * xi - ai[i] * xr;
            }
        }
        double g = 0.0;  // v^H w, real for a Hermitian
        for (int i = f; i < k; ++i) g += hr[i] * wr[i] + hi[i] * wi[i];
        g *= 0.5 * b;
        for (int i = f; i < k; ++i) {
            wr[i] -= g * hr[i];
            wi[i] -= g * hi[i];
        }
        for (int i = f; i < k; ++i) {  // a -= v w^H + w v^H
            double *ar = &re[static_cast<size_t>(i) * k], *ai = &im[static_cast<size_t>(i) * k];
            const double vir = hr[i], vii = hi[i], wir = wr[i], wii = wi[i];
            for (int j = f; j < k; ++j) {
                ar[j] -= (vir * wr[j] + vii * wi[j]) + (wir * hr[j] + wii * hi[j]);
                ai[j] -= (vii * wr[j] - vir * wi[j]) + (wii * hr[j] - wir * hi[j]);
            }
        }
    }
    for (int i = 0; i < k; ++i) d[i] = re[static_cast<size_t>(i) * k + i];
    for (int i = 0; i + 1 < k; ++i) e[i] = std::abs(sub[i]);
    // implicit QR on (d, e); row j of z becomes the j-th eigenvector
    std::vector<double> z(kk, 0.0);
    for (int i = 0; i < k; ++i) z[static_cast<size_t>(i) * k + i] = 1.0;
    const double eps = 2.3e-16;
    for (int hi = k - 1, steps = 0; hi > 0;) {
        for (int i = 0; i < hi; ++i)
            if (std::fabs(e[i]) <= eps * (std::fabs(d[i]) + std::fabs(d[i + 1]))) e[i] = 0.0;
        if (e[hi - 1] == 0.0 || ++steps > 30 * k) {  // found, or given up on (NaN): two steps are usual
            e[hi - 1] = 0.0;
            --hi;
            continue;
        }
        int lo = hi - 1;
        while (lo > 0 && e[lo - 1] != 0.0) --lo;
        const double h = 0.5 * (d[hi - 1] - d[hi]), e2 = e[hi - 1] * e[hi - 1];
        const double mu = d[hi] - e2 / (h + (h >= 0.0 ? 1.0 : -1.0) * std::sqrt(h * h + e2));
        double x = d[lo] - mu, y = e[lo];  // the rotation that takes (x, y) to (r, 0)
        for (int i = lo; i < hi; ++i) {
            const double r = std::sqrt(x * x + y * y);
            if (r == 0.0) break;  // the bulge is gone: what is left is tridiagonal
            const double c = x / r, s = y / r;
            if (i > lo) e[i - 1] = r;
            const double p = d[i], q = d[i + 1], o = e[i];
            d[i] = c * (c * p + s * o) + s * (c * o + s * q);
            d[i + 1] = s * (s * p - c * o) + c * (c * q - s * o);
            e[i] = c * (c * o - s * p) + s * (c * q - s * o);
            if (i + 1 < hi) {
                x = e[i];
                y = s * e[i + 1];
                e[i + 1] *= c;
            }
            double *z0 = &z[static_cast<size_t>(i) * k], *z1 = z0 + k;
            for (int j = 0; j < k; ++j) {
                const double u = z0[j], t = z1[j];
                z0[j] = c * u + s * t;
                z1[j] = c * t - s * u;
            }
        }
    }
    const int top = static_cast<int>(std::max_element(d.begin(), d.end()) - d.begin());
    // back: the phases that made the sub-diagonal real, then the reflections, last one first
    out.assign(k, cd(0.0, 0.0));
    cd ph(1.0, 0.0);
    for (int i = 0; i < k; ++i) {
        out[i] = ph * z[static_cast<size_t>(top) * k + i];
        if (i + 1 < k && sub[i] != cd(0.0, 0.0)) ph *= sub[i] / std::abs(sub[i]);
    }
    for (int p = k - 2; p >= 0; --p) {
        if (beta[p] == 0.0) continue;
        const double *hr = &vr[static_cast<size_t>(p) * k], *hi = &vi[static_cast<size_t>(p) * k];
        cd g(0.0, 0.0);
        for (int i = p + 1; i < k; ++i) g += cd(hr[i], -hi[i]) * out[i];
        g *= beta[p];
        for (int i = p + 1; i < k; ++i) out[i] -= g * cd(hr[i], hi[i]);
    }
    int r0 = 0;
    while (r0 < k && !(std::abs(out[r0]) > 1e-14)) ++r0;
    if (r0 == k) return;
    const double mag = std::abs(out[r0]);
    const cd turn = std::conj(out[r0]) / mag;
    for (int r = 0; r < k; ++r) out[r] *= turn;
    out[r0] = mag;
}

}  // namespace dense
}  // namespace afc
