// ORACLE / TEST INFRASTRUCTURE ONLY.
//
// A plain FP64 statement of gate application on a dense vector, for hosts where
// the reference's csim kernels are not built (oracle/csim_ref.py picks).  Every
// gate is a 2^k x 2^k matrix over its target qubits (matrix bit i on target i),
// applied to the amplitudes whose control qubits have the wanted values.
// Vectors are complex128 (interleaved re, im) of length dim.
#include <algorithm>
#include <complex>
#include <cstdint>
#include <vector>

#ifdef _OPENMP
#include <omp.h>
#endif

typedef std::complex<double> cplx;

namespace {

void apply(const unsigned *targets, unsigned nt, uint64_t control_mask, uint64_t control_bits, const cplx *m, cplx *s,
           uint64_t dim) {
    const int rows = 1 << nt;
    std::vector<uint64_t> offset(rows, 0);
    for (int r = 0; r < rows; ++r)
        for (unsigned i = 0; i < nt; ++i)
            if ((r >> i) & 1) offset[r] |= uint64_t(1) << targets[i];
    const uint64_t used = offset[rows - 1];
#pragma omp parallel
    {
        std::vector<cplx> x(rows);
#pragma omp for
        for (uint64_t base = 0; base < dim; ++base) {
            if ((base & used) || (base & control_mask) != control_bits) continue;
            for (int r = 0; r < rows; ++r) x[r] = s[base | offset[r]];
            for (int r = 0; r < rows; ++r) {
                cplx sum = 0;
                for (int c = 0; c < rows; ++c) sum += m[r * rows + c] * x[c];
                s[base | offset[r]] = sum;
            }
        }
    }
}

}  // namespace

extern "C" {

void qsor_dense_dense1(unsigned t, const double *m, double *s, uint64_t dim) {
    apply(&t, 1, 0, 0, reinterpret_cast<const cplx *>(m), reinterpret_cast<cplx *>(s), dim);
}

void qsor_dense_dense2(unsigned t0, unsigned t1, const double *m, double *s, uint64_t dim) {
    const unsigned t[2] = {t0, t1};
    apply(t, 2, 0, 0, reinterpret_cast<const cplx *>(m), reinterpret_cast<cplx *>(s), dim);
}

void qsor_dense_dense_multi(const unsigned *targets, unsigned nt, const double *m, double *s, uint64_t dim) {
    apply(targets, nt, 0, 0, reinterpret_cast<const cplx *>(m), reinterpret_cast<cplx *>(s), dim);
}

void qsor_dense_controlled(const unsigned *controls, const unsigned *values, unsigned nc, const unsigned *targets,
                           unsigned nt, const double *m, double *s, uint64_t dim) {
    uint64_t mask = 0, bits = 0;
    for (unsigned i = 0; i < nc; ++i) {
        mask |= uint64_t(1) << controls[i];
        if (values[i]) bits |= uint64_t(1) << controls[i];
    }
    apply(targets, nt, mask, bits, reinterpret_cast<const cplx *>(m), reinterpret_cast<cplx *>(s), dim);
}

void qsor_dense_cnot(unsigned c, unsigned t, double *s, uint64_t dim) {
    const cplx x[4] = {0, 1, 1, 0};
    apply(&t, 1, uint64_t(1) << c, uint64_t(1) << c, x, reinterpret_cast<cplx *>(s), dim);
}

void qsor_dense_cz(unsigned c, unsigned t, double *s, uint64_t dim) {
    const cplx z[4] = {1, 0, 0, -1};
    apply(&t, 1, uint64_t(1) << c, uint64_t(1) << c, z, reinterpret_cast<cplx *>(s), dim);
}

void qsor_dense_swap(unsigned a, unsigned b, double *s, uint64_t dim) {
    const unsigned t[2] = {a, b};
    const cplx m[16] = {1, 0, 0, 0, 0, 0, 1, 0, 0, 1, 0, 0, 0, 0, 0, 1};
    apply(t, 2, 0, 0, m, reinterpret_cast<cplx *>(s), dim);
}

double qsor_dense_norm_squared(const double *s, uint64_t dim) {
    double sum = 0;
    for (uint64_t i = 0; i < 2 * dim; ++i) sum += s[i] * s[i];
    return sum;
}

void qsor_dense_inner_product(const double *bra, const double *ket, uint64_t dim, double *out2) {
    cplx sum = 0;
    for (uint64_t i = 0; i < dim; ++i)
        sum += std::conj(cplx(bra[2 * i], bra[2 * i + 1])) * cplx(ket[2 * i], ket[2 * i + 1]);
    out2[0] = sum.real();
    out2[1] = sum.imag();
}

void qsor_dense_init_zero(double *s, uint64_t dim) {
    std::fill(s, s + 2 * dim, 0.0);
    s[0] = 1.0;
}

int qsor_dense_max_threads(void) {
#ifdef _OPENMP
    return omp_get_max_threads();
#else
    return 1;
#endif
}

}  // extern "C"
