// Label-symmetric problems: between the stored label and the full layout.
//
// A contact that treats every spin-isospin label alike gives each label the
// same t1[P_g, H_g] and each pair of labels the same t2 block, so a
// label-symmetric problem (bits 24-31 of the tuning word) stores one label
// and one block.  These kernels check that amplitudes of the full layout
// have that form and write the full layout from the stored parts.

#include <cuda_runtime.h>
#include <stdio.h>

#include "nulattice_b200.h"

void nlb_internal_set_error(const char* msg);

namespace {

#include "common.cuh"

int sfail(int code, const char* msg) {
    nlb_internal_set_error(msg);
    return code;
}

int scheck(const char* where) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        char buf[512];
        snprintf(buf, sizeof(buf), "%s: %s", where, cudaGetErrorString(e));
        nlb_internal_set_error(buf);
        return NLB_ERR_LAUNCH;
    }
    return NLB_OK;
}

constexpr int kT = 256;

int sgrid(int64_t n) {
    const int64_t g = (n + kT - 1) / kT;
    return (int)(g < 1 ? 1 : (g < 148 * 8 ? g : 148 * 8));
}

// Particle order and hole order of all m labels, label by label.
struct Orders {
    const int32_t *p, *h;
};

// out[0] != 0: t1 or t2 differs between labels or is NaN, or t1 joins two labels;
// out[1], out[2]: largest |B[a,b,i,j] - B[b,a,j,i]| and |B[a,b,i,j]| of the
// block, as the bit patterns of non-negative doubles (which order like them);
// t1_out (optional): t1 of the first label.
template <typename T>
__global__ void __launch_bounds__(kT) k_sym_check(int m, int np, int nh, Orders o, const double* t1, const T* t2,
                                                  double* t1_out, unsigned long long* out) {
    const int64_t n0 = (int64_t)np * np * nh * nh, nb = (int64_t)np * nh;
    const int P = m * np, H = m * nh, pairs = m * (m - 1) / 2;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool bad = false;
    double asym = 0.0, big = 0.0;
    for (int64_t e = tid; e < n0; e += stride) {
        const T v = t2[e];
        bad |= v != v;
        for (int c = 1; c < pairs; ++c) bad |= !(t2[c * n0 + e] == v);
        const int ab = (int)(e / (nh * nh)), ij = (int)(e - (int64_t)ab * nh * nh);
        const int a = ab / np, b = ab - a * np, i = ij / nh, j = ij - i * nh;
        asym = fmax(asym, fabs((double)v - (double)t2[(((int64_t)b * np + a) * nh + j) * nh + i]));
        big = fmax(big, fabs((double)v));
    }
    for (int64_t u = tid; u < (int64_t)P * H; u += stride) {
        const int x = (int)(u / H), y = (int)(u - (int64_t)x * H);
        const int g = x / np, gh = y / nh;
        const double v = t1[(int64_t)o.p[x] * H + o.h[y]];
        if (g != gh) bad |= v != 0.0;
        else bad |= !(v == t1[(int64_t)o.p[x - g * np] * H + o.h[y - g * nh]]);   // label 0: NaN alone
    }
    if (t1_out)
        for (int64_t u = tid; u < nb; u += stride) t1_out[u] = t1[(int64_t)o.p[u / nh] * H + o.h[u % nh]];
    for (int s = 16; s > 0; s >>= 1) {
        asym = fmax(asym, __shfl_xor_sync(0xffffffffu, asym, s));
        big = fmax(big, __shfl_xor_sync(0xffffffffu, big, s));
    }
    bad = __any_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (bad) atomicMax(out, 1ull);
        atomicMax(out + 1, (unsigned long long)__double_as_longlong(asym));
        atomicMax(out + 2, (unsigned long long)__double_as_longlong(big));
    }
}

__global__ void k_sym_t1(int m, int np, int nh, Orders o, const double* t1, double* full) {
    const int P = m * np, H = m * nh;
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < (int64_t)P * H;
         u += (int64_t)gridDim.x * blockDim.x) {
        const int x = (int)(u / H), y = (int)(u - (int64_t)x * H);
        const int g = x / np, k = y - g * nh;
        full[(int64_t)o.p[x] * H + o.h[y]] = (k >= 0 && k < nh) ? t1[(int64_t)(x - g * np) * nh + k] : 0.0;
    }
}

template <typename T>
__global__ void k_sym_copies(const T* t2, T* full, int64_t n0, int pairs) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n0; e += (int64_t)gridDim.x * blockDim.x) {
        const T v = t2[e];
        for (int c = 0; c < pairs; ++c) __stcs(full + c * n0 + e, v);
    }
}

// dense[a, b, i, j] (zero-filled by the caller) with the four antisymmetric images of every pair of labels
template <typename T>
__global__ void k_sym_dense(int m, int np, int nh, Orders o, const T* t2, double* full) {
    const int64_t n0 = (int64_t)np * np * nh * nh, p = (int64_t)m * np, h = (int64_t)m * nh;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n0; e += (int64_t)gridDim.x * blockDim.x) {
        const int ab = (int)(e / (nh * nh)), ij = (int)(e - (int64_t)ab * nh * nh);
        const int ap = ab / np, bp = ab - ap * np, ip = ij / nh, jp = ij - ip * nh;
        const double v = (double)t2[e];
        for (int g = 0; g < m; ++g)
            for (int k = g + 1; k < m; ++k) {
                const int64_t a = o.p[g * np + ap], b = o.p[k * np + bp], i = o.h[g * nh + ip], j = o.h[k * nh + jp];
                full[((a * p + b) * h + i) * h + j] = v;
                full[((b * p + a) * h + i) * h + j] = -v;
                full[((a * p + b) * h + j) * h + i] = -v;
                full[((b * p + a) * h + j) * h + i] = v;
            }
    }
}

int sym_ok(const nlb_struct_problem* P, const int32_t* po, const int32_t* ho, int32_t dtype, const char* who) {
    if (!P || !po || !ho || (dtype != NLB_F64 && dtype != NLB_F32)) return sfail(NLB_ERR_ARG, who);
    if (sym_labels(*P) < 2 || P->p <= 0 || P->h <= 0 || P->n_t2 != (int64_t)P->p * P->p * P->h * P->h)
        return sfail(NLB_ERR_ARG, who);
    return NLB_OK;
}

}  // namespace

extern "C" {

int nlb_sym_check(const nlb_struct_problem* P, const int32_t* p_ord, const int32_t* h_ord, const double* t1,
                  const void* t2, int32_t dtype, double* t1_out, uint64_t* out, nlb_stream_t stream) {
    int rc = sym_ok(P, p_ord, h_ord, dtype, "nlb_sym_check: bad argument");
    if (rc) return rc;
    if (!t1 || !t2 || !out) return sfail(NLB_ERR_ARG, "nlb_sym_check: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    const Orders o{p_ord, h_ord};
    const int m = sym_labels(*P), g = sgrid(P->n_t2);
    unsigned long long* r = reinterpret_cast<unsigned long long*>(out);
    cudaMemsetAsync(out, 0, 3 * sizeof(uint64_t), s);
    if (dtype == NLB_F64) k_sym_check<double><<<g, kT, 0, s>>>(m, P->p, P->h, o, t1, (const double*)t2, t1_out, r);
    else k_sym_check<float><<<g, kT, 0, s>>>(m, P->p, P->h, o, t1, (const float*)t2, t1_out, r);
    return scheck("nlb_sym_check");
}

int nlb_sym_expand(const nlb_struct_problem* P, const int32_t* p_ord, const int32_t* h_ord, const double* t1,
                   double* t1_full, const void* t2, int32_t dtype, void* t2_full, int32_t dense, nlb_stream_t stream) {
    int rc = sym_ok(P, p_ord, h_ord, dtype, "nlb_sym_expand: bad argument");
    if (rc) return rc;
    if ((t1 && !t1_full) || (t2 && !t2_full)) return sfail(NLB_ERR_ARG, "nlb_sym_expand: null output");
    cudaStream_t s = (cudaStream_t)stream;
    const Orders o{p_ord, h_ord};
    const int m = sym_labels(*P), np = P->p, nh = P->h, pairs = m * (m - 1) / 2, g = sgrid(P->n_t2);
    if (t1) k_sym_t1<<<sgrid((int64_t)m * np * m * nh), kT, 0, s>>>(m, np, nh, o, t1, t1_full);
    if (t2 && dense) {
        if (dtype == NLB_F64) k_sym_dense<double><<<g, kT, 0, s>>>(m, np, nh, o, (const double*)t2, (double*)t2_full);
        else k_sym_dense<float><<<g, kT, 0, s>>>(m, np, nh, o, (const float*)t2, (double*)t2_full);
    } else if (t2) {
        if (dtype == NLB_F64)
            k_sym_copies<double><<<g, kT, 0, s>>>((const double*)t2, (double*)t2_full, P->n_t2, pairs);
        else k_sym_copies<float><<<g, kT, 0, s>>>((const float*)t2, (float*)t2_full, P->n_t2, pairs);
    }
    return scheck("nlb_sym_expand");
}

}  // extern "C"
