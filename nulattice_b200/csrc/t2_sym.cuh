// One step of a label-symmetric problem in two launches.  Included by
// ccsd_struct.cu inside its anonymous namespace.
//
// The one stored channel is symmetric under exchange of its two labels,
// B[a,b,i,j] = B[b,a,j,i], and so is its residual:
//   R[a,b,i,j] = S[a,b,i,j] + S[b,a,j,i],
// with S the off-diagonal terms that act on the second label (f_pp and the
// rank-h part of X_pp along b, X_hh along j) and half of the ladders and of the
// diagonal, which act on both.  The half diagonal comes first in the sum, so
// that S stays small near the solution and FP32 keeps its digits (relative
// error of nine FP32 steps against FP64, rms over 12 couplings each at L=3-6 and
// two, three and seven sites: 6.4-7.9e-8, 7.1e-8 on average; a residual summed
// whole, with every label stored, 6.3-7.8e-8 and 7.2e-8; with the diagonal added
// at the end 8.0-12e-8).  S of a row needs only that row:
//
// * k_sym_row: S of each row a into the output buffer, and the T1 update of
//   particle a (its T1 Fock term needs only the row, too);
// * k_sym_update: the pairs a <= b: both S, the Jacobi update into both places
//   (so the block stays symmetric bit for bit), and at its end the
//   convergence test.
//
// Against a residual formed whole (tables and Ga, k_t2_lat, T1, test: four
// launches) this is half of the multiply-adds, no reads of other rows and no
// Ga table.  A solve of A=28 L=6 on one B200: nine FP32 steps 610 -> 411 us,
// twenty FP64 steps 1810 -> 1310 us; A=28 L=4 FP32 346 -> 287 us.
//
// Terms: CCM/coupled_cluster.py:498-536, CCM/ccDgrams.py:215-251, 502-578.

constexpr int kSymNf = 6;          // off-diagonal f_pp entries of a particle (its neighbours)
constexpr int kSymFph = 6;         // staged f_ph entries of a hole
constexpr int kSymU = 8;           // columns of a thread of the update pass whose loads go out together

// ------------------------------------------------------------ row pass ----
// A block takes a run of columns b of one row a, a thread one b and sym_rows
// of its hole rows i: its sums are registers, its f_pp row and t1 sit in shared
// memory, Gb and X_hh are shared-memory broadcasts.  The particles of a warp
// are NH^2 elements apart in the staged row (49: an odd stride, no bank
// conflicts).  The loops over f_pp entries and holes are not unrolled: a block
// runs its code once (unrolled: the same time, four times the code).
// Bound by latency at the sizes that fit L2: one wave of blocks, each a chain
// of table loads, Gb, the sums and the stores, at 30% of the issue slots and
// 37% of the shared-memory bandwidth (A=28 L=6 FP32); so rows are cut into runs
// until every SM has two blocks, and FP64 halves the sums of a thread (33.6 ->
// 32.2 us there; FP32 gains nothing: 16.5 -> 24 us).
template <typename T>
__host__ __device__ constexpr int sym_rows(int nh) {
    return sizeof(T) == 8 && nh > 4 ? 4 : nh;
}
template <typename T>
__host__ __device__ constexpr int sym_parts(int nh) {   // threads of a column
    return (nh + sym_rows<T>(nh) - 1) / sym_rows<T>(nh);
}
constexpr int kSymMost = 256;      // most columns of a block

struct SymSmem {
    int64_t gb, x2, hh, ta, f, off, t, row, total;
};

template <typename T, int NH>
__host__ __device__ inline SymSmem sym_smem(int64_t np, int64_t cols) {
    constexpr int64_t el = sizeof(T);
    SymSmem s;
    s.gb = 0;
    s.x2 = s.gb + lat_round16(el * NH * NH * 8);
    s.hh = s.x2 + lat_round16(el * NH * 8);
    s.ta = s.hh + lat_round16(el * NH * NH);
    s.f = s.ta + lat_round16(el * 8);
    s.off = s.f + lat_round16(el * kSymNf * cols);
    s.t = s.off + lat_round16(4 * kSymNf * cols);
    s.row = s.t + lat_round16(el * NH * cols);
    s.total = s.row + lat_round16(el * (np * NH * NH + 16 / el));
    return s;
}

// v[0..N) += c x: FP32 two at a time as packed multiply-adds, which halves
// their issue slots.
template <int N>
__device__ __forceinline__ void sym_axpy(double (&v)[N], double c, const double* x) {
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] += c * x[e];
}
template <int N>
__device__ __forceinline__ void sym_axpy(float (&v)[N], float c, const float* x) {
#pragma unroll
    for (int e = 0; e + 1 < N; e += 2) {
        const float2 r = __ffma2_rn(make_float2(c, c), make_float2(x[e], x[e + 1]), make_float2(v[e], v[e + 1]));
        v[e] = r.x;
        v[e + 1] = r.y;
    }
    if (N % 2) v[N - 1] += c * x[N - 1];
}

template <typename T, int NH>
__global__ void __launch_bounds__(kSymMost * sym_parts<T>(NH), sizeof(T) == 4 ? 2 : 1) k_sym_row(nlb_struct_problem P, nlb_struct_state S, int runs) {
    constexpr int NHP = NH * NH, VEC = 16 / (int)sizeof(T), IR = sym_rows<T>(NH), PARTS = sym_parts<T>(NH), NE = IR * NH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // f_ph column lists of the holes (a lattice hole has at most six particle
    // neighbours; longer lists continue in global memory)
    __shared__ T sfv[NH * kSymFph];
    __shared__ int32_t sfo[NH * kSymFph], sfe[NH];
    // the T1 update of particle a, FP64 (holes in label order): Q, X_hh of the
    // T1 equation, the f_pp neighbours' terms, t1, f_ph, energy and step parts
    __shared__ T sdd[NH];   // half of the diagonal of X_hh
    __shared__ double sq[NHP], sxh[NHP], sft[(kSymNf + 1) * NH], st1[NH], sfh[NH], s_sum, sen[NH], sdn[NH];
    const nlb_ctrl* c = S.ctrl;
    if (c->status != NLB_RUNNING) return;
    const int par = c->parity;
    const bool t2 = !c->ccs;
    const double* __restrict__ t1 = t1_buf(S, par);
    const PrepView V = prep_view(S.prep, P);
    const nlb_channel& ch = P.chan[0];
    const int np = P.p, tid = threadIdx.x, nt = blockDim.x;
    const int a = blockIdx.x / runs, run = blockIdx.x - a * runs;
    const int c0 = (int)((int64_t)run * np / runs), c1 = (int)((int64_t)(run + 1) * np / runs);
    const int ncol = nt / PARTS, part = tid / ncol, col = tid - part * ncol;   // ncol: whole warps
    const SymSmem L = sym_smem<T, NH>(np, ncol);
    T* sgb = reinterpret_cast<T*>(smem_raw + L.gb);   // [k][i][8]
    T* sx2 = reinterpret_cast<T*>(smem_raw + L.x2);
    T* shh = reinterpret_cast<T*>(smem_raw + L.hh);
    T* sta = reinterpret_cast<T*>(smem_raw + L.ta);
    const int64_t rbase = ch.offset + (int64_t)a * np * NHP;
    const T* src = t2_buf<const T>(S, par) + rbase;
    const int rowlen = np * NHP;
    const int mis = (int)((reinterpret_cast<uintptr_t>(src) / sizeof(T)) & (VEC - 1));
    T* sr = reinterpret_cast<T*>(smem_raw + L.row) + mis;
    if (t2) {
        // the row at the shift that makes 16-byte copies aligned on both sides
        const int head = min((VEC - mis) & (VEC - 1), rowlen), nvec = (rowlen - head) / VEC;
        for (int e = tid; e < head; e += nt) cp_async_el<sizeof(T)>(sr + e, src + e);
        for (int v = tid; v < nvec; v += nt) cp_async16(sr + head + v * VEC, src + head + v * VEC);
        for (int e = head + nvec * VEC + tid; e < rowlen; e += nt) cp_async_el<sizeof(T)>(sr + e, src + e);
        cp_async_commit();
    }
    const int ga = P.p_ord[a];
    // X_hh of the T2 equation, and the tables of the T1 update
    for (int u = tid; u < NHP; u += nt) {
        const int k = u / NH, j = u - k * NH, kk = P.h_ord[k], jj = P.h_ord[j];
        const double q = q_entry(P, t1, kk, jj), f = P.f_hh[(int64_t)kk * NH + jj];
        sx2[k * 8 + j] = k == j ? T(0) : (T)(-f - q);   // the diagonal is in the denominator
        if (k == j) sdd[k] = (T)(0.5 * (-f - q));
        sq[u] = q;
        sxh[u] = -f - 0.5 * q;
        if (blockIdx.x == 0 && k == j) V.dhc[k] = -f - q;   // for the update pass
    }
    if (run == 0) {
        for (int u = nt - 1 - tid; u < (kSymNf + 1) * NH; u += nt) {
            const int q = u / NH, i = u - q * NH, x = P.fpp_ptr[a] + q;
            sft[u] = x < P.fpp_ptr[a + 1] ? P.fpp_val[x] * t1[(int64_t)P.p_ord[P.fpp_col[x]] * NH + P.h_ord[i]] : 0.0;
        }
        if (tid == nt - 1) {
            s_sum = s_entry(P, t1, ga);
            V.dpc[a] = P.fpp_diag[ga] - s_sum;   // for the update pass
        }
    }
    if (tid < NH) {
        const int64_t x = (int64_t)ga * NH + P.h_ord[tid];
        st1[tid] = t1[x];
        sta[tid] = (T)t1[x];
        sfh[tid] = P.f_ph[x];
    }
    if (t2) {
        const int32_t* hptr = P.hh_ptr + ch.hh_ptr_off;
        for (int e = tid; e < NHP; e += nt)
            shh[e] = hptr[e + 1] > hptr[e] ? T(0.5) * (T)P.hh_val[ch.hh_col_off + hptr[e]] : T(0);
        for (int w = tid; w < NH * kSymFph; w += nt) {
            const int k = w / kSymFph, q = P.fph_ptr[k] + w - k * kSymFph, q1 = P.fph_ptr[k + 1];
            sfv[w] = q < q1 ? (T)P.fph_val[q] : T(0);
            sfo[w] = q < q1 ? P.fph_col[q] * NHP : 0;
            if (w == k * kSymFph) sfe[k] = q1;
        }
    }
    const int b = c0 + col;
    const bool act = t2 && b < c1;
    T* sf = reinterpret_cast<T*>(smem_raw + L.f) + col;            // [q][column], as the next two
    int32_t* so = reinterpret_cast<int32_t*>(smem_raw + L.off) + col;
    T* st = reinterpret_cast<T*>(smem_raw + L.t) + col;
    T cpp = T(0), dab = T(0);   // of the pair (a, b): half of its ladder and of its f_pp diagonals
    if (act) {
        const int32_t* pptr = P.pp_ptr + ch.pp_ptr_off + (int64_t)a * np + b;
        if (pptr[1] > pptr[0]) cpp = T(0.5) * (T)P.pp_val[ch.pp_col_off + pptr[0]];
        dab = (T)(0.5 * (P.fpp_diag[ga] + P.fpp_diag[P.p_ord[b]]));
        if (part == PARTS - 1) {
            const double* tb = t1 + (int64_t)P.p_ord[b] * NH;
#pragma unroll
            for (int k = 0; k < NH; ++k) st[k * ncol] = (T)tb[P.h_ord[k]];
        }
        if (part == 0) {
            // the neighbours; the diagonal is in the update pass
            const int q0 = P.fpp_ptr[b], q1 = P.fpp_ptr[b + 1];
            int n = 0;
#pragma unroll
            for (int q = 0; q <= kSymNf; ++q) {
                const int c2 = q0 + q < q1 ? P.fpp_col[q0 + q] : b;
                const T f = q0 + q < q1 ? (T)P.fpp_val[q0 + q] : T(0);
                if (c2 == b) continue;
                sf[n * ncol] = f;
                so[n * ncol] = c2 * NHP;
                ++n;
            }
            for (; n < kSymNf; ++n) {
                sf[n * ncol] = T(0);
                so[n * ncol] = b * NHP;
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();
    if (t2) {
        // Gb[k][i,j] = sum_c f_ck B[a,c,i,j]
        for (int e = tid; e < NH * NHP; e += nt) {
            const int k = e / NHP, h2 = e - k * NHP;
            T acc = T(0);
#pragma unroll
            for (int q = 0; q < kSymFph; ++q) acc += sfv[k * kSymFph + q] * sr[sfo[k * kSymFph + q] + h2];
            for (int q = P.fph_ptr[k] + kSymFph; q < sfe[k]; ++q) acc += (T)P.fph_val[q] * sr[P.fph_col[q] * NHP + h2];
            sgb[(k * NH + h2 / NH) * 8 + h2 % NH] = acc;
        }
        __syncthreads();
    }
    // T1 update of (a, i): R1 = f_ph + F2 of every other label + X_pp t1 + t1
    // X_hh with F2 = sum_k Gb[k][i,k] (coupled_cluster.py:342-414), by the last
    // threads (the first have a column each); F2 is added in FP64 for either type
    if (run == 0 && nt - 1 - tid < NH) {
        const int i = nt - 1 - tid;
        double f2 = 0.0;
        if (t2) {
#pragma unroll
            for (int k = 0; k < NH; ++k) f2 += (double)sgb[(k * NH + i) * 8 + k];
        }
        double h1 = sfh[i] + sym_others(P) * f2;
#pragma unroll
        for (int q = 0; q <= kSymNf; ++q) h1 += sft[q * NH + i];
#pragma unroll
        for (int k = 0; k < NH; ++k) h1 += st1[k] * (sxh[k * NH + i] - 0.5 * sq[k * NH + i]);
        const double d1 = -((P.fpp_diag[ga] - 0.5 * s_sum) + sxh[i * NH + i]);
        const double m = c->mixing, x = st1[i], out = m * x + (1.0 - m) * (x + h1 / d1), d = out - x;
        const int64_t at = (int64_t)ga * NH + P.h_ord[i];
        t1_buf(S, par ^ 1)[at] = out;
        if (S.diis_t1 != nullptr && c->max_diis > 0 && c->diis_count < c->max_diis)
            S.diis_t1[(int64_t)c->diis_count * np * NH + at] = d;
        sen[i] = sfh[i] * out;
        sdn[i] = d * d;
    }
    // sums of hole rows i0 .. i0 + IR (the last part's may begin in the rows of
    // the one before, which then writes them)
    const int i0 = min(part * IR, NH - IR);
    T acc[NE];
    if (act) {
        const T* own = sr + b * NHP + i0 * NH;
        // half of both ladders (diagonal, on tau = t2 + t1 t1)
        {
            T t[NH];
#pragma unroll
            for (int k = 0; k < NH; ++k) t[k] = st[k * ncol];
#pragma unroll
            for (int e = 0; e < NE; ++e) acc[e] = (dab + (sdd[i0 + e / NH] + sdd[e % NH])) * own[e] + (shh[i0 * NH + e] + cpp) * (own[e] + sta[i0 + e / NH] * t[e % NH]);
        }
        // f_pp along b
#pragma unroll 1
        for (int q = 0; q < kSymNf; ++q) sym_axpy<NE>(acc, sf[q * ncol], sr + so[q * ncol] + i0 * NH);
        // rank-h part of X_pp along b (-t1_bk Gb[k]), and X_hh along j
#pragma unroll 1
        for (int k = 0; k < NH; ++k) {
            const T tk = -st[k * ncol];
            T x[8];
            lds8(sx2 + k * 8, x);
#pragma unroll
            for (int i = 0; i < IR; ++i) {
                T g[8];
                lds8(sgb + (k * NH + i0 + i) * 8, g);
                const T bi = own[i * NH + k];
#pragma unroll
                for (int j = 0; j < NH; ++j) acc[i * NH + j] += tk * g[j] + x[j] * bi;
            }
        }
    }
    __syncthreads();   // every read of the row is done: the sums take its place
    if (run == 0 && tid == nt - 1) {   // particle a's parts of the energy and the T1 step, in hole order
        double e = 0.0, d = 0.0;
#pragma unroll
        for (int i = 0; i < NH; ++i) {
            e += sen[i];
            d += sdn[i];
        }
        V.slots(kRedE)[a] = sym_labels(P) * e;
        V.slots(kRedDt1)[a] = sym_labels(P) * d;
    }
    if (act) {
        T* own = sr + b * NHP + i0 * NH;
        const int e0 = (part * IR - i0) * NH;
#pragma unroll
        for (int e = 0; e < NE; ++e)
            if (e >= e0) own[e] = acc[e];
    }
    __syncthreads();
    T* dst = t2_buf<T>(S, par ^ 1) + rbase;
    if (t2)
        for (int e = c0 * NHP + tid; e < c1 * NHP; e += nt) __stcg(dst + e, sr[e]);
}

// --------------------------------------------------------- update pass ----
// Blocks of the pairs a <= b: row a takes ceil((np - a) / cols) blocks of up
// to `cols` columns from a on.
__host__ __device__ inline int64_t sym_blocks(int np, int cols) {
    const int q = (np + cols - 1) / cols;      // blocks of row 0
    return (int64_t)q * (np - (q - 1) * cols) + (int64_t)cols * q * (q - 1) / 2;
}

// Block `blk`: row a, first column b0 (rows with q blocks come in groups).
__device__ __forceinline__ void sym_block(int np, int cols, int blk, int& a, int& b0) {
    int q = (np + cols - 1) / cols, rows = np - (q - 1) * cols, first = 0;
    while (blk >= rows * q) {
        blk -= rows * q;
        first += rows;
        rows = cols;
        --q;
    }
    const int r = blk / q;
    a = first + r;
    b0 = a + (blk - r * q) * cols;
}

template <typename T, int NH>
__device__ void sym_update_body(const nlb_struct_problem& P, const nlb_struct_state& S, int blk, int cols) {
    constexpr int NHP = NH * NH;
    const nlb_ctrl* c = S.ctrl;
    const PrepView V = prep_view(S.prep, P);
    const int64_t off0 = P.chan[0].offset;
    const int np = P.p, par = c->parity;
    const T* __restrict__ B = t2_buf<const T>(S, par) + off0;
    T* Bo = t2_buf<T>(S, par ^ 1) + off0;
    T* E2 = (S.diis_t2 != nullptr && c->max_diis > 0 && c->diis_count < c->max_diis)
                ? static_cast<T*>(S.diis_t2) + (int64_t)c->diis_count * P.n_t2 + off0 : nullptr;
    const T m = (T)c->mixing, om = (T)(1.0 - c->mixing);
    int a, b0;
    sym_block(np, cols, blk, a, b0);
    const int b1 = b0 + cols < np ? b0 + cols : np;
    // a thread owns one hole pair (i, j) of every CPB-th column
    constexpr int CPB = kThreads / NHP;
    const int cl = threadIdx.x / NHP, hp = threadIdx.x - cl * NHP, i = hp / NH, j = hp - i * NH;
    // denominators: the diagonals of X_pp and X_hh added in FP64 and rounded once
    const double da = V.dpc[a] + (V.dhc[i] + V.dhc[j]);
    T nrm = T(0);
    if (cl < CPB) {
        int64_t e0 = ((int64_t)a * np + b0 + cl) * NHP + hp;              // (a, b, i, j)
        int64_t x0 = ((int64_t)(b0 + cl) * np + a) * NHP + j * NH + i;    // (b, a, j, i)
        const int64_t xs = (int64_t)CPB * np * NHP;
        // kSymU columns whose loads go out together
        for (int b = b0 + cl; b < b1; b += kSymU * CPB) {
            T x[kSymU], s1[kSymU], s2[kSymU];
            double db[kSymU];
#pragma unroll
            for (int u = 0; u < kSymU; ++u) {
                const int bu = b + u * CPB;
                if (bu >= b1) continue;
                x[u] = B[e0 + u * CPB * NHP];
                s1[u] = __ldcg(Bo + e0 + u * CPB * NHP);
                s2[u] = __ldcg(Bo + x0 + u * xs);
                db[u] = V.dpc[bu];
            }
#pragma unroll
            for (int u = 0; u < kSymU; ++u) {
                const int bu = b + u * CPB;
                // (i, j) of column a stands for (j, i), too
                if (bu >= b1 || (bu == a && i > j)) continue;
                const T r = s1[u] + s2[u];
                const T tn = x[u] - lat_div(r, (T)(da + db[u]));
                const T out = m * x[u] + om * tn, d = out - x[u];
                const bool two = bu != a || i != j;   // two places, and twice in the norm
                nrm += (two ? T(2) : T(1)) * d * d;
                __stcg(Bo + e0 + u * CPB * NHP, out);
                if (E2) __stcg(E2 + e0 + u * CPB * NHP, d);
                if (two) {
                    __stcg(Bo + x0 + u * xs, out);
                    if (E2) __stcg(E2 + x0 + u * xs, d);
                }
            }
            e0 += kSymU * CPB * NHP;
            x0 += kSymU * xs;
        }
    }
    const double s = block_sum((double)nrm);
    if (threadIdx.x == 0) V.slots(kRedDt2)[blk] = t2_weight(P) * s;
}

// The update pass, and the convergence test by its last block to finish (the
// counter is in the control block and back at zero afterwards).  fin = 0: only
// the update.
template <typename T, int NH>
__global__ void __launch_bounds__(kThreads) k_sym_update(nlb_struct_problem P, nlb_struct_state S, int cols, int fin) {
    nlb_ctrl* c = S.ctrl;
    if (c->status != NLB_RUNNING) return;
    if (!c->ccs) sym_update_body<T, NH>(P, S, blockIdx.x, cols);
    if (!fin) return;
    __shared__ int last;
    unsigned* count = reinterpret_cast<unsigned*>(&c->gram[120]);
    if (threadIdx.x == 0) {
        __threadfence();   // this block's partial sums before its count
        last = atomicAdd(count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) *count = 0;
    finish_body(c, prep_view(S.prep, P).red, P.p, (int)gridDim.x);
}
