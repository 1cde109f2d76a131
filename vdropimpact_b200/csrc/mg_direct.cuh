// Exact solve of a separable finest level (included by mg.cu).
//
// The MAC operator (cell-centred, 5-point) and the FEM operator
// (node-centred bilinear, 9-point) have constant coefficients and natural
// ends in x on the whole grid, so cosines diagonalise their x part: DCT-II
// over the cells, DCT-I over the nodes. Writing the residual's rows in that
// basis leaves one tridiagonal system in y per mode, constant but for its
// first and last row. A solve from iterate z is then
//   dr_forward_k : r = b - A z, ||b||^2, ||r||^2, the first decision, and the
//                  rows of r transformed (two rows as one complex FFT)
//   dr_modal_k   : the tridiagonal systems
//   dr_inverse_k : the rows transformed back and added to z
//   dr_check_k   : ||b - A z||^2 and the decision
// in place of every V-cycle. Whatever tolerance rounding leaves unreached
// goes to the V-cycles of mg.cu, which start from this z.
//
// Row lengths that are a power of two (cells, or node intervals) use a
// power-of-two FFT in shared memory; any other length uses Bluestein's
// chirp convolution over a padded power of two. Grids whose padded row
// exceeds DR_MAX_P points or whose columns exceed DR_MAX_ROWS rows keep the
// V-cycles.
//
// Bound: the four launches move 9 words a point through L2 and DRAM (b and z
// read twice, the modal array written, updated and read, z updated), 151 MB
// at 2048 x 1024, 23 us at the measured copy rate; the transforms are bound
// by shared-memory passes and the barriers between them. Whole calls of
// vdi_mg_solve from zero to 1e-10, the V-cycles against this path: MAC 64 x
// 32 297 and 58 us, 1000 x 500 4860 and 92 us, 2048 x 1024 991 and 112-143 us
// (with and without the sweep of dr_relax_k), FEM 1025 x 513 428 and 83 us.

static constexpr int DR_MAX_P = 8192;      // 147 KB of shared memory with its padding
static constexpr int DR_MAX_CHUNKS = 128;  // chunks of a column, 4 modes a block: 512 threads
static constexpr int DR_MAX_L = 32;
static constexpr long DR_MAX_ROWS = long(DR_MAX_CHUNKS) * DR_MAX_L;

/** Device tables of one level's exact solve. */
struct DirectPlan {
    int m = 0, n = 0;
    int logp = 0;              // FFT length 2^logp
    int len = 0;               // length of the DFT a row needs (chirp form)
    int j0 = 0, R = 0;         // first solved row and their count (a Dirichlet row lies below row j0 = 1)
    int L = 0, S = 0;          // rows of a chunk, chunks of a column
    int modes = 0;             // modes a block of dr_modal_k takes
    double row0 = 1;           // factor of the Dirichlet row's source
    const double2* tw = nullptr;     // exp(-2 pi i k / P)
    const double2* post = nullptr;   // cells: (cos, sin)(pi k / 2m); then the modes' norms
    const double* norm = nullptr;    // 1 / C_k
    const double2* chirp = nullptr;  // exp(-pi i k^2 / len)
    const double2* bhat = nullptr;   // transform of the conjugate chirp over P
    const double* off = nullptr;     // [m] off-diagonal of mode k
    // per chunk kind (0 first, 1 middle, 2 last), row of the chunk and mode
    const double *inv = nullptr, *pp = nullptr, *qq = nullptr;
    // per chunk and mode: the separators' system
    const double *ri = nullptr, *rl = nullptr, *rc = nullptr;
    double* work = nullptr;    // n x m modal array
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cswap(double2 a) { return make_double2(a.y, a.x); }

__device__ __forceinline__ void dft2(double2& a, double2& b) {
    const double2 t = csub(a, b);
    a = cadd(a, b);
    b = t;
}
/** Forward DFT of four values in natural order. */
__device__ __forceinline__ void dft4(double2& a, double2& b, double2& c, double2& d) {
    dft2(a, c);
    dft2(b, d);
    d = make_double2(d.y, -d.x);   // -i d
    dft2(a, b);
    dft2(c, d);
    const double2 t = b;
    b = c;
    c = t;
}
/** Forward DFT of eight values in natural order. */
__device__ __forceinline__ void dft8(double2 (&v)[8]) {
    constexpr double H = 0.70710678118654752440;
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    const double2 t1 = make_double2(H * (v[3].x + v[3].y), H * (v[3].y - v[3].x));     // e^{-i pi/4}
    const double2 t2 = make_double2(v[5].y, -v[5].x);                                  // -i
    const double2 t3 = make_double2(H * (v[7].y - v[7].x), -H * (v[7].x + v[7].y));    // e^{-3 i pi/4}
    const double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], t0 = v[1];
    v[0] = cadd(e0, t0);
    v[4] = csub(e0, t0);
    v[1] = cadd(e1, t1);
    v[5] = csub(e1, t1);
    v[2] = cadd(e2, t2);
    v[6] = csub(e2, t2);
    v[3] = cadd(e3, t3);
    v[7] = csub(e3, t3);
}

/** Shared-memory place of element i: one 16-byte word of padding after
 * every eight keeps the eight lanes of an access phase in different banks
 * in every pass of dr_fft (strides 2, 4 and 8 on writing, 1 on reading). */
__device__ __forceinline__ int dr_at(int i) { return i + (i >> 3); }

/** Forward DFT of the P = 2^logp complex values at sm[dr_at(.)], in place,
 * by the block's first P/8 threads: Stockham passes of radix 8 after one of
 * radix 2, 4 or 8. Every thread of the block calls it; it starts and ends
 * with a barrier. */
__device__ __forceinline__ void dr_fft(double2* sm, int logp, const double2* __restrict__ tw) {
    const int t = threadIdx.x, n8 = 1 << (logp - 3), rem = logp % 3;
    const bool on = t < n8;
    double2 v[8];
    __syncthreads();
    if (on) {
#pragma unroll
        for (int q = 0; q < 8; q++) v[q] = sm[dr_at(t + q * n8)];
    }
    __syncthreads();
    int ns, lns;
    if (rem == 0) {
        if (on) {
            dft8(v);
#pragma unroll
            for (int r = 0; r < 8; r++) sm[dr_at(8 * t + r)] = v[r];
        }
        lns = 3;
    } else if (rem == 1) {
        if (on) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                dft2(v[u], v[u + 4]);
                sm[dr_at(2 * (t + u * n8))] = v[u];
                sm[dr_at(2 * (t + u * n8) + 1)] = v[u + 4];
            }
        }
        lns = 1;
    } else {
        if (on) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                dft4(v[u], v[u + 2], v[u + 4], v[u + 6]);
#pragma unroll
                for (int r = 0; r < 4; r++) sm[dr_at(4 * (t + u * n8) + r)] = v[u + 2 * r];
            }
        }
        lns = 2;
    }
    for (; lns < logp; lns += 3) {
        ns = 1 << lns;
        const int k = t & (ns - 1), st = logp - 3 - lns;
        __syncthreads();
        if (on) {
            const double2 w1 = __ldg(tw + (k << st)), w2 = __ldg(tw + (2 * k << st)), w4 = __ldg(tw + (4 * k << st));
#pragma unroll
            for (int q = 0; q < 8; q++) v[q] = sm[dr_at(t + q * n8)];
            v[1] = cmul(v[1], w1);
            v[2] = cmul(v[2], w2);
            v[4] = cmul(v[4], w4);
            v[3] = cmul(v[3], cmul(w1, w2));
            v[5] = cmul(v[5], cmul(w1, w4));
            const double2 w6 = cmul(w2, w4);
            v[6] = cmul(v[6], w6);
            v[7] = cmul(v[7], cmul(w1, w6));
            dft8(v);
        }
        __syncthreads();
        if (on) {
            const int o = ((t - k) << 3) + k;
#pragma unroll
            for (int r = 0; r < 8; r++) sm[dr_at(o + r * ns)] = v[r];
        }
    }
    __syncthreads();
}

/** The DFT of length p.len (or 2^logp when not BLUE) of the values in sm;
 * BLUE: the caller has multiplied them by the chirp and padded with zeros,
 * and multiplies element k of the swapped result by chirp[k] (dr_out). */
template <bool BLUE>
__device__ __forceinline__ void dr_dft(double2* sm, const DirectPlan& p) {
    dr_fft(sm, p.logp, p.tw);
    if constexpr (BLUE) {
        const int P = 1 << p.logp;
        for (int i = threadIdx.x; i < P; i += blockDim.x) {
            double2* w = sm + dr_at(i);
            *w = cswap(cmul(*w, __ldg(p.bhat + i)));
        }
        dr_fft(sm, p.logp, p.tw);
    }
}
template <bool BLUE>
__device__ __forceinline__ double2 dr_out(const double2* sm, const DirectPlan& p, int k) {
    const double2 v = sm[dr_at(k)];
    if constexpr (BLUE) return cmul(cswap(v), __ldg(p.chirp + k));
    return v;
}
/** Stores v as element i of the DFT's input. */
template <bool BLUE>
__device__ __forceinline__ void dr_in(double2* sm, const DirectPlan& p, int i, double2 v) {
    if constexpr (BLUE) v = cmul(v, __ldg(p.chirp + i));
    sm[dr_at(i)] = v;
}
template <bool BLUE>
__device__ __forceinline__ void dr_pad(double2* sm, const DirectPlan& p) {
    if constexpr (BLUE)
        for (int i = p.len + threadIdx.x; i < (1 << p.logp); i += blockDim.x) sm[dr_at(i)] = make_double2(0, 0);
}

/** V-cycles that the exact solve stands for in the caller's count and cap:
 * the decades the residual has to fall over those a V-cycle gains. */
__device__ __forceinline__ int dr_equivalent(const SolveCtl* ctl, double r2, double decades) {
    const double d = 0.5 * log10(r2 / (ctl->rtol * ctl->rtol * ctl->bnorm2));
    return max(1, int(ceil(fmin(d, 1e6) / decades)));
}

/** Residual of rows 2B and 2B + 1 (block B), their norms, and the rows'
 * modal source into p.work. The last block makes the first decision of the
 * solve (a zero source zeroes z) and sets ctl->direct when the exact solve
 * is to run: the count it stands for lies within the V-cycle cap. */
template <int MAXT, class OP, bool BLUE>
__global__ void __launch_bounds__(MAXT) dr_forward_k(OP c, DirectPlan p, double* __restrict__ z,
                                                    const double* __restrict__ b, Reduce rd, SolveCtl* ctl,
                                                    double decades, int use_cond, cudaGraphConditionalHandle h) {
    constexpr bool NODE = std::is_same<OP, FEMc<double>>::value;
    extern __shared__ __align__(16) unsigned char dr_raw[];
    __shared__ int zero_src;
    double2* sm = reinterpret_cast<double2*>(dr_raw);
    const int m = p.m, n = p.n, ja = 2 * blockIdx.x, jb = ja + 1;
    const bool two = jb < n;
    double sb = 0, sr = 0;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const long ka = long(ja) * m + i;
        const double ba = b[ka];
        double ra = op_resid(c, z + ka, ba, m, i, ja), rb = 0;
        sb += ba * ba;
        sr += ra * ra;
        if (two) {
            const double bb = b[ka + m];
            rb = op_resid(c, z + ka + m, bb, m, i, jb);
            sb += bb * bb;
            sr += rb * rb;
        }
        if (NODE && ja == 0) ra *= p.row0;
        if constexpr (NODE) {
            const bool end = i == 0 || i == m - 1;
            const double2 v = end ? make_double2(ra, rb) : make_double2(0.5 * ra, 0.5 * rb);
            dr_in<BLUE>(sm, p, i, v);
            if (!end) dr_in<BLUE>(sm, p, 2 * (m - 1) - i, v);
        } else {
            dr_in<BLUE>(sm, p, (i & 1) ? m - 1 - (i >> 1) : (i >> 1), make_double2(ra, rb));
        }
    }
    dr_pad<BLUE>(sm, p);
    dr_dft<BLUE>(sm, p);
    double* wa = p.work + long(ja) * m;
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        const double s = __ldg(p.norm + k);
        double xa, xb;
        const double2 zk = dr_out<BLUE>(sm, p, k);
        if constexpr (NODE) {
            xa = zk.x;
            xb = zk.y;
        } else {
            // the two rows' spectra from the packed one, then the quarter-
            // sample shift of the even-odd reordering
            const double2 zm = dr_out<BLUE>(sm, p, k ? m - k : 0), w = __ldg(p.post + k);
            xa = 0.5 * (w.x * (zk.x + zm.x) + w.y * (zk.y - zm.y));
            xb = 0.5 * (w.x * (zk.y + zm.y) + w.y * (zm.x - zk.x));
        }
        wa[k] = xa * s;
        if (two) wa[m + k] = xb * s;
    }
    sb = block_sum(sb);
    __syncthreads();
    sr = block_sum(sr);
    double b2, r2;
    if (!grid_sum2(sb, sr, rd, &b2, &r2)) return;
    if (threadIdx.x == 0) {
        ctl->bnorm2 = b2;
        ctl->it = 0;
        ctl->done = 0;
        ctl->status = 0;
        ctl->direct = 0;
        ctl->polish = 0;
        solve_decide(ctl, b2 == 0. ? 0. : r2, 0, use_cond, h);
        if (!ctl->done) {
            // below the cap, so that a V-cycle may follow
            const int e = dr_equivalent(ctl, r2, decades);
            if (e < ctl->max_it) ctl->direct = e;
        }
        zero_src = b2 == 0.;
    }
    __syncthreads();
    if (zero_src)
        for (long k = threadIdx.x; k < long(m) * n; k += blockDim.x) z[k] = 0.;
}

/** The tridiagonal systems of C modes over all rows, in place in
 * p.work. A thread holds one mode's rows of one chunk in registers: the
 * chunk's interior is eliminated with precomputed factors, the chunks' last
 * rows (the separators) form a small tridiagonal system that one thread per
 * mode solves in shared memory, and each thread then corrects its interior
 * for its two separators. One read and one write of the modal array, and a
 * serial chain of 2 L + 2 S steps instead of 2 R. */
template <int L, int C>
__global__ void __launch_bounds__(512) dr_modal_k(DirectPlan p, const SolveCtl* ctl) {
    if (!ctl->direct) return;
    __shared__ double sg[512 / C][C], sl[512 / C][C], sc[512 / C][C];
    const int c = threadIdx.x % C, s = threadIdx.x / C, k = blockIdx.x * C + c, m = p.m;
    const bool on = k < m;
    const int kk = on ? k : 0;
    const int S = p.S, len = min(L, p.R - s * L), ni = len - 1;
    const int kind = s == 0 ? 0 : (s == S - 1 ? 2 : 1);
    double* w = p.work + long(p.j0 + s * L) * m + kk;
    const double o = p.off[kk];
    const double* inv = p.inv + long(kind) * L * m + kk;
    double y[L];
#pragma unroll
    for (int i = 0; i < L; i++) y[i] = i < len ? w[long(i) * m] : 0.;
    if (p.j0 && s == 0) y[0] -= o * p.work[kk];
    double ds = y[0];
#pragma unroll
    for (int i = 1; i < L; i++)
        if (i == ni) ds = y[i];
    double yl = 0;
    if (ni > 0) {
        y[0] *= inv[0];
        yl = y[0];
    }
#pragma unroll
    for (int i = 1; i < L; i++)
        if (i < ni) {
            y[i] = (y[i] - o * y[i - 1]) * inv[long(i) * m];
            yl = y[i];
        }
#pragma unroll
    for (int i = L - 2; i >= 0; i--)
        if (i < ni - 1) y[i] -= o * inv[long(i) * m] * y[i + 1];
    sg[s][c] = ni > 0 ? y[0] : 0.;
    __syncthreads();
    const double yn = s < S - 1 ? sg[s + 1][c] : 0.;
    __syncthreads();
    {
        const long q = long(s) * m + kk;
        sg[s][c] = (ds - o * (ni > 0 ? yl : 0.) - o * yn) * p.ri[q];
        sl[s][c] = p.rl[q];
        sc[s][c] = p.rc[q];
    }
    __syncthreads();
    if (threadIdx.x < C) {
        double g = sg[0][c];
#pragma unroll 4
        for (int q = 1; q < S; q++) {
            g = sg[q][c] - sl[q][c] * g;
            sg[q][c] = g;
        }
#pragma unroll 4
        for (int q = S - 2; q >= 0; q--) {
            g = sg[q][c] - sc[q][c] * g;
            sg[q][c] = g;
        }
    }
    __syncthreads();
    if (!on) return;
    const double xs = sg[s][c], xp = s > 0 ? sg[s - 1][c] : 0.;
    const double* P = p.pp + long(kind) * L * m + kk;
    const double* Q = p.qq + long(kind) * L * m + kk;
#pragma unroll
    for (int i = 0; i < L; i++) {
        if (i < ni) w[long(i) * m] = y[i] - P[long(i) * m] * xp - Q[long(i) * m] * xs;
        else if (i == ni) w[long(i) * m] = xs;
    }
}

/** z += the modal array transformed back, rows 2B and 2B + 1. */
template <int MAXT, bool NODE, bool BLUE>
__global__ void __launch_bounds__(MAXT) dr_inverse_k(DirectPlan p, double* __restrict__ z, const SolveCtl* ctl) {
    if (!ctl->direct) return;
    extern __shared__ __align__(16) unsigned char dr_raw[];
    double2* sm = reinterpret_cast<double2*>(dr_raw);
    const int m = p.m, ja = 2 * blockIdx.x;
    const bool two = ja + 1 < p.n;
    const double* wa = p.work + long(ja) * m;
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        const double a = wa[k], b = two ? wa[m + k] : 0.;
        if constexpr (NODE) {
            const bool end = k == 0 || k == m - 1;
            const double2 v = end ? make_double2(a, b) : make_double2(0.5 * a, 0.5 * b);
            dr_in<BLUE>(sm, p, k, v);
            if (!end) dr_in<BLUE>(sm, p, 2 * (m - 1) - k, v);
        } else {
            // the packed spectrum of the reordered rows, stored swapped: the
            // inverse DFT is the swapped forward DFT
            const double f = k ? 0.5 : 1.;
            const double am = k ? 0.5 * wa[m - k] : 0., bm = k && two ? 0.5 * wa[2 * m - k] : 0.;
            const double2 w = __ldg(p.post + k);
            const double ar = w.x * (f * a) + w.y * am, ai = w.y * (f * a) - w.x * am;
            const double br = w.x * (f * b) + w.y * bm, bi = w.y * (f * b) - w.x * bm;
            dr_in<BLUE>(sm, p, k, make_double2(ai + br, ar - bi));
        }
    }
    dr_pad<BLUE>(sm, p);
    dr_dft<BLUE>(sm, p);
    double* za = z + long(ja) * m;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        double2 v;
        if constexpr (NODE) v = dr_out<BLUE>(sm, p, i);
        else v = cswap(dr_out<BLUE>(sm, p, (i & 1) ? m - 1 - (i >> 1) : (i >> 1)));
        za[i] += v.x;
        if (two) za[m + i] += v.y;
    }
}

/** ||b - A z||^2 after the exact solve and the decision, counting it. With
 * polish, a residual above the tolerance asks for the sweep of dr_relax_k. */
template <class OP>
__global__ void dr_check_k(OP c, const double* __restrict__ z, const double* __restrict__ b, Reduce rd, SolveCtl* ctl,
                           int polish, int use_cond, cudaGraphConditionalHandle h) {
    if (!ctl->direct) return;
    double s = 0;
    strip_walk(op_m(c), op_n(c), [&](long k, int i, int j) {
        const double r = op_resid(c, z + k, b[k], op_m(c), i, j);
        s += r * r;
    });
    s = block_sum(s);
    double total;
    if (grid_sum(s, rd, &total) && threadIdx.x == 0) {
        ctl->it += ctl->direct;
        ctl->direct_solves += 1;
        ctl->direct_cycles += ctl->direct;
        ctl->direct = 0;
        solve_decide(ctl, total, 0, use_cond, h);
        ctl->polish = polish && !ctl->done;
    }
}

/** One colour of a Gauss-Seidel sweep on a cell-centred level, in place:
 * what the exact solve leaves of a residual is the rounding of z at the
 * scale of the grid, which one sweep removes. Every row is walked by the
 * cells of one colour; 24 bytes a cell. */
__global__ void __launch_bounds__(256) dr_relax_k(CCc<double> c, double* __restrict__ z, const double* __restrict__ b,
                                                  const SolveCtl* ctl, int color) {
    if (!ctl->polish) return;
    const int m = c.m, h = (m + 1) >> 1;
    const long tot = long(h) * c.n;
    for (long q = blockIdx.x * long(blockDim.x) + threadIdx.x; q < tot; q += long(gridDim.x) * blockDim.x) {
        const int j = int(q / h), i = 2 * int(q - long(j) * h) + ((color + j) & 1);
        if (i >= m) continue;
        const long k = long(j) * m + i;
        z[k] = op_relaxed(c, z + k, b[k], m, i, j);
    }
}

/** The residual norm after that sweep, and the decision; v is the condition
 * of the V-cycle that follows in a captured loop. Without a sweep the V-cycle
 * follows at once. */
__global__ void dr_polish_check_k(CCc<double> c, const double* __restrict__ z, const double* __restrict__ b, Reduce rd,
                                  SolveCtl* ctl, int use_cond, cudaGraphConditionalHandle h,
                                  cudaGraphConditionalHandle v) {
    if (!ctl->polish) {
        if (use_cond && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(v, 1);
        return;
    }
    double s = 0;
    strip_walk(c.m, c.n, [&](long k, int i, int j) {
        const double r = op_resid(c, z + k, b[k], c.m, i, j);
        s += r * r;
    });
    s = block_sum(s);
    double total;
    if (grid_sum(s, rd, &total) && threadIdx.x == 0) {
        ctl->polish = 0;
        solve_decide(ctl, total, 0, use_cond, h);
        if (use_cond) cudaGraphSetConditional(v, !ctl->done);
    }
}

/** The modal systems' tables, one thread a mode: per chunk kind the inverse
 * pivots of the interior and the interior's response to its two separators
 * (times the off-diagonal), then the eliminated separators' system. */
__global__ void dr_tables_k(DirectPlan p, const double* __restrict__ di, const double* __restrict__ d0,
                            const double* __restrict__ dt, bool pin0, double* inv, double* pp, double* qq, double* ri,
                            double* rl, double* rc) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= p.m) return;
    const long ml = p.m;
    const int L = p.L, S = p.S, last = p.R - (S - 1) * L;
    const double o = p.off[k];
    double pl[3], pf[3], ql[3], qf[3];
    for (int kind = 0; kind < 3; kind++) {
        const int ni = ((kind == 2 || S == 1) ? last : L) - 1;
        const long base = long(kind) * L * ml + k;
        pl[kind] = pf[kind] = ql[kind] = qf[kind] = 0;
        double iv = 0;
        for (int i = 0; i < ni; i++) {
            const double d = kind == 0 && i == 0 ? d0[k] : di[k];
            iv = 1.0 / (i ? d - o * o * iv : d);
            inv[base + i * ml] = iv;
        }
        for (int side = 0; side < 2 && ni > 0; side++) {
            double* t = side == 0 ? pp : qq;
            double x = 0;
            for (int i = 0; i < ni; i++) {
                const double src = side == 0 ? (i == 0 ? 1. : 0.) : (i == ni - 1 ? 1. : 0.);
                x = (src - (i ? o * x : 0.)) * inv[base + i * ml];
                t[base + i * ml] = x;
            }
            (side == 0 ? pl : ql)[kind] = o * x;
            for (int i = ni - 2; i >= 0; i--) {
                x = t[base + i * ml] - o * inv[base + i * ml] * x;
                t[base + i * ml] = x;
            }
            (side == 0 ? pf : qf)[kind] = o * x;
            for (int i = 0; i < ni; i++) t[base + i * ml] *= (side == 0 && kind == 0) ? 0. : o;
        }
    }
    double cp = 0;
    for (int s = 0; s < S; s++) {
        const int kind = s == 0 ? 0 : (s == S - 1 ? 2 : 1), ni = (s == S - 1 ? last : L) - 1;
        double d = s == S - 1 ? dt[k] : di[k], lo = 0, up = 0;
        if (ni > 0) d -= o * ql[kind];
        if (s > 0) lo = ni > 0 ? -o * pl[kind] : o;
        if (s < S - 1) {
            const int kn = s + 1 == S - 1 ? 2 : 1, nn = (s + 1 == S - 1 ? last : L) - 1;
            if (nn > 0) d -= o * pf[kn];
            up = nn > 0 ? -o * qf[kn] : o;
        }
        double r = 1.0 / (d - lo * cp);
        if (pin0 && k == 0 && s == S - 1) r = 0;
        ri[long(s) * ml + k] = r;
        rl[long(s) * ml + k] = lo * r;
        cp = up * r;
        rc[long(s) * ml + k] = cp;
    }
}

// -------------------------------------------------------------------- host
/** exp(-2 pi i k / n), the angle reduced to an octant in integers. */
static double2 dr_unit(long k, long n) {
    k %= n;
    if (k < 0) k += n;
    // octant o and the remainder r / n of it; odd octants are measured back
    // from their end, so that t stays below pi / 4
    const long o = 8 * k / n, r = 8 * k - o * n;
    const double t = 0.78539816339744830962 * ((o & 1) ? double(n - r) / double(n) : double(r) / double(n));
    double c = std::cos(t), s = std::sin(t);
    double x, y;
    switch (o) {
        case 0: x = c; y = s; break;
        case 1: x = s; y = c; break;
        case 2: x = -s; y = c; break;
        case 3: x = -c; y = s; break;
        case 4: x = -c; y = -s; break;
        case 5: x = -s; y = -c; break;
        case 6: x = s; y = -c; break;
        default: x = c; y = -s; break;
    }
    return make_double2(x, -y);
}

/** Forward DFT of a power-of-two length on the host. */
static void dr_host_fft(std::vector<double2>& v) {
    const long n = long(v.size());
    for (long i = 1, j = 0; i < n; i++) {
        long bit = n >> 1;
        for (; j & bit; bit >>= 1) j ^= bit;
        j ^= bit;
        if (i < j) std::swap(v[i], v[j]);
    }
    std::vector<double2> w(n / 2 > 0 ? n / 2 : 1);
    for (long k = 0; k < n / 2; k++) w[k] = dr_unit(k, n);
    for (long len = 2; len <= n; len <<= 1)
        for (long i = 0; i < n; i += len)
            for (long k = 0; k < len / 2; k++) {
                const double2 a = v[i + k], b = v[i + k + len / 2], t = w[k * (n / len)];
                const double2 q = make_double2(b.x * t.x - b.y * t.y, b.x * t.y + b.y * t.x);
                v[i + k] = make_double2(a.x + q.x, a.y + q.y);
                v[i + k + len / 2] = make_double2(a.x - q.x, a.y - q.y);
            }
}

/** The modes' tridiagonal systems: off-diagonal, interior diagonal and the
 * diagonals of the first and last row. */
struct DirectModes {
    std::vector<double> off, di, d0, dt;
    bool pin0 = false;   // mode 0 is singular (constants): its last value is set to zero
};

/** Sizes of a plan for an m x n level; false where the grid is left to the
 * V-cycles (header comment). Chunks of 8 rows up to 512, 16 up to 2048: the
 * serial chain is 2 L + 2 S steps. A block takes 8 modes (64-byte segments
 * of a row) while its S threads a mode stay within 512, then 4. */
static bool dr_sizes(int m, int n, bool node, DirectPlan& p, bool& blue) {
    const int N = node ? m - 1 : m;
    if (N < 8 || n < (node ? 3 : 2)) return false;
    p.m = m;
    p.n = n;
    p.len = node ? 2 * N : N;
    blue = (N & (N - 1)) != 0;
    const long need = blue ? (node ? 3L * N : 2L * N - 1) : long(p.len);
    p.logp = 3;
    while ((1L << p.logp) < need) p.logp++;
    if ((1L << p.logp) > DR_MAX_P) return false;
    p.j0 = node ? 1 : 0;
    p.R = n - p.j0;
    p.L = p.R <= 512 ? 8 : (p.R <= 2048 ? 16 : 32);
    p.S = (p.R + p.L - 1) / p.L;
    p.modes = p.S <= 64 ? 8 : 4;
    return p.R <= DR_MAX_ROWS && p.S <= DR_MAX_CHUNKS;
}

/** Builds the plan's tables on the host and uploads them in one allocation
 * (*arena, freed by the caller); p holds dr_sizes' result. */
static int dr_build(DirectPlan& p, bool node, bool blue, const DirectModes& M, void** arena) {
    const int m = p.m, L = p.L, S = p.S;
    const long P = 1L << p.logp, ml = m;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~size_t(255);
        return o;
    };
    const size_t o_tw = take(P * 16), o_post = take(ml * 16), o_norm = take(ml * 8),
                 o_chirp = take(blue ? size_t(p.len) * 16 : 0), o_bhat = take(blue ? P * 16 : 0), o_off = take(ml * 8),
                 o_di = take(ml * 8), o_d0 = take(ml * 8), o_dt = take(ml * 8), from_host = off,
                 o_inv = take(3 * L * ml * 8), o_pp = take(3 * L * ml * 8), o_qq = take(3 * L * ml * 8),
                 o_ri = take(S * ml * 8), o_rl = take(S * ml * 8), o_rc = take(S * ml * 8);
    std::vector<unsigned char> host(from_host, 0);
    auto d2 = [&](size_t o) { return reinterpret_cast<double2*>(host.data() + o); };
    auto d1 = [&](size_t o) { return reinterpret_cast<double*>(host.data() + o); };
    for (long k = 0; k < P; k++) d2(o_tw)[k] = dr_unit(k, P);
    const int N = node ? m - 1 : m;
    for (int k = 0; k < m; k++) {
        const double2 u = dr_unit(k, 4L * m);   // exp(-i pi k / 2m)
        d2(o_post)[k] = make_double2(u.x, -u.y);
        const bool half = node ? (k == 0 || k == N) : k == 0;
        d1(o_norm)[k] = (half ? 1.0 : 2.0) / N;
        d1(o_off)[k] = M.off[k];
        d1(o_di)[k] = M.di[k];
        d1(o_d0)[k] = M.d0[k];
        d1(o_dt)[k] = M.dt[k];
    }
    if (blue) {
        const long len = p.len;
        std::vector<double2> q(P, make_double2(0, 0));
        for (long k = 0; k < len; k++) {
            const double2 u = dr_unit((k * k) % (2 * len), 2 * len);   // exp(-pi i k^2 / len)
            d2(o_chirp)[k] = u;
            const double2 cj = make_double2(u.x / P, -u.y / P);
            // the convolution's kernel at distances -(len-1) .. (outputs - 1)
            if (k < (node ? N + 1 : len)) q[k] = cj;
            if (k > 0) q[P - k] = cj;
        }
        dr_host_fft(q);
        std::copy(q.begin(), q.end(), d2(o_bhat));
    }
    unsigned char* dev = nullptr;
    VDI_CUDA(cudaMalloc(&dev, off + size_t(p.n) * m * 8));
    *arena = dev;
    VDI_CUDA(cudaMemcpy(dev, host.data(), from_host, cudaMemcpyHostToDevice));
    auto g2 = [&](size_t o) { return reinterpret_cast<const double2*>(dev + o); };
    auto g1 = [&](size_t o) { return reinterpret_cast<const double*>(dev + o); };
    p.tw = g2(o_tw);
    p.post = g2(o_post);
    p.norm = g1(o_norm);
    p.chirp = g2(o_chirp);
    p.bhat = g2(o_bhat);
    p.off = g1(o_off);
    p.inv = g1(o_inv);
    p.pp = g1(o_pp);
    p.qq = g1(o_qq);
    p.ri = g1(o_ri);
    p.rl = g1(o_rl);
    p.rc = g1(o_rc);
    p.work = reinterpret_cast<double*>(dev + off);
    auto w1 = [&](size_t o) { return reinterpret_cast<double*>(dev + o); };
    dr_tables_k<<<(m + 31) / 32, 32>>>(p, g1(o_di), g1(o_d0), g1(o_dt), M.pin0, w1(o_inv), w1(o_pp), w1(o_qq), w1(o_ri),
                                       w1(o_rl), w1(o_rc));
    VDI_CUDA(cudaGetLastError());
    VDI_CUDA(cudaDeviceSynchronize());
    return VDI_OK;
}

static int dr_threads(const DirectPlan& p) { return std::max(32, (1 << p.logp) >> 3); }
static size_t dr_smem(const DirectPlan& p) { return size_t((1 << p.logp) + ((1 << p.logp) >> 3)) * sizeof(double2); }

/** Raises the dynamic shared-memory limit of a plan's transform kernels. */
template <int MAXT, class OP, bool BLUE>
static cudaError_t dr_attr(size_t bytes) {
    constexpr bool NODE = std::is_same<OP, FEMc<double>>::value;
    cudaError_t e = cudaFuncSetAttribute(dr_forward_k<MAXT, OP, BLUE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(bytes));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(dr_inverse_k<MAXT, NODE, BLUE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(bytes));
    return e;
}

/** Calls f(MAXT, BLUE) as integral constants for the plan's block size. */
template <class F>
static auto dr_select(const DirectPlan& p, bool blue, F f) {
    using I512 = std::integral_constant<int, 512>;
    using I1024 = std::integral_constant<int, 1024>;
    if (dr_threads(p) <= 512) return blue ? f(I512{}, std::true_type{}) : f(I512{}, std::false_type{});
    return blue ? f(I1024{}, std::true_type{}) : f(I1024{}, std::false_type{});
}

/** The largest padding of any plan, so that one attribute call serves all. */
template <class OP>
static cudaError_t dr_prepare(const DirectPlan& p, bool blue) {
    return dr_select(p, blue, [&](auto t, auto bl) {
        constexpr int MAXT = decltype(t)::value;
        return dr_attr<MAXT, OP, decltype(bl)::value>(size_t(MAXT) * 9 * sizeof(double2));
    });
}

/** The start of a solve with the exact solve behind it (header comment). */
template <class OP>
static int dr_enqueue(cudaStream_t s, const OP& c, const DirectPlan& p, bool blue, double decades, double* z,
                      const double* b, const Reduce& rd, SolveCtl* ctl, int nb, int use_cond,
                      cudaGraphConditionalHandle h) {
    constexpr bool NODE = std::is_same<OP, FEMc<double>>::value;
    const int pairs = (p.n + 1) / 2, T = dr_threads(p);
    const size_t bytes = dr_smem(p);
    dr_select(p, blue, [&](auto t, auto bl) {
        dr_forward_k<decltype(t)::value, OP, decltype(bl)::value><<<pairs, T, bytes, s>>>(c, p, z, b, rd, ctl, decades,
                                                                                         use_cond, h);
        return 0;
    });
    const int mb = (p.m + p.modes - 1) / p.modes, mt = p.modes * p.S;
    if (p.L == 8) dr_modal_k<8, 8><<<mb, mt, 0, s>>>(p, ctl);
    else if (p.L == 32) dr_modal_k<32, 4><<<mb, mt, 0, s>>>(p, ctl);
    else if (p.modes == 8) dr_modal_k<16, 8><<<mb, mt, 0, s>>>(p, ctl);
    else dr_modal_k<16, 4><<<mb, mt, 0, s>>>(p, ctl);
    dr_select(p, blue, [&](auto t, auto bl) {
        dr_inverse_k<decltype(t)::value, NODE, decltype(bl)::value><<<pairs, T, bytes, s>>>(p, z, ctl);
        return 0;
    });
    dr_check_k<<<nb, 256, 0, s>>>(c, z, b, rd, ctl, !NODE, use_cond, h);
    VDI_CUDA(cudaGetLastError());
    return VDI_OK;
}
