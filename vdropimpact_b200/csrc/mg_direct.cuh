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
// at 2048 x 1024, 23 us at the measured copy rate. The transforms are bound
// by what a block waits for (its rows, the passes through shared memory and
// the barriers between them, about 12 us for a block alone) and by how many
// blocks an SM holds; hence loads in batches ahead of their use, twiddles
// fetched before the barrier they follow, and the chunks' separators by
// parallel reduction. Launches at 2048 x 1024 (MAC), warm: forward 25 us,
// modal 20, inverse 16, check 13; 8, 5, 4 and 7 us at 256 x 128; FEM 2049 x
// 1025 40, 21, 28 and 18. Without these measures 26, 23, 18 and 12; 14, 6, 8
// and 10; 42, 25, 30 and 17. Whole calls of vdi_mg_solve from zero to 1e-10,
// the V-cycles against this path: MAC 64 x 32 318 and 55 us, 1000 x 500 5080
// and 82 us, 2048 x 1024 1000 and 129 us (with the sweep of dr_relax_k), FEM
// 1025 x 513 441 and 78 us.

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
    bool pin0 = false;         // mode 0 is singular: solved with its last value zero, then made mean-free
    const double2* tw = nullptr;     // exp(-2 pi i k / P)
    const double2* post = nullptr;   // cells: (cos, sin)(pi k / 2m)
    double norm = 0;                 // 1 / C_k, twice that of the first (nodes: and last) mode
    const double2* chirp = nullptr;  // exp(-pi i k^2 / len)
    const double2* bhat = nullptr;   // transform of the conjugate chirp over P
    const double* off = nullptr;     // [m] off-diagonal of mode k
    // per chunk kind (0 first, 1 middle, 2 last), row of the chunk and mode
    const double *inv = nullptr, *pp = nullptr, *qq = nullptr;
    // per chunk and mode: the separators' system, its couplings and the
    // excess of its diagonal over them, relative to the diagonal, and the
    // inverse diagonal
    const double *ra = nullptr, *rc = nullptr, *rs = nullptr, *ri = nullptr;
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
    // the next pass's twiddles are fetched before the barriers of this one
    double2 w1, w2, w4;
    auto twiddle = [&](int lns) {
        const int k = t & ((1 << lns) - 1), st = logp - 3 - lns;
        if (on && lns < logp) {
            w1 = __ldg(tw + (k << st));
            w2 = __ldg(tw + (2 * k << st));
            w4 = __ldg(tw + (4 * k << st));
        }
    };
    int lns = rem == 0 ? 3 : rem;
    twiddle(lns);
    __syncthreads();
    // from 64 points on, equal steps between a thread's elements are equal
    // steps in padded memory: one address and multiples of a stride
    const bool big = logp >= 6;
    const int st0 = n8 + (n8 >> 3);
    double2* const s0 = sm + dr_at(t);
    if (on) {
        if (big) {
#pragma unroll
            for (int q = 0; q < 8; q++) v[q] = s0[q * st0];
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++) v[q] = sm[dr_at(t + q * n8)];
        }
    }
    __syncthreads();
    if (rem == 0) {
        if (on) {
            dft8(v);
#pragma unroll
            for (int r = 0; r < 8; r++) sm[9 * t + r] = v[r];
        }
    } else if (rem == 1) {
        if (on) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                dft2(v[u], v[u + 4]);
                sm[dr_at(2 * (t + u * n8))] = v[u];
                sm[dr_at(2 * (t + u * n8) + 1)] = v[u + 4];
            }
        }
    } else {
        if (on) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                dft4(v[u], v[u + 2], v[u + 4], v[u + 6]);
#pragma unroll
                for (int r = 0; r < 4; r++) sm[dr_at(4 * (t + u * n8) + r)] = v[u + 2 * r];
            }
        }
    }
    for (; lns < logp; lns += 3) {
        const int ns = 1 << lns, k = t & (ns - 1);
        __syncthreads();
        if (on) {
            if (big) {
#pragma unroll
                for (int q = 0; q < 8; q++) v[q] = s0[q * st0];
            } else {
#pragma unroll
                for (int q = 0; q < 8; q++) v[q] = sm[dr_at(t + q * n8)];
            }
            v[1] = cmul(v[1], w1);
            v[2] = cmul(v[2], w2);
            v[4] = cmul(v[4], w4);
            v[3] = cmul(v[3], cmul(w1, w2));
            v[5] = cmul(v[5], cmul(w1, w4));
            const double2 w6 = cmul(w2, w4);
            v[6] = cmul(v[6], w6);
            v[7] = cmul(v[7], cmul(w1, w6));
            twiddle(lns + 3);
            dft8(v);
        }
        __syncthreads();
        if (on) {
            const int o = ((t - k) << 3) + k;
            if (lns >= 3) {
                double2* const d = sm + dr_at(o);
                const int ds = ns + (ns >> 3);
#pragma unroll
                for (int r = 0; r < 8; r++) d[r * ds] = v[r];
            } else {
#pragma unroll
                for (int r = 0; r < 8; r++) sm[dr_at(o + r * ns)] = v[r];
            }
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

/** Sums of two values over the block, valid in thread 0. */
__device__ void dr_block_sum2(double& a, double& b) {
    __shared__ double ws[2][32];
    a = warp_sum(a);
    b = warp_sum(b);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        ws[0][w] = a;
        ws[1][w] = b;
    }
    __syncthreads();
    if (w == 0) {
        const bool in = lane < int(blockDim.x >> 5);
        a = warp_sum(in ? ws[0][lane] : 0.);
        b = warp_sum(in ? ws[1][lane] : 0.);
    }
}

/** V-cycles that the exact solve stands for in the caller's count: the
 * decades the residual has to fall over those a V-cycle gains. 0 where they,
 * one V-cycle more, and those for the decades beyond the 14 that rounding
 * lets the exact solve gain, at 0.8 each, are not all within the cap: V-cycles
 * alone may then meet a cap that they do not meet behind it. */
__device__ __forceinline__ int dr_equivalent(const SolveCtl* ctl, double r2, double decades) {
    const double d = fmin(0.5 * log10(r2 / (ctl->rtol * ctl->rtol * ctl->bnorm2)), 1e6);
    const int e = max(1, int(ceil(d / decades)));
    const int more = d > 14 ? 1 + int(ceil((d - 14) / 0.8)) : 0;
    return e + more < ctl->max_it ? e : 0;
}

/** Blocks of the transform kernels an SM should hold: they are bound by the
 * latency of their passes and barriers, so registers are kept for that. */
constexpr int dr_min_blocks(int maxt) { return maxt == 256 ? 4 : (maxt == 512 ? 2 : 1); }

/** Residual of rows 2B and 2B + 1 (block B), their norms, and the rows'
 * modal source into p.work. The last block makes the first decision of the
 * solve (a zero source zeroes z) and sets ctl->direct when the exact solve
 * is to run (dr_equivalent). */
template <int MAXT, class OP, bool BLUE>
__global__ void __launch_bounds__(MAXT, dr_min_blocks(MAXT)) dr_forward_k(OP c, DirectPlan p, double* __restrict__ z,
                                                    const double* __restrict__ b, Reduce rd, SolveCtl* ctl,
                                                    double decades, int use_cond, cudaGraphConditionalHandle h) {
    constexpr bool NODE = std::is_same<OP, FEMc<double>>::value;
    extern __shared__ __align__(16) unsigned char dr_raw[];
    __shared__ int zero_src;
    double2* sm = reinterpret_cast<double2*>(dr_raw);
    const int m = p.m, n = p.n, ja = 2 * blockIdx.x, jb = ja + 1;
    const bool two = jb < n;
    double sb = 0, sr = 0;
    const double* zr = z + long(ja) * m;
    const double* br = b + long(ja) * m;
    const bool below = ja > 0, above = ja + 2 < n;
    // a batch of columns a thread at a time, every load of it before its use;
    // side neighbours by shuffle (a warp's columns are consecutive), the
    // warp's two outer ones loaded
    constexpr int BATCH = MAXT == 256 && !NODE ? 2 : 1;
    const int lane = threadIdx.x & 31;
    const int e = lane == 0 ? -1 : 1;
    for (int base = threadIdx.x & ~31; base < m; base += BATCH * blockDim.x) {
        double w[BATCH][4], we[BATCH][4], bv[BATCH][2];
#pragma unroll
        for (int u = 0; u < BATCH; u++) {
            const int i = base + u * blockDim.x + lane;
            const bool in = i < m, out = (lane == 0 || lane == 31) && i + e >= 0 && i + e < m;
#pragma unroll
            for (int d = 0; d < 4; d++) {
                const bool row = d == 0 ? below : (d == 1 ? true : (d == 2 ? two : above));
                const double* q = zr + long(d - 1) * m + i;
                w[u][d] = in && row ? q[0] : 0.;
                // the 5-point operator takes side neighbours on its own rows only
                if (NODE || d == 1 || d == 2) we[u][d] = out && row ? q[e] : 0.;
            }
            bv[u][0] = in ? br[i] : 0.;
            bv[u][1] = in && two ? br[m + i] : 0.;
        }
#pragma unroll
        for (int u = 0; u < BATCH; u++) {
            const int i = base + u * blockDim.x + lane;
            double l[4], r[4];
#pragma unroll
            for (int d = 0; d < 4; d++)
                if (NODE || d == 1 || d == 2) {
                    const double x = __shfl_up_sync(0xffffffffu, w[u][d], 1), y = __shfl_down_sync(0xffffffffu, w[u][d], 1);
                    l[d] = lane == 0 ? we[u][d] : x;
                    r[d] = lane == 31 ? we[u][d] : y;
                }
            if (i >= m) continue;
            double res[2];
#pragma unroll
            for (int d = 0; d < 2; d++) {
                double off;
                if constexpr (NODE)
                    off = fem_off_vals(c, i, ja + d, l[d], w[u][d], r[d], l[d + 1], r[d + 1], l[d + 2], w[u][d + 2],
                                       r[d + 2]);
                else
                    off = c.ox * (l[d + 1] + r[d + 1]) + c.oy * (w[u][d] + w[u][d + 2]);
                res[d] = bv[u][d] - pick3(c.d, cls(i, m), cls(ja + d, n)) * w[u][d + 1] - off;
                if (d == 1 && !two) res[d] = 0.;
                sb += bv[u][d] * bv[u][d];
                sr += res[d] * res[d];
            }
            if (NODE && ja == 0) res[0] *= p.row0;
            if constexpr (NODE) {
                const bool end = i == 0 || i == m - 1;
                const double2 v = end ? make_double2(res[0], res[1]) : make_double2(0.5 * res[0], 0.5 * res[1]);
                dr_in<BLUE>(sm, p, i, v);
                if (!end) dr_in<BLUE>(sm, p, 2 * (m - 1) - i, v);
            } else {
                dr_in<BLUE>(sm, p, (i & 1) ? m - 1 - (i >> 1) : (i >> 1), make_double2(res[0], res[1]));
            }
        }
    }
    dr_pad<BLUE>(sm, p);
    dr_dft<BLUE>(sm, p);
    double* wa = p.work + long(ja) * m;
    if constexpr (NODE) {
#pragma unroll 2
        for (int k = threadIdx.x; k < m; k += blockDim.x) {
            const double2 zk = dr_out<BLUE>(sm, p, k);
            const double s = k == 0 || k == m - 1 ? 0.5 * p.norm : p.norm;
            wa[k] = zk.x * s;
            if (two) wa[m + k] = zk.y * s;
        }
    } else {
        // modes k and m - k together: the two rows' spectra from the packed
        // one, then the quarter-sample shift of the even-odd reordering
        const double hs = 0.5 * p.norm;
#pragma unroll 4
        for (int k = threadIdx.x; k <= m / 2; k += blockDim.x) {
            const double2 w = __ldg(p.post + k);
            const double2 zk = dr_out<BLUE>(sm, p, k), zm = dr_out<BLUE>(sm, p, k ? m - k : 0);
            const double s = k ? hs : 0.5 * hs;
            const double ax = zk.x + zm.x, ay = zk.y - zm.y, bx = zk.y + zm.y, by = zm.x - zk.x;
            wa[k] = s * (w.x * ax + w.y * ay);
            if (two) wa[m + k] = s * (w.x * bx + w.y * by);
            if (k && 2 * k != m) {
                wa[m - k] = s * (w.y * ax - w.x * ay);
                if (two) wa[2 * m - k] = s * (w.y * bx - w.x * by);
            }
        }
    }
    dr_block_sum2(sb, sr);
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
        if (!ctl->done) ctl->direct = dr_equivalent(ctl, r2, decades);
        zero_src = b2 == 0.;
    }
    __syncthreads();
    if (zero_src)
        for (long k = threadIdx.x; k < long(m) * n; k += blockDim.x) z[k] = 0.;
}

/** The tridiagonal systems of C modes over all rows, in place in p.work. A
 * thread holds one mode's rows of one chunk in registers: the chunk's interior
 * is eliminated with precomputed factors, the chunks' last rows (the
 * separators) form a tridiagonal system with unit diagonals that is solved by
 * parallel cyclic reduction, one row a thread, and each thread then corrects
 * its interior for its two separators. One read and one write of the modal
 * array, and log2(S) barriers. (A serial solve of the separators by one
 * thread a mode took a third of the kernel.) */
template <int L, int C, int NT, bool PIN>
__global__ void __launch_bounds__(NT, L == 8 ? 2 : 1) dr_modal_k(DirectPlan p, const SolveCtl* ctl) {
    if (!ctl->direct) return;
    __shared__ double sx[2][4][NT];
    const int tid = threadIdx.x, c = tid % C, s = tid / C, k = blockIdx.x * C + c, m = p.m;
    const bool on = k < m;
    const int kk = on ? k : 0;
    const int S = p.S, len = min(L, p.R - s * L), ni = len - 1;
    const int kind = s == 0 ? 0 : (s == S - 1 ? 2 : 1);
    double* w = p.work + long(p.j0 + s * L) * m + kk;
    const double o = __ldg(p.off + kk);
    const double* inv = p.inv + long(kind) * L * m + kk;
    const long sq = long(s) * m + kk;
    double y[L];
#pragma unroll
    for (int i = 0; i < L; i++) y[i] = i < len ? w[long(i) * m] : 0.;
    double A = __ldg(p.ra + sq), Cc = __ldg(p.rc + sq), E = __ldg(p.rs + sq);
    const double ri = __ldg(p.ri + sq);
    if (p.j0 && s == 0) y[0] -= o * p.work[kk];
    double ds = y[0];
#pragma unroll
    for (int i = 1; i < L; i++)
        if (i == ni) ds = y[i];
    double yl = 0;
    if (ni > 0) {
        y[0] *= __ldg(inv);
        yl = y[0];
    }
#pragma unroll
    for (int i = 1; i < L; i++)
        if (i < ni) {
            y[i] = (y[i] - o * y[i - 1]) * __ldg(inv + long(i) * m);
            yl = y[i];
        }
#pragma unroll
    for (int i = L - 2; i >= 0; i--)
        if (i < ni - 1) y[i] -= o * __ldg(inv + long(i) * m) * y[i + 1];
    sx[0][0][tid] = ni > 0 ? y[0] : 0.;
    __syncthreads();
    const double yn = s < S - 1 ? sx[0][0][tid + C] : 0.;
    double D = (ds - o * (ni > 0 ? yl : 0.) - o * yn) * ri;
    int q = 1;
    for (int d = 1; d < S; d <<= 1, q ^= 1) {
        // the buffer of two steps ago, which every thread has read
        sx[q][0][tid] = A;
        sx[q][1][tid] = Cc;
        sx[q][2][tid] = D;
        sx[q][3][tid] = E;
        __syncthreads();
        const bool l = s >= d, r = s + d < S;
        const int tl = tid - d * C, tr = tid + d * C;
        const double Al = l ? sx[q][0][tl] : 0., Dl = l ? sx[q][2][tl] : 0., El = l ? sx[q][3][tl] : 0.;
        const double Cr = r ? sx[q][1][tr] : 0., Dr = r ? sx[q][2][tr] : 0., Er = r ? sx[q][3][tr] : 0.;
        // 1 - A Cl - Cc Ar with each 1 written as |A| + |C| + E: the sum of
        // positive terms keeps the slowest modes' small excess to its last bits
        const double ex = E + fabs(A) * El + fabs(Cc) * Er;
        const double rb = 1. / (ex + fabs(A * Al) + fabs(Cc * Cr));
        E = ex * rb;
        D = (D - A * Dl - Cc * Dr) * rb;
        A = -A * Al * rb;
        Cc = -Cc * Cr * rb;
    }
    sx[q][0][tid] = D;
    __syncthreads();
    if (!on) return;
    const double xp = s > 0 ? sx[q][0][tid - C] : 0.;
    const double* P = p.pp + long(kind) * L * m + kk;
    const double* Q = p.qq + long(kind) * L * m + kk;
#pragma unroll
    for (int i = 0; i < L; i++) {
        if (i < ni) y[i] -= __ldg(P + long(i) * m) * xp + __ldg(Q + long(i) * m) * D;
        else if (i == ni) y[i] = D;
    }
    if (PIN && blockIdx.x == 0) {
        // The pinned solution's mean is arbitrary, as large as z's error was:
        // added to z it would be rounded at that scale in every later V-cycle.
        // (m >= 8: the first block's threads all hold a mode. Tested at run
        // time for every system, this took 22.1 us of a launch in place of 20.3.)
        double t = 0;
#pragma unroll
        for (int i = 0; i < L; i++)
            if (i <= ni) t += y[i];
        sx[q][1][tid] = t;
        __syncthreads();
        if (c == 0) {
            double mean = 0;
            for (int r = 0; r < S; r++) mean += sx[q][1][r * C];
            mean /= p.R;
#pragma unroll
            for (int i = 0; i < L; i++) y[i] -= mean;
        }
    }
#pragma unroll
    for (int i = 0; i < L; i++)
        if (i <= ni) w[long(i) * m] = y[i];
}

/** z += the modal array transformed back, rows 2B and 2B + 1. */
template <int MAXT, bool NODE, bool BLUE>
__global__ void __launch_bounds__(MAXT, dr_min_blocks(MAXT)) dr_inverse_k(DirectPlan p, double* __restrict__ z, const SolveCtl* ctl) {
    if (!ctl->direct) return;
    extern __shared__ __align__(16) unsigned char dr_raw[];
    double2* sm = reinterpret_cast<double2*>(dr_raw);
    const int m = p.m, ja = 2 * blockIdx.x;
    const bool two = ja + 1 < p.n;
    const double* __restrict__ wa = p.work + long(ja) * m;
    if constexpr (NODE) {
#pragma unroll 4
        for (int k = threadIdx.x; k < m; k += blockDim.x) {
            const double a = wa[k], b = two ? wa[m + k] : 0.;
            const bool end = k == 0 || k == m - 1;
            const double2 v = end ? make_double2(a, b) : make_double2(0.5 * a, 0.5 * b);
            dr_in<BLUE>(sm, p, k, v);
            if (!end) dr_in<BLUE>(sm, p, 2 * (m - 1) - k, v);
        }
    } else {
        // modes k and m - k together: the packed spectrum of the reordered
        // rows, stored swapped (the inverse DFT is the swapped forward DFT)
#pragma unroll 4
        for (int k = threadIdx.x; k <= m / 2; k += blockDim.x) {
            const double a = wa[k], b = two ? wa[m + k] : 0.;
            const double am = k ? wa[m - k] : 0., bm = k && two ? wa[2 * m - k] : 0.;
            const double2 w = __ldg(p.post + k);
            const double f = k ? 0.5 : 1.;
            const double ar = f * (w.x * a + w.y * am), ai = f * (w.y * a - w.x * am);
            const double br = f * (w.x * b + w.y * bm), bi = f * (w.y * b - w.x * bm);
            dr_in<BLUE>(sm, p, k, make_double2(ai + br, ar - bi));
            if (k && 2 * k != m) dr_in<BLUE>(sm, p, m - k, make_double2(br - ai, ar + bi));
        }
    }
    dr_pad<BLUE>(sm, p);
    dr_dft<BLUE>(sm, p);
    // z's loads of a batch of columns before its stores
    constexpr int BATCH = MAXT == 256 ? 4 : 2;
    double* za = z + long(ja) * m;
    for (int i0 = threadIdx.x; i0 < m; i0 += BATCH * blockDim.x) {
        double x[BATCH][2];
#pragma unroll
        for (int u = 0; u < BATCH; u++) {
            const int i = i0 + u * blockDim.x;
            x[u][0] = i < m ? za[i] : 0.;
            x[u][1] = i < m && two ? za[m + i] : 0.;
        }
#pragma unroll
        for (int u = 0; u < BATCH; u++) {
            const int i = i0 + u * blockDim.x;
            if (i >= m) break;
            double2 v;
            if constexpr (NODE) v = dr_out<BLUE>(sm, p, i);
            else v = cswap(dr_out<BLUE>(sm, p, (i & 1) ? m - 1 - (i >> 1) : (i >> 1)));
            za[i] = x[u][0] + v.x;
            if (two) za[m + i] = x[u][1] + v.y;
        }
    }
}

/** Squared residuals of a level summed by warps over strips of 64 columns
 * and rows rows, two columns a lane. The rows of z slide through registers
 * (each is read once, side neighbours by shuffle) and DR_ROWS rows of z and b
 * are in flight at a time, 16 bytes a lane where vec (even m, aligned). */
static constexpr int DR_ROWS = 4;
template <class OP>
__device__ double dr_resid_sum(const OP& c, const double* __restrict__ z, const double* __restrict__ b, int rows,
                               bool vec) {
    constexpr bool NODE = std::is_same<OP, FEMc<double>>::value;
    const int m = op_m(c), n = op_n(c), lane = threadIdx.x & 31;
    const int sx = (m + 63) >> 6, ns = sx * ((n + rows - 1) / rows);
    double s = 0;
    for (int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); q < ns; q += gridDim.x * (blockDim.x >> 5)) {
        const int sj = q / sx, i0 = (q - sj * sx) * 64 + 2 * lane, i1 = i0 + 1;
        const int y0 = sj * rows, y1 = min(y0 + rows, n);
        const bool in0 = i0 < m, in1 = i1 < m;
        const int ie = lane == 0 ? i0 - 1 : i0 + 2;   // the strip's side neighbours
        const bool edge = (lane == 0 || lane == 31) && unsigned(ie) < unsigned(m);
        // the lane's columns on interior rows: diagonals, and the FEM's
        // vertical coupling, halved at the side ends
        double dg[2], fy[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int x = i0 + k < m ? cls(i0 + k, m) : 1;
            dg[k] = c.d[x][1];
            if constexpr (NODE) fy[k] = x == 1 ? c.fey : c.hey;
        }
        auto load = [&](const double* p, int j, double& a, double& d) {
            a = d = 0.;
            if (unsigned(j) >= unsigned(n)) return;
            const double* r = p + long(j) * m + i0;
            if (vec) {
                if (in0) {
                    const double2 v = *reinterpret_cast<const double2*>(r);
                    a = v.x;
                    d = v.y;
                }
            } else {
                if (in0) a = r[0];
                if (in1) d = r[1];
            }
        };
        // rows j - 1, j, j + 1: left, own two, right
        double w[DR_ROWS + 2][4];
        auto sides = [&](double (&r)[4], double e) {
            const double l = __shfl_up_sync(0xffffffffu, r[2], 1), t = __shfl_down_sync(0xffffffffu, r[1], 1);
            r[0] = lane == 0 ? e : l;
            r[3] = lane == 31 ? e : t;
        };
        auto side = [&](int j) { return edge && unsigned(j) < unsigned(n) ? z[long(j) * m + ie] : 0.; };
#pragma unroll
        for (int d = 0; d < 2; d++) {
            load(z, y0 - 1 + d, w[d][1], w[d][2]);
            sides(w[d], side(y0 - 1 + d));
        }
        for (int j = y0; j < y1; j += DR_ROWS) {
            double bv[DR_ROWS][2], e[DR_ROWS];
#pragma unroll
            for (int d = 0; d < DR_ROWS; d++) {
                load(z, j + d + 1, w[d + 2][1], w[d + 2][2]);
                e[d] = side(j + d + 1);
                load(b, j + d, bv[d][0], bv[d][1]);
            }
#pragma unroll
            for (int d = 0; d < DR_ROWS; d++) {
                sides(w[d + 2], e[d]);
                if (j + d < y1) {
                    const double(&dn)[4] = w[d], (&ce)[4] = w[d + 1], (&up)[4] = w[d + 2];
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        const int i = i0 + k;
                        double off, dv = dg[k];
                        if (unsigned(j + d - 1) >= unsigned(n - 2)) dv = c.d[i < m ? cls(i, m) : 1][cls(j + d, n)];
                        if constexpr (NODE) {
                            if (unsigned(j + d - 1) >= unsigned(n - 2))
                                off = fem_off_vals(c, i, j + d, dn[k], dn[k + 1], dn[k + 2], ce[k], ce[k + 2], up[k],
                                                   up[k + 1], up[k + 2]);
                            else
                                off = c.fc * (dn[k] + dn[k + 2] + up[k] + up[k + 2]) + fy[k] * (dn[k + 1] + up[k + 1]) +
                                      c.fex * (ce[k] + ce[k + 2]);
                        } else {
                            off = c.ox * (ce[k] + ce[k + 2]) + c.oy * (dn[k + 1] + up[k + 1]);
                        }
                        const double r = bv[d][k] - dv * ce[k + 1] - off;
                        if (k ? in1 : in0) s += r * r;
                    }
                }
            }
#pragma unroll
            for (int d = 0; d < 2; d++)
#pragma unroll
                for (int k = 0; k < 4; k++) w[d][k] = w[d + DR_ROWS][k];
        }
    }
    return s;
}

/** ||b - A z||^2 after the exact solve and the decision, counting it. With
 * polish, a residual above the tolerance asks for the sweep of dr_relax_k. */
template <class OP>
__global__ void __launch_bounds__(256, 3) dr_check_k(OP c, const double* __restrict__ z, const double* __restrict__ b,
                                                  int rows, int vec, Reduce rd, SolveCtl* ctl, int polish, int use_cond,
                                                  cudaGraphConditionalHandle h) {
    if (!ctl->direct) return;
    double s = dr_resid_sum(c, z, b, rows, vec);
    s = block_sum(s);
    double total;
    if (grid_sum(s, rd, &total) && threadIdx.x == 0) {
        ctl->it += ctl->direct;
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

static constexpr unsigned long long DR_POLISH_LAUNCHES = 3;   // the sweep's two colours and its check

/** The residual norm after that sweep, and the decision; v is the condition
 * of the V-cycle that follows in a captured loop. Without a sweep the V-cycle
 * follows at once. */
__global__ void __launch_bounds__(256, 3) dr_polish_check_k(CCc<double> c, const double* __restrict__ z,
                                                         const double* __restrict__ b, int rows, int vec, Reduce rd,
                                                         SolveCtl* ctl, int use_cond, cudaGraphConditionalHandle h,
                                                         cudaGraphConditionalHandle v) {
    if (!ctl->polish) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            atomicAdd(&ctl->more_launches, DR_POLISH_LAUNCHES);   // not waited for
            if (use_cond) cudaGraphSetConditional(v, 1);
        }
        return;
    }
    double s = dr_resid_sum(c, z, b, rows, vec);
    s = block_sum(s);
    double total;
    if (grid_sum(s, rd, &total) && threadIdx.x == 0) {
        ctl->polish = 0;
        atomicAdd(&ctl->more_launches, DR_POLISH_LAUNCHES);
        solve_decide(ctl, total, 0, use_cond, h);
        if (use_cond) cudaGraphSetConditional(v, !ctl->done);
    }
}

/** The modal systems' tables, one thread a mode: per chunk kind the inverse
 * pivots of the interior and the interior's response to its two separators
 * (times the off-diagonal), then the separators' system. Its diagonals are
 * sums of the couplings and of the rows' excess (ei, e0, et: how far a
 * diagonal exceeds its neighbours' coefficients), never differences: the
 * excess of the slowest modes is 1e-6 of the diagonal and less. */
__global__ void dr_tables_k(DirectPlan p, const double* __restrict__ di, const double* __restrict__ d0,
                            const double* __restrict__ ei, const double* __restrict__ e0,
                            const double* __restrict__ et, bool pin0, double* inv, double* pp, double* qq, double* ri,
                            double* ra, double* rc, double* rs) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= p.m) return;
    const long ml = p.m;
    const int L = p.L, S = p.S, last = p.R - (S - 1) * L;
    const double o = p.off[k];
    const double oa = fabs(o), sign = di[k] < 0 ? -1. : 1.;
    double pl[3], pf[3], ql[3], qf[3], xf[3], xl[3];   // xf, xl: the interior's excess seen by its separators
    for (int kind = 0; kind < 3; kind++) {
        const int ni = ((kind == 2 || S == 1) ? last : L) - 1;
        const long base = long(kind) * L * ml + k;
        pl[kind] = pf[kind] = ql[kind] = qf[kind] = xf[kind] = xl[kind] = 0;
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
        double up = 0, dn = 0;
        for (int i = 0; i < ni; i++) {
            up = (kind == 0 && i == 0 ? e0[k] : ei[k]) + oa * up;
            up *= fabs(inv[base + i * ml]);
        }
        // downwards the pivots are those of the rows above, by symmetry the
        // interior's own but for a first chunk, whose lower end has no separator
        for (int i = 0; i < ni; i++) dn = (ei[k] + oa * dn) * fabs(inv[base + i * ml]);
        xl[kind] = oa * up;
        if (kind) xf[kind] = oa * dn;
    }
    for (int s = 0; s < S; s++) {
        const int kind = s == 0 ? 0 : (s == S - 1 ? 2 : 1), ni = (s == S - 1 ? last : L) - 1;
        double lo = 0, up = 0, ex = (s == S - 1 ? et[k] : ei[k]) + xl[kind];
        if (s > 0) lo = ni > 0 ? -o * pl[kind] : o;
        if (s < S - 1) {
            const int kn = s + 1 == S - 1 ? 2 : 1, nn = (s + 1 == S - 1 ? last : L) - 1;
            ex += xf[kn];
            up = nn > 0 ? -o * qf[kn] : o;
        }
        // a pinned last separator is zero
        const double d = fabs(lo) + fabs(up) + ex;
        const bool pin = pin0 && k == 0 && s == S - 1;
        const double r = pin ? 0. : sign / d;
        ri[long(s) * ml + k] = r;
        ra[long(s) * ml + k] = lo * r;
        rc[long(s) * ml + k] = up * r;
        rs[long(s) * ml + k] = pin ? 1. : ex / d;
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

/** The modes' tridiagonal systems: off-diagonal, interior diagonal and that
 * of the first row, and the excess of an interior, the first and the last
 * row's diagonal over its neighbours' coefficients (magnitudes). */
struct DirectModes {
    std::vector<double> off, di, d0, ei, e0, et;
    bool pin0 = false;   // mode 0 is singular (constants): its last value is set to zero
};

/** Sizes of a plan for an m x n level; false where the grid is left to the
 * V-cycles (header comment). Chunks of 8 rows up to 1024, 16 up to 2048, 32
 * beyond: short chunks make short chains and hold few registers. A block takes
 * 8 modes (64-byte segments of a row) while that is at most 512 threads, then
 * 4 (one 32-byte sector). */
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
    p.L = p.R <= 1024 ? 8 : (p.R <= 2048 ? 16 : 32);
    p.S = (p.R + p.L - 1) / p.L;
    p.modes = p.L == 8 && p.S <= 64 ? 8 : 4;
    return p.R <= DR_MAX_ROWS && p.S <= DR_MAX_CHUNKS;
}

/** Builds the plan's tables on the host and uploads them in one allocation
 * (*arena, freed by the caller; null when the device has no room for it); p
 * holds dr_sizes' result. */
static int dr_build(DirectPlan& p, bool node, bool blue, const DirectModes& M, void** arena) {
    const int m = p.m, L = p.L, S = p.S;
    const long P = 1L << p.logp, ml = m;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~size_t(255);
        return o;
    };
    const size_t o_tw = take(P * 16), o_post = take(ml * 16),
                 o_chirp = take(blue ? size_t(p.len) * 16 : 0), o_bhat = take(blue ? P * 16 : 0), o_off = take(ml * 8),
                 o_di = take(ml * 8), o_d0 = take(ml * 8), o_ei = take(ml * 8),
                 o_e0 = take(ml * 8), o_et = take(ml * 8), from_host = off,
                 o_inv = take(3 * L * ml * 8), o_pp = take(3 * L * ml * 8), o_qq = take(3 * L * ml * 8),
                 o_ri = take(S * ml * 8), o_ra = take(S * ml * 8), o_rc = take(S * ml * 8),
                 o_rs = take(S * ml * 8);
    std::vector<unsigned char> host(from_host, 0);
    auto d2 = [&](size_t o) { return reinterpret_cast<double2*>(host.data() + o); };
    auto d1 = [&](size_t o) { return reinterpret_cast<double*>(host.data() + o); };
    for (long k = 0; k < P; k++) d2(o_tw)[k] = dr_unit(k, P);
    const int N = node ? m - 1 : m;
    for (int k = 0; k < m; k++) {
        const double2 u = dr_unit(k, 4L * m);   // exp(-i pi k / 2m)
        d2(o_post)[k] = make_double2(u.x, -u.y);
        d1(o_off)[k] = M.off[k];
        d1(o_di)[k] = M.di[k];
        d1(o_d0)[k] = M.d0[k];
        d1(o_ei)[k] = M.ei[k];
        d1(o_e0)[k] = M.e0[k];
        d1(o_et)[k] = M.et[k];
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
    const cudaError_t e = cudaMalloc(&dev, off + size_t(p.n) * m * 8);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return VDI_OK;
    }
    VDI_CUDA(e);
    *arena = dev;
    VDI_CUDA(cudaMemcpy(dev, host.data(), from_host, cudaMemcpyHostToDevice));
    auto g2 = [&](size_t o) { return reinterpret_cast<const double2*>(dev + o); };
    auto g1 = [&](size_t o) { return reinterpret_cast<const double*>(dev + o); };
    p.tw = g2(o_tw);
    p.post = g2(o_post);
    p.norm = 2.0 / N;
    p.pin0 = M.pin0;
    p.chirp = g2(o_chirp);
    p.bhat = g2(o_bhat);
    p.off = g1(o_off);
    p.inv = g1(o_inv);
    p.pp = g1(o_pp);
    p.qq = g1(o_qq);
    p.ri = g1(o_ri);
    p.ra = g1(o_ra);
    p.rc = g1(o_rc);
    p.rs = g1(o_rs);
    p.work = reinterpret_cast<double*>(dev + off);
    auto w1 = [&](size_t o) { return reinterpret_cast<double*>(dev + o); };
    dr_tables_k<<<(m + 31) / 32, 32>>>(p, g1(o_di), g1(o_d0), g1(o_ei), g1(o_e0), g1(o_et), M.pin0, w1(o_inv), w1(o_pp),
                                       w1(o_qq), w1(o_ri), w1(o_ra), w1(o_rc), w1(o_rs));
    VDI_CUDA(cudaGetLastError());
    VDI_CUDA(cudaDeviceSynchronize());
    return VDI_OK;
}

/** Threads of the transform kernels: the FFT uses P / 8, the loops over a
 * row's points at least 128. */
static int dr_threads(const DirectPlan& p) { return std::max(128, (1 << p.logp) >> 3); }
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
    using I256 = std::integral_constant<int, 256>;
    using I512 = std::integral_constant<int, 512>;
    using I1024 = std::integral_constant<int, 1024>;
    if (dr_threads(p) <= 256) return blue ? f(I256{}, std::true_type{}) : f(I256{}, std::false_type{});
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

/** Launch shape of dr_resid_sum: 4 rows a warp, the least its batches allow,
 * up to 24 warps an SM (one resident wave), then up to 16 rows (a strip reads
 * two rows beyond its own). */
struct DirectCheck {
    int rows, blocks, vec;
};
static DirectCheck dr_check_shape(int m, int n, const double* z, const double* b) {
    DirectCheck k;
    const long sx = (m + 63) / 64;
    k.rows = DR_ROWS;
    while (k.rows < 16 && sx * ((n + k.rows - 1) / k.rows) > 24L * sm_count()) k.rows *= 2;
    k.blocks = int(std::min(long(MAX_PARTIALS), (sx * ((n + k.rows - 1) / k.rows) + 7) / 8));
    auto al = [](const void* q) { return reinterpret_cast<uintptr_t>(q) % 16 == 0; };
    k.vec = m % 2 == 0 && al(z) && al(b);
    return k;
}

/** The start of a solve with the exact solve behind it (header comment). */
template <class OP>
static int dr_enqueue(cudaStream_t s, const OP& c, const DirectPlan& p, bool blue, double decades, double* z,
                      const double* b, const Reduce& rd, SolveCtl* ctl, int use_cond,
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
    auto modal = [&](auto pin) {
        constexpr bool PIN = decltype(pin)::value;
        if (p.L == 8 && p.modes == 8) dr_modal_k<8, 8, 512, PIN><<<mb, mt, 0, s>>>(p, ctl);
        else if (p.L == 8) dr_modal_k<8, 4, 512, PIN><<<mb, mt, 0, s>>>(p, ctl);
        else if (p.L == 16) dr_modal_k<16, 4, 512, PIN><<<mb, mt, 0, s>>>(p, ctl);
        else dr_modal_k<32, 4, 512, PIN><<<mb, mt, 0, s>>>(p, ctl);
    };
    if (!NODE && p.pin0) modal(std::bool_constant<!NODE>{});
    else modal(std::false_type{});
    dr_select(p, blue, [&](auto t, auto bl) {
        dr_inverse_k<decltype(t)::value, NODE, decltype(bl)::value><<<pairs, T, bytes, s>>>(p, z, ctl);
        return 0;
    });
    const DirectCheck k = dr_check_shape(p.m, p.n, z, b);
    dr_check_k<<<k.blocks, 256, 0, s>>>(c, z, b, k.rows, k.vec, rd, ctl, !NODE, use_cond, h);
    VDI_CUDA(cudaGetLastError());
    return VDI_OK;
}
