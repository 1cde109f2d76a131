// Red-black successive over-relaxation of a cell-centred level (included by
// mg.cu): the solver of the implicit viscous systems.
//
// The viscous operator is the identity plus a weak coupling: the Jacobi
// radius is at most rho = s / (1 + s), s = 2 (vfx + vfy), and red-black SOR
// with the Chebyshev sequence of relaxation factors gains a factor
// (omega - 1) a sweep, omega = 2 / (1 + sqrt(1 - rho^2)): 0.12 at the 100 cSt
// workload's vfx = vfy = 0.4, where a V-cycle of four sweeps and its coarse
// levels gains 0.01. RX_SWEEPS sweeps run in one pass over memory.
//
// cc_stream_k: a warp owns a strip of 64 columns, two per lane in registers,
// and walks down the rows with all 2 RX_SWEEPS colour phases in flight: at
// step t phase p updates row t - p, whose lower neighbour phase p - 1 has just
// updated. Vertical neighbours are the lane's own registers, horizontal ones
// its other column and one shuffle, so the phases need no barrier. A step
// updates the same column of the pair in every phase (rows and colours
// alternate together). Rows of z and b arrive RX_AHEAD steps early by
// asynchronous copies into rings in shared memory, split by column parity;
// z moves on to registers, b is read where a phase needs it. The strip's
// outer RX_HALO columns and 9 rows on either side of a chunk are recomputed
// by the neighbours.
//
// Bound: instructions and the latency they wait for (215 a step, 55 of them
// FP64; 6.3 cycles between a warp's issues at 14 warps an SM, a third of them
// on the FP64 results just before, IPC 0.4 a scheduler), times the redundancy
// of 64/44 columns and (R + 20)/R rows, against 24 bytes a point of memory
// traffic for four sweeps. A pass at 2048 x 1024 takes 43 us, a solve's first
// 50 (48 and 57 with the diagonals of the edge rows in registers, which
// spilled; they are looked up in the operator instead). Whole solves to 1e-10
// at vfx = vfy = 0.4, V-cycles against this: 1024 x 512 227 and 121 us, 2048 x
// 1024 356 and 171 us.
//
// Slower and not kept: four columns a lane at 168 registers (94 us a pass:
// too few warps for the same chain), the rows' loop unrolled over a
// register ring of 14 rows (75 us, instruction fetch), and two dependent
// operations a phase instead of four (178 us a solve: one more instruction
// costs more than the shorter chain gains).

static constexpr int RX_SWEEPS = 4;
static constexpr int RX_PH = 2 * RX_SWEEPS;         // colour phases
static constexpr int RX_HALO = RX_PH + 2;           // even, one more than the residual needs
static constexpr int RX_COLS = 64 - 2 * RX_HALO;    // columns a strip finishes
static constexpr int RX_WARPS = 4;
static constexpr int RX_AHEAD = 4;                  // rows in flight: t + 2 .. t + 1 + RX_AHEAD
static constexpr int RX_BRING = 16;                 // rows of b kept: t - 8 .. t + 5
static constexpr int RX_ZRING = 8;                  // rows of z on their way to registers
static constexpr int RX_ROW = 72;                   // doubles a row: 32 even columns, 8 of padding, 32 odd ones
static constexpr int RX_ODD = 40;
static constexpr size_t RX_SMEM = size_t(RX_WARPS) * (RX_BRING + RX_ZRING) * RX_ROW * sizeof(double);

struct RelaxArgs {
    const double* zin;
    double* zout;
    const double* b;
    double om[RX_PH];      // relaxation factors of the phases
    int R;                 // rows of a chunk
    int strips, chunks;
    int vec;               // 16-byte accesses: even m, aligned arrays
    int role;              // 0 first pass of a solve, 1 odd pass, 2 even pass (copies z back when done)
    Reduce rd;
    SolveCtl* ctl;
    int use_cond;
    cudaGraphConditionalHandle h;
};

/** What the pass behind the current one does (SolveCtl::direct). */
enum { RX_STOP = 0, RX_SWEEP = 1, RX_COPY = 2 };

/** grid_sum of three values: partials k, nb + k and 2 nb + k. */
__device__ bool grid_sum3(const double (&v)[3], Reduce rd, double (&tot)[3]) {
    __shared__ int last;
    const int nb = gridDim.x;
    if (threadIdx.x == 0) {
        for (int q = 0; q < 3; q++) rd.partials[q * nb + blockIdx.x] = v[q];
        __threadfence();
        last = atomicAdd(rd.counter, 1u) == unsigned(nb - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double a[3] = {0, 0, 0};
    for (int k = threadIdx.x; k < nb; k += blockDim.x)
        for (int q = 0; q < 3; q++) a[q] += __ldcg(rd.partials + q * nb + k);
    for (int q = 0; q < 3; q++) {
        __syncthreads();
        tot[q] = block_sum(a[q]);
    }
    if (threadIdx.x == 0) *rd.counter = 0;
    return true;
}

__device__ __forceinline__ void rx_copy8(uint32_t dst, const double* src, int bytes) {
    // 0 bytes: nothing is read, the destination is zero-filled
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

/** What a lane of rx_walk keeps beside its rows. */
struct RxLane {
    double iv[2];                          // inverse diagonals on interior rows (0: a column outside)
    int xc[2];                             // column classes, for the other rows' and the diagonals
    bool use0, use1;                       // columns this lane finishes
    int na, nb;                            // bytes of its two copies of a row (0: outside, zero-filled)
    const double *pz, *pb;                 // its first column of the next row to copy
    uint32_t az, ab;                       // shared addresses of its copies in the rings
    double raw;                            // row t - 1 before its phase 0, in the column that phase updated
    double sb, s0, s1;
};

static constexpr int RX_U = 4;                  // steps an iteration
static constexpr int RX_W = RX_PH + 2 + RX_U;   // rows t - 9 .. t + RX_U in registers
static constexpr int RX_T = RX_PH + 1;          // place of row t at the start of an iteration

/** Asynchronous copies of row r. */
__device__ __forceinline__ void rx_copy_row(RxLane& L, int r, int n, int m) {
    const bool in = unsigned(r) < unsigned(n);
    const uint32_t oz = L.az + uint32_t(r & (RX_ZRING - 1)) * (RX_ROW * 8),
                   ob = L.ab + uint32_t(r & (RX_BRING - 1)) * (RX_ROW * 8);
    const int na = in ? L.na : 0, nb = in ? L.nb : 0;
    rx_copy8(oz, L.pz, na);
    rx_copy8(oz + 128, L.pz + 32, nb);
    rx_copy8(ob, L.pb, na);
    rx_copy8(ob + 128, L.pb + 32, nb);
    asm volatile("cp.async.commit_group;" ::: "memory");
    L.pz += m;
    L.pb += m;
}

/** RX_U steps from row t (a multiple of 4): SLOW while a row they touch is
 * the grid's first or last, whose diagonal differs, or lies outside, where a
 * zero inverse diagonal keeps z zero. */
template <bool FIRST, bool SLOW>
__device__ __forceinline__ void rx_steps(const CCc<double>& c, const RelaxArgs& a, RxLane& L, double (&z)[RX_W][2],
                                         const double* sz, const double* sbv, int t, int i0, int y0, int y1) {
    const int m = c.m, n = c.n;
    auto inv = [&](int r, int k) -> double {
        if (!SLOW) return L.iv[k];
        const bool on = unsigned(r) < unsigned(n) && L.iv[k] != 0.;
        return on ? c.invd[L.xc[k]][r == 0 ? 0 : (r == n - 1 ? 2 : 1)] : 0.;
    };
    auto diag = [&](int r, int k) -> double {
        if (!SLOW) return c.d[L.xc[k]][1];
        return c.d[L.xc[k]][r == 0 ? 0 : (r == n - 1 ? 2 : 1)];
    };
    const double ox = -c.ox, oy = -c.oy;
    // row t + d sits in group (t + d) / 4 of its ring: three base addresses
    // and constants
    const int g = t >> 2;
    const double* bg[4];
#pragma unroll
    for (int k = 0; k < 4; k++) bg[k] = sbv + (((g - k) & (RX_BRING / 4 - 1)) * 4) * RX_ROW;
    auto bat = [&](int d, int q) -> double {   // row t + d, column parity q
        const int k = d >= 0 ? 0 : (3 - d) / 4, o = d + 4 * k;
        return bg[k][o * RX_ROW + q * RX_ODD];
    };
    const double* zg0 = sz + ((g & 1) * 4) * RX_ROW;
    const double* zg1 = sz + (((g + 1) & 1) * 4) * RX_ROW;
#pragma unroll
    for (int s = 0; s < RX_U; s++) {
        const int q = s & 1, h0 = RX_T + s, tt = t + s;
        // row tt + 1 is there once only the RX_AHEAD groups after it are pending
        rx_copy_row(L, tt + RX_AHEAD + 1, n, m);
        asm volatile("cp.async.wait_group %0;" ::"n"(RX_AHEAD) : "memory");
        __syncwarp();
        {
            const double* w = s + 1 < 4 ? zg0 + (s + 1) * RX_ROW : zg1;
            z[h0 + 1][0] = w[0];
            z[h0 + 1][1] = w[RX_ODD];
        }
        double bv[RX_PH];
#pragma unroll
        for (int p = 0; p < RX_PH; p++) bv[p] = bat(s - p, q);
        if constexpr (FIRST) {
            if (tt >= y0 && tt < y1) {
                const double l = __shfl_up_sync(0xffffffffu, z[h0][1], 1);
                const double r = __shfl_down_sync(0xffffffffu, z[h0][0], 1);
                const double b0 = q ? bat(s, 0) : bv[0], b1 = q ? bv[0] : bat(s, 1);
                const double d0 = q ? L.raw : z[h0 - 1][0], d1 = q ? z[h0 - 1][1] : L.raw;
                const double r0 = b0 - diag(tt, 0) * z[h0][0] + (ox * (l + z[h0][1]) + oy * (d0 + z[h0 + 1][0]));
                const double r1 = b1 - diag(tt, 1) * z[h0][1] + (ox * (z[h0][0] + r) + oy * (d1 + z[h0 + 1][1]));
                if (L.use0) { L.s0 += r0 * r0; L.sb += b0 * b0; }
                if (L.use1) { L.s0 += r1 * r1; L.sb += b1 * b1; }
            }
            L.raw = z[h0][q];
        }
#pragma unroll
        for (int p = 0; p < RX_PH; p++) {
            const int h = h0 - p;
            const double nb = q ? __shfl_down_sync(0xffffffffu, z[h][0], 1) : __shfl_up_sync(0xffffffffu, z[h][1], 1);
            double x = fma(ox, nb + z[h][1 - q], bv[p]);
            x = fma(oy, z[h - 1][q] + z[h + 1][q], x);
            z[h][q] = fma(a.om[p], fma(x, inv(tt - p, q), -z[h][q]), z[h][q]);
        }
        {
            const int h = h0 - RX_PH + 1, r = tt - RX_PH + 1;
            if (r >= y0 && r < y1 && L.use0) {
                double* o = a.zout + long(r) * m + i0;
                if (a.vec) {
                    // even m and x0: both columns lie inside
                    *reinterpret_cast<double2*>(o) = make_double2(z[h][0], z[h][1]);
                } else {
                    o[0] = z[h][0];
                    if (L.use1) o[1] = z[h][1];
                }
            }
        }
        if (tt - RX_PH >= y0 && tt - RX_PH < y1) {
            const int h = h0 - RX_PH, rr = tt - RX_PH;
            const double l = __shfl_up_sync(0xffffffffu, z[h][1], 1);
            const double r = __shfl_down_sync(0xffffffffu, z[h][0], 1);
            const double r0 =
                bat(s - RX_PH, 0) - diag(rr, 0) * z[h][0] + (ox * (l + z[h][1]) + oy * (z[h - 1][0] + z[h + 1][0]));
            const double r1 =
                bat(s - RX_PH, 1) - diag(rr, 1) * z[h][1] + (ox * (z[h][0] + r) + oy * (z[h - 1][1] + z[h + 1][1]));
            if (L.use0) L.s1 += r0 * r0;
            if (L.use1) L.s1 += r1 * r1;
        }
    }
}

/** One warp's strip and chunk: RX_SWEEPS sweeps from a.zin to a.zout, with
 * the residual sum after them (s1) and, FIRST, before them (s0) and the
 * source's (sb). The rows of z move up in the registers by RX_U every RX_U
 * steps: a loop unrolled over a whole register ring is bound by instruction
 * fetch. */
template <bool FIRST>
__device__ __forceinline__ void rx_walk(const CCc<double>& c, const RelaxArgs& a, double* sz, double* sbv, int x0,
                                        int y0, int y1, RxLane& L) {
    const int m = c.m, n = c.n, lane = threadIdx.x & 31, i0 = x0 + 2 * lane;
    const bool in0 = unsigned(i0) < unsigned(m), in1 = unsigned(i0 + 1) < unsigned(m);
    L.use0 = in0 && lane >= RX_HALO / 2 && lane < 32 - RX_HALO / 2;
    L.use1 = L.use0 && in1;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const bool in = k ? in1 : in0;
        const int x = in ? cls(i0 + k, m) : 0;
        L.iv[k] = in ? c.invd[x][1] : 0.;
        L.xc[k] = x;
    }
    // x0 + t even at the first step of an iteration (x0 is even): step s then
    // updates column s & 1 of the pair. y0 is a multiple of 4.
    int t = y0 - 12;
    const int tend = y1 - 1 + RX_PH;
    // this lane's share of a row's copies: columns lane and lane + 32
    const int ca = x0 + lane;
    L.na = unsigned(ca) < unsigned(m) ? 8 : 0;
    L.nb = unsigned(ca + 32) < unsigned(m) ? 8 : 0;
    const uint32_t dcol = uint32_t(((lane & 1) * RX_ODD + (lane >> 1)) * 8);
    L.az = static_cast<uint32_t>(__cvta_generic_to_shared(sz)) + dcol;
    L.ab = static_cast<uint32_t>(__cvta_generic_to_shared(sbv)) + dcol;
    L.pz = a.zin + long(t) * m + ca;
    L.pb = a.b + long(t) * m + ca;
    double z[RX_W][2];
#pragma unroll
    for (int d = 0; d < RX_W; d++) z[d][0] = z[d][1] = 0.;
    // rows below the first copied one read b from the ring: finite values, as
    // a zero inverse diagonal then keeps z zero outside the grid
    for (int k = lane; k < RX_BRING * RX_ROW; k += 32) sbv[k] = 0.;
    __syncwarp();
#pragma unroll
    for (int d = 0; d <= RX_AHEAD; d++) rx_copy_row(L, t + d, n, m);
    asm volatile("cp.async.wait_group %0;" ::"n"(RX_AHEAD) : "memory");
    __syncwarp();
    const double *zl = sz + lane, *bl = sbv + lane;
    {
        const double* w = zl + (t & (RX_ZRING - 1)) * RX_ROW;
        z[RX_T][0] = w[0];
        z[RX_T][1] = w[RX_ODD];
    }
    L.raw = 0.;
    for (; t <= tend; t += RX_U) {
        // rows t - 8 .. t + 4
        if (t - RX_PH > 0 && t + RX_U < n - 1) rx_steps<FIRST, false>(c, a, L, z, zl, bl, t, i0, y0, y1);
        else rx_steps<FIRST, true>(c, a, L, z, zl, bl, t, i0, y0, y1);
#pragma unroll
        for (int d = 0; d + RX_U < RX_W; d++) {
            z[d][0] = z[d + RX_U][0];
            z[d][1] = z[d + RX_U][1];
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

/** RX_SWEEPS sweeps from zin to zout. FIRST: also ||b||^2 and the residual
 * norm of zin, and the decision that starts a solve (a zero source zeroes
 * zin, which is then the caller's iterate). */
template <bool FIRST>
__global__ void __launch_bounds__(32 * RX_WARPS, 16 / RX_WARPS) cc_stream_k(CCc<double> c, RelaxArgs a) {
    const int m = c.m, n = c.n;
    SolveCtl* ctl = a.ctl;
    extern __shared__ __align__(16) unsigned char rx_raw[];
    __shared__ int mode;
    if (!FIRST) {
        // every block reads the mode before the last one to finish sets it
        if (threadIdx.x == 0) mode = ctl->direct;
        __syncthreads();
        if (mode == RX_STOP) return;
        if (mode == RX_COPY) {
            // the previous pass met the tolerance (or the cap) in its output
            if (a.role == 2) {
                const long st = long(gridDim.x) * blockDim.x, k0 = blockIdx.x * long(blockDim.x) + threadIdx.x;
                if (a.vec) {
                    const double2* src = reinterpret_cast<const double2*>(a.zin);
                    double2* dst = reinterpret_cast<double2*>(a.zout);
#pragma unroll 8
                    for (long k = k0; k < long(m) * n / 2; k += st) dst[k] = src[k];
                } else {
#pragma unroll 8
                    for (long k = k0; k < long(m) * n; k += st) a.zout[k] = a.zin[k];
                }
            }
            return;
        }
    }
    const int wid = blockIdx.x * RX_WARPS + (threadIdx.x >> 5);
    RxLane L;
    L.sb = L.s0 = L.s1 = 0;
    if (wid < a.strips * a.chunks) {
        const int chunk = wid / a.strips, x0 = (wid - chunk * a.strips) * RX_COLS - RX_HALO;
        const int y0 = chunk * a.R, y1 = min(y0 + a.R, n);
        double* sz = reinterpret_cast<double*>(rx_raw) + size_t(threadIdx.x >> 5) * (RX_ZRING + RX_BRING) * RX_ROW;
        rx_walk<FIRST>(c, a, sz, sz + RX_ZRING * RX_ROW, x0, y0, y1, L);
    }
    double v[3] = {FIRST ? block_sum(L.sb) : 0., 0., 0.}, tot[3];
    __syncthreads();
    v[1] = FIRST ? block_sum(L.s0) : 0.;
    __syncthreads();
    v[2] = block_sum(L.s1);
    if (!grid_sum3(v, a.rd, tot)) return;
    if (threadIdx.x == 0) {
        int next = RX_SWEEP;
        if (FIRST) {
            ctl->bnorm2 = tot[0];
            ctl->it = 0;
            ctl->done = 0;
            ctl->status = 0;
            solve_decide(ctl, tot[0] == 0. ? 0. : tot[1], 0, a.use_cond, a.h);
            if (ctl->done) {
                next = RX_STOP;
                atomicAdd(&ctl->more_launches, 2ull);   // this pass and its pair's other, which returns
            }
        }
        if (next == RX_SWEEP) {
            // a pair of passes counts as one V-cycle, an odd last pass too:
            // the cap is looked at behind the even ones
            const bool odd = a.role != 2 && tot[2] > ctl->rtol * ctl->rtol * ctl->bnorm2;
            solve_decide(ctl, tot[2], !odd, a.use_cond, a.h);
            // an odd pass's result moves to the caller's array either way
            if (ctl->done) next = a.role == 2 ? RX_STOP : RX_COPY;
        }
        ctl->direct = next;
        mode = FIRST && tot[0] == 0.;
    }
    if (FIRST) {
        __syncthreads();
        if (mode)
            for (long k = threadIdx.x; k < long(m) * n; k += blockDim.x) const_cast<double*>(a.zin)[k] = 0.;
    }
}

// -------------------------------------------------------------------- host
/** Relaxation factors of a viscous level's phases (Chebyshev sequence of
 * red-black SOR), and whether the solver uses them (MG::setup_relax). */
struct RelaxPlan {
    bool on = false;
    double rho2 = 0;       // square of the bound on the Jacobi radius
    double om_inf = 1;     // limit of the factors
    int R = 16;
    double* tmp = nullptr; // the odd passes' output
};

/** Rows of a chunk: about 16 warps an SM, what the registers hold, with at least 8 rows
 * against the 20 steps that a chunk adds, and few enough blocks for the
 * partial sums; 0 where one chunk a strip is too many (rows of more than
 * 480,000 points). */
static int rx_rows(int m, int n) {
    const long strips = (long(m) + RX_COLS - 1) / RX_COLS;
    long R = (strips * n + 2399) / 2400;
    R = (std::min(64L, std::max(8L, R)) + 3) / 4 * 4;   // whole iterations of the walk
    while (strips * ((n + R - 1) / R) / RX_WARPS + 1 > MAX_PARTIALS / 3) {
        if (R >= n) return 0;
        R *= 2;
    }
    return int(R);
}

static cudaError_t rx_prepare() {
    cudaError_t e = cudaFuncSetAttribute(cc_stream_k<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(RX_SMEM));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(cc_stream_k<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(RX_SMEM));
    return e;
}

static int rx_enqueue(cudaStream_t s, const CCc<double>& c, const RelaxPlan& p, int role, int pass, const double* zin,
                      double* zout, const double* b, const Reduce& rd, SolveCtl* ctl, int use_cond,
                      cudaGraphConditionalHandle h) {
    RelaxArgs a{};
    a.zin = zin;
    a.zout = zout;
    a.b = b;
    double om = 1;
    for (int k = 0; k < pass * RX_PH + RX_PH && k < 3 * RX_PH; k++) {
        if (k == 1) om = 1 / (1 - 0.5 * p.rho2);
        else if (k > 1) om = 1 / (1 - 0.25 * p.rho2 * om);
        if (k >= pass * RX_PH) a.om[k - pass * RX_PH] = om;
    }
    if (pass >= 2)
        for (double& w : a.om) w = p.om_inf;
    a.R = p.R;
    a.strips = (c.m + RX_COLS - 1) / RX_COLS;
    a.chunks = (c.n + p.R - 1) / p.R;
    auto al = [](const void* q) { return reinterpret_cast<uintptr_t>(q) % 16 == 0; };
    a.vec = c.m % 2 == 0 && al(zin) && al(zout) && al(b);
    a.role = role;
    a.rd = rd;
    a.ctl = ctl;
    a.use_cond = use_cond;
    a.h = h;
    const int nb = (a.strips * a.chunks + RX_WARPS - 1) / RX_WARPS;
    if (role == 0) cc_stream_k<true><<<nb, 32 * RX_WARPS, RX_SMEM, s>>>(c, a);
    else cc_stream_k<false><<<nb, 32 * RX_WARPS, RX_SMEM, s>>>(c, a);
    VDI_CUDA(cudaGetLastError());
    return VDI_OK;
}
