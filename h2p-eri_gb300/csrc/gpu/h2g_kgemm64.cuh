/*
 * FP64 products of the exchange build on the tensor cores.
 *
 * What bounds it. FP64 FMAs run at 2 per clock and SM, so the FP64 GEMMs took
 * 70-80 % of that pipe's time and nothing else could help. bf16 MMAs run some
 * 2000 times as fast; with the exact slicing of the operands (Ozaki, Ogita,
 * Oishi, Rump, Numer. Algorithms 59, 2012) an FP64 product takes 55 of them.
 *
 * Arithmetic. Every row of an operand (64 values along k) is scaled by the
 * power of two of its largest entry to 80-bit integers, written as ten
 * signed 8-bit digits, x = 2^(e - 79) sum_i d_i 256^(9 - i), d_i in [-128, 127],
 * as bf16 values. Digit products with i + j = l are summed over k and over
 * (i, j) in one FP32 accumulator per level l = 0 .. 9: with 64 values of k at
 * most 10 * 64 products of at most 2^14, so every partial sum is an integer
 * below 2^24 and exact. Levels above 9 are left out. The levels are added as
 * 96-bit integers, rounded once to FP64 and added to the output.
 *
 * Accuracy. A term is off by at most 2^-76 of 2^(e_P + e_Q), the power of two
 * above the product of the two rows' largest entries (the levels left out
 * 9 * 2^-80, the cut to 80 bits 2^-78). An output v of at least 2^-20 of that
 * is then off by less than 2^-56 |v| per term, below the 2^-53 |a||b| that each
 * step of an FP64 chain may add. One below it (rows that are small where the
 * other is large, cancellation), or with an infinity or a NaN in its rows, is
 * summed anew with FP64 FMAs, by the warp that drains it: 0.03 % of the outputs
 * of C5H12, 0.6 % of C10H22's (all in the two upward inner levels: some SMs
 * have the FP64 pipe 80 % busy there, others 1 %). With eight digits the line
 * would lie at 2^-9, and 2 to 11 % of the outputs below it. An output of finite
 * rows, one of which is zero, is not written. (Outputs of rows that are zero
 * wherever the other is not are 0.1 to 0.2 % of C10H22's; a bit per two k to
 * know them cost more than it saved, 110 against 107 ms.)
 *
 * Layout. One CTA per SM walks the launch's tiles: 128 rows of one side of the
 * product (the MMA's rows, P) against the other side in steps of 16 (the MMA's
 * columns, Q). The digits of P (64 k, 160 KB) stay in shared memory for all
 * steps; those of Q are double-buffered (2 x 20 KB, digit-major rows, so that
 * digit i of P and digits 0 .. 9 - i of Q are one MMA of N = 16 (10 - i) columns
 * whose columns are the levels i .. 9). Warp roles, handing over through
 * mbarriers (bounded waits): one warp forms the tiles' descriptors and the
 * offsets of Q's rows ahead of the others (a tile starts with four dependent
 * loads, which the others would all wait for), eight gather and slice (8, 16 or
 * 32 lanes along k per row, by K; P together, the steps of Q in two groups in
 * turn), one thread issues the MMAs, eight warps drain one of two 160-column
 * accumulators. The hand-overs are the bound: each role works about half the
 * time. P is the side along which C is contiguous, so that the drain's atomics
 * are (strided ones ran at 31 G/s on a 2 GB array, contiguous ones at 270):
 *  - rows of C contiguous (wide): P = rows of C, Q = columns in runs of kZRun;
 *    every column value is sliced once per 128 rows, P's once per run. K is cut
 *    into tiles of 64 whose sums meet in the output's atomics.
 *  - else P = columns of C, Q = all its rows; with one step (up to 16 rows) up to
 *    kZGroup = 128 of k are summed before the drain: levels 0 .. 7 stay below 2^24
 *    and exact, 8 and 9 can pass it and then round to even integers, 2^-77 of the
 *    largest product.
 * Measured (with the near field on k_near64): K of C10H22 (266 GFLOP, QR 1e-6)
 * 345 ms with FP64 FMAs, 107 here (57 with eight digits in steps of 32), of C30H62
 * 5.97 and 1.49 s, of C5H12 through host arrays 13.4 and 4.0 ms (2.9); error of C5H12's K against 80-bit
 * arithmetic 1.25e-15 and 0.93e-15.
 */
#ifndef H2G_KGEMM64_CUH
#define H2G_KGEMM64_CUH

namespace h2g {

constexpr int kZP = 128, kZQ = 16, kZK = 64, kZD = 10;
constexpr int kZRun = 512, kZGroup = 128;
constexpr int kZProd = 8, kZEpi = 8, kZCols = 4 * kZQ / kZEpi;
constexpr int kZThreads = 32 * (kZProd + 2 + kZEpi);
constexpr uint32_t kZPlane = kZP * kZK * 2;                    /* one digit of P */
constexpr uint32_t kZQBuf = kZD * kZQ * kZK * 2;               /* all digits of one step of Q */
constexpr uint32_t kZOffQ = kZD * kZPlane;
constexpr uint32_t kZOffD = kZOffQ + 2 * kZQBuf;               /* descriptors of kZSlots tiles */
constexpr int kZSlots = 3;
constexpr uint32_t kZDesc = 128 + (2 * kZP + 2 * kZGroup) * 8;
constexpr int kZRows = 8;                                      /* ring of steps' rows of Q */
constexpr uint32_t kZOffE = kZOffD + kZSlots * kZDesc;         /* exponents of P [4 tiles][128], rows of Q [kZRows][16] */
constexpr uint32_t kZOffBar = kZOffE + 4 * kZP * 4 + kZRows * kZQ * 24;
constexpr uint32_t kZSmem = kZOffBar + 272;
constexpr uint32_t kZSmemLaunch = kZSmem + 1024;               /* + slack to align to 1024 bytes */
static_assert(kZSmemLaunch <= 227 * 1024, "shared memory of the FP64 exchange kernel");
constexpr int kZBadExp = 2047;                                 /* exponents from here on: infinities, NaNs */
constexpr unsigned kZMargin = 0x2100;                          /* rows from 1.992 2^e on take the next exponent */

__host__ __device__ constexpr long long z_ceil(long long a, long long b) { return (a + b - 1) / b; }
__host__ __device__ constexpr int z_kgroup(int M, bool wide) { return wide || M > kZQ ? kZK : kZGroup; }
__host__ __device__ constexpr long long z_tiles(int M, int N, int K, int Z, bool wide)
{
    const long long NZ = (long long)N * Z;
    return z_ceil(K, z_kgroup(M, wide)) * (wide ? z_ceil(M, kZP) * z_ceil(NZ, kZRun) : z_ceil(NZ, kZP));
}

/* x 2^(79 - E), E = emax - 1022, cut to an integer (of a negative one the words
 * are inverted, one unit off), plus 128 in every byte */
struct ZFixed {
    unsigned w0, w1, w2;
};
__device__ __forceinline__ ZFixed z_fixed(double x, int emax)
{
    const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
    const unsigned m1 = (unsigned)(hi & 0xfffff) | (e ? 0x100000u : 0u), m0 = (unsigned)__double2loint(x), s = (unsigned)(hi >> 31);
    const int d = min(6 + emax - max(e, 1), 95);   /* (m1, m0, 0) >> d */
    const bool p1 = d >= 32, p2 = d >= 64;
    const unsigned x0 = p2 ? m1 : p1 ? m0 : 0u, x1 = p2 ? 0u : p1 ? m1 : m0, x2 = p1 ? 0u : m1;
    ZFixed r{__funnelshift_r(x0, x1, d) ^ s, __funnelshift_r(x1, x2, d) ^ s, __funnelshift_r(x2, 0u, d) ^ s};
    asm("add.cc.u32 %0, %0, 0x80808080;\n\taddc.cc.u32 %1, %1, 0x80808080;\n\taddc.u32 %2, %2, 0x8080;"
        : "+r"(r.w0), "+r"(r.w1), "+r"(r.w2));
    return r;
}
/* digit d (0: the top byte of the 80 bits) of two such numbers as bf16: byte -
 * 128, from 128 + (byte & 127) - (byte < 128 ? 256 : 128) */
template <int D>
__device__ __forceinline__ uint32_t z_digit2(const ZFixed &a, const ZFixed &b)
{
    constexpr unsigned k = (9 - D) & 3, sel = k | (k << 4) | ((4 + k) << 8) | ((4 + k) << 12);
    const uint32_t w = D < 2 ? __byte_perm(a.w2, b.w2, sel) : D < 6 ? __byte_perm(a.w1, b.w1, sel) : __byte_perm(a.w0, b.w0, sel);
    uint32_t r;
    asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"((w & 0x007f007fu) | 0x43004300u), "r"((w & 0x00800080u) ^ 0xC380C380u));
    return r;
}

/* Biased exponent e of a row whose largest high word is h: |x| < 2^(e - 1022),
 * with room for the top digit below 128; 0 for a row of zeros. */
__device__ __forceinline__ int z_biased(int h) { return h == 0 ? 0 : max((int)(((unsigned)h + kZMargin) >> 20), 1); }
__device__ __forceinline__ int z_exp(int h, int lpr)   /* over the row's lpr lanes */
{
    for (int o = lpr >> 1; o > 0; o >>= 1) h = max(h, __shfl_xor_sync(0xffffffffu, h, o));
    return z_biased(h);
}
/* |x|'s high word; 1 in place of 0 where x is not zero */
__device__ __forceinline__ int z_top(double x)
{
    return (__double2hiint(x) & 0x7fffffff) | (__double2loint(x) != 0 ? 1 : 0);
}
/* Slices two rows: this lane's two values of each (k = 2 kl, 2 kl + 1), `lpr`
 * lanes per row, digit planes `plane` bytes apart from the rows' places in the
 * first; ex < 0: the rows' exponents are found here. (As a called function it
 * saved and restored registers in local memory, with little L1 beside 220 KB
 * of shared memory.) */
__device__ __forceinline__ int2 z_slice(double x0, double x1, double y0, double y1, int lpr, unsigned char *dx,
                                     unsigned char *dy, uint32_t plane, int ex, int ey)
{
    if (ex < 0) {
        int h = max(z_top(x0), z_top(x1)), g = max(z_top(y0), z_top(y1));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int h1 = __shfl_xor_sync(0xffffffffu, h, o), g1 = __shfl_xor_sync(0xffffffffu, g, o);
            h = o < lpr ? max(h, h1) : h;
            g = o < lpr ? max(g, g1) : g;
        }
        ex = z_biased(h);
        ey = z_biased(g);
    }
    const ZFixed a = z_fixed(x0, ex), b = z_fixed(x1, ex), c = z_fixed(y0, ey), d = z_fixed(y1, ey);
#define Z_DIGIT(i)                                                                  \
    *reinterpret_cast<uint32_t *>(dx + i * plane) = z_digit2<i>(a, b);              \
    *reinterpret_cast<uint32_t *>(dy + i * plane) = z_digit2<i>(c, d);
    Z_DIGIT(0) Z_DIGIT(1) Z_DIGIT(2) Z_DIGIT(3) Z_DIGIT(4) Z_DIGIT(5) Z_DIGIT(6) Z_DIGIT(7)
    Z_DIGIT(8) Z_DIGIT(9)
#undef Z_DIGIT
    return make_int2(ex, ey);
}

/* (sum_l L_l 256^(9 - l)) 2^s: the sum is hi 2^64 + w1 2^32 + w0; its 63 leading
 * bits are rounded to FP64 (one conversion on the FP64 pipe, the rest integer).
 * sure: it is at least 2^66, 2^-20 of the largest product. */
__device__ __forceinline__ double z_combine(const uint32_t (&r)[kZD], int s, bool &sure)
{
    auto L = [&](int l) { return __float2int_rn(__uint_as_float(r[l])); };
    auto four = [&](int l) {
        long long t = L(l + 3);
        t += (long long)L(l + 2) * 256;
        t += (long long)L(l + 1) * 65536;
        t += (long long)L(l) * 16777216;
        return t;
    };
    const long long lo = four(6), mid = four(2) + (lo >> 32);
    const int hi = L(0) * 256 + L(1) + (int)(mid >> 32);
    sure = (unsigned)(hi + 4) >= 8u;
    const int sh = 33 - __clz(hi ^ (hi >> 31));   /* 1 .. 31 */
    const unsigned w0 = (unsigned)lo, w1 = (unsigned)mid;
    const unsigned t0 = __funnelshift_r(w0, w1, sh), t1 = __funnelshift_r(w1, (unsigned)hi, sh);
    const double d = (double)(long long)(((unsigned long long)t1 << 32) | t0);
    const int w = __double2hiint(d), e = ((w >> 20) & 0x7ff) + s + sh;
    if (w == 0) return 0.0;
    if (e < 1 || e > 2046) return scalbn(d, s + sh);
    return __hiloint2double(w + (int)((unsigned)(s + sh) << 20), __double2loint(d));
}

__device__ __forceinline__ long long z_idx(const int *g, long long i) { return g ? (long long)__ldg(g + i) : i; }

/* One side of a product: its rows (rows of A, or columns (z, j) of B) and the
 * k of its elements; offsets are in elements of p. */
struct ZSide {
    const void *p;
    const int *gc, *gz, *gk;
    long long sc, sz, sk, rows;
    int N;
    __device__ __forceinline__ long long row(long long i) const
    {
        if (i >= rows) return -1;
        const int z = (int)i / N, c = (int)i - z * N;
        return z_idx(gz, z) * sz + z_idx(gc, c) * sc;
    }
    __device__ __forceinline__ long long k(int i) const { return z_idx(gk, i) * sk; }
};
__device__ __forceinline__ ZSide z_side_a(const GemmTask &T)
{
    return ZSide{T.a.p, T.a.gr, nullptr, T.a.gc, T.a.sr, 0, T.a.sc, T.M, 0x7fffffff};
}
__device__ __forceinline__ ZSide z_side_b(const GemmTask &T)
{
    return ZSide{T.b.p, T.b.gc, T.b.gz, T.b.gr, T.b.sc, T.b.sz, T.b.sr,
                 (long long)T.N * T.Z, T.N};
}

/* C's offsets along its rows and along its columns */
__device__ __forceinline__ ZSide z_side_c_rows(const GemmTask &T)
{
    return ZSide{nullptr, T.c.gr, nullptr, nullptr, T.c.sr, 0, 0, T.M, 0x7fffffff};
}
__device__ __forceinline__ ZSide z_side_c_cols(const GemmTask &T)
{
    return ZSide{nullptr, T.c.gc, T.c.gz, nullptr, T.c.sc, T.c.sz, 0, (long long)T.N * T.Z, T.N};
}

/* Descriptor of a tile: what the roles need of it, and after it the offsets of
 * P's 128 rows in their operand and in C (-1 past the end) and of the k of both
 * sides. */
struct ZTile {
    const double *p, *q;        /* operands */
    double *out;
    const GemmTask *task;
    long long p0, q0;           /* first row of P, of Q */
    int k0, kn, steps, wide;    /* k range [k0, k0 + kn), steps of Q, P = rows of C */
    int rows;                   /* rows of P */
};
static_assert(sizeof(ZTile) <= 128, "tile descriptor");
__device__ __forceinline__ ZTile z_tile(long long tile, const GemmTask *__restrict__ tasks,
                                        const long long *__restrict__ tile_start, const int *__restrict__ tile_task)
{
    ZTile t;
    const int task = tile_task[tile];
    const GemmTask &T = tasks[task];
    long long loc = tile - tile_start[task];
    const long long NZ = (long long)T.N * T.Z;
    t.task = &T;
    t.wide = T.swap;
    const int kg = z_kgroup(T.M, t.wide), nk = (T.K + kg - 1) / kg;
    t.k0 = (int)(loc % nk) * kg;
    t.kn = min(kg, T.K - t.k0);
    loc /= nk;
    if (t.wide) {
        const int np = (T.M + kZP - 1) / kZP;
        t.p0 = (loc % np) * kZP;
        t.q0 = (loc / np) * kZRun;
        t.steps = (int)((min(NZ - t.q0, (long long)kZRun) + kZQ - 1) / kZQ);
        t.rows = (int)min((long long)T.M - t.p0, (long long)kZP);
        t.p = reinterpret_cast<const double *>(T.a.p);
        t.q = reinterpret_cast<const double *>(T.b.p);
    } else {
        t.p0 = loc * kZP;
        t.q0 = 0;
        t.steps = (T.M + kZQ - 1) / kZQ;
        t.rows = (int)min(NZ - t.p0, (long long)kZP);
        t.p = reinterpret_cast<const double *>(T.b.p);
        t.q = reinterpret_cast<const double *>(T.a.p);
    }
    t.out = reinterpret_cast<double *>(const_cast<void *>(T.c.p));
    return t;
}

/* Wait for a phase of an mbarrier, suspended by the hardware in slices of
 * 20 us (a spinning warp would take issue slots from the working ones), at
 * most 50000 of them. */
__device__ __forceinline__ bool z_wait(uint32_t bar, uint32_t parity)
{
    for (int i = 0; i < 50000; i++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity), "r"(20000u)
                     : "memory");
        if (ok) return true;
    }
    return false;
}

/* A row of Q of one step: its offset in its operand, in C, and its exponent. */
struct __align__(8) ZRow {
    long long src, off;
    int e, pad_;
};

__global__ void __launch_bounds__(kZThreads, 1) k_gemm_z(const GemmTask *__restrict__ tasks,
                                                         const long long *__restrict__ tile_start, int n_task,
                                                         const int *__restrict__ tile_task, unsigned *err)
{
    extern __shared__ __align__(16) unsigned char z_raw[];
    unsigned char *sm = z_raw + ((1024u - (umma::smem_u32(z_raw) & 1023u)) & 1023u);
    const uint32_t sbase = umma::smem_u32(sm), bar0 = sbase + kZOffBar;
    int *eP = reinterpret_cast<int *>(sm + kZOffE);
    ZRow *rQ = reinterpret_cast<ZRow *>(eP + 4 * kZP);
    const uint32_t pfull = bar0, pfree = bar0 + 8;
    auto qfull = [&](int b) { return bar0 + 16u + 8u * b; };
    auto qfree = [&](int b) { return bar0 + 32u + 8u * b; };
    auto afull = [&](int b) { return bar0 + 48u + 8u * b; };
    auto afree = [&](int b) { return bar0 + 64u + 8u * b; };
    auto rfull = [&](uint32_t a) { return bar0 + 80u + 8u * (a % kZRows); };
    auto rfree = [&](uint32_t a) { return bar0 + 144u + 8u * (a % kZRows); };
    auto rturn = [](uint32_t a) { return (a / kZRows) & 1; };
    auto rows_of = [&](uint32_t a) { return rQ + (a % kZRows) * kZQ; };
    auto dfull = [&](uint32_t slot) { return bar0 + 208u + 8u * slot; };
    auto dfree = [&](uint32_t slot) { return bar0 + 232u + 8u * slot; };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + kZOffBar + 256);
    volatile int *dead = reinterpret_cast<volatile int *>(sm + kZOffBar + 260);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long ntiles = tile_start[n_task];

    if (tid == 0) {
        auto init = [](uint32_t b, int n) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(n) : "memory");
        };
        init(pfull, kZProd);
        init(pfree, 1);
        for (int b = 0; b < 2; b++) {
            init(qfull(b), kZProd / 2);
            init(qfree(b), 1);
            init(afull(b), 1);
            init(afree(b), kZEpi);
        }
        for (uint32_t a = 0; a < (uint32_t)kZRows; a++) {
            init(rfull(a), 1);
            init(rfree(a), kZEpi);
        }
        for (uint32_t d = 0; d < kZSlots; d++) {
            init(dfull(d), 1);
            init(dfree(d), kZProd + 1 + kZEpi);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *dead = 0;
    }
    if (warp == kZProd) umma::tmem_alloc(tmem_slot, 512);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
        if (*dead) return false;
        if (z_wait(bar, parity)) return true;
        atomicOr(err, kTcErrBit);
        *dead = 1;
        return false;
    };
    auto warp_wait = [&](uint32_t bar, uint32_t parity) -> bool {
        bool ok = true;
        if (lane == 0) ok = wait(bar, parity);
        return __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    };
    auto arrive = [&](uint32_t bar) {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
    };

    /* the descriptor slots, and their turn */
    uint32_t slot = 0, turn = 0;
    auto next_slot = [&]() {
        if (++slot == kZSlots) {
            slot = 0;
            turn ^= 1;
        }
    };
    auto desc = [&]() -> unsigned char * { return sm + kZOffD + slot * kZDesc; };

    if (warp < kZProd) {
        /* ---- producers ---- */
        uint32_t np = 0, nt = 0, nq = 0, na = 0;   /* slices of P, tiles, slices of Q, accumulators so far */
        const int grp = warp >> 2, wg = warp & 3;  /* slices of Q of parity grp */
        bool ok = true;
        for (long long tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, nt++) {
            if (!(ok = warp_wait(dfull(slot), turn))) break;
            const ZTile &ti = *reinterpret_cast<const ZTile *>(desc());
            const long long *const poff = reinterpret_cast<const long long *>(desc() + 128);
            const long long *const kp = poff + 2 * kZP, *const kq = kp + kZGroup;
            const int kn = ti.kn, steps = ti.steps, rows = ti.rows;
            const bool several = kn > kZK;      /* chunks of k: exponents over all of them */
            const int base = 16 * warp;         /* this warp's rows of P */
            int *const ep = eP + (nt & 3) * kZP + base;
            for (int c0 = 0; ok && c0 < kn; c0 += kZK, np++) {
                const int kc = min(kZK, kn - c0);
                const int lpr = kc <= 16 ? 8 : kc <= 32 ? 16 : 32, rpp = 32 / lpr, gap = 8 / rpp;
                const int kl = lane & (lpr - 1), sub = lane / lpr, k = 2 * kl;
                {
                    const double *const src = ti.p;
                    if (several && c0 == 0) {
                        for (int r = 0; r < 16; r++) {
                            const long long o = poff[base + r];
                            int h = 0;
                            for (int kk = lane; o >= 0 && kk < kn; kk += 32)
                                h = max(h, z_top(__ldg(src + o + kp[kk])));
                            __syncwarp();
                            const int e = z_exp(h, 32);
                            if (lane == 0) ep[r] = e;
                        }
                        __syncwarp();
                    }
                    const long long k0 = k < kc ? kp[c0 + k] : -1, k1 = k + 1 < kc ? kp[c0 + k + 1] : -1;
                    /* warps without rows slice nothing: what their planes give is not stored */
                    const int passes = base < rows ? 16 / rpp : 4;
                    for (int p0 = 0; p0 < passes; p0 += 4) {   /* four passes' loads in flight */
                        double x[4][2];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const int p = p0 + u, row = (p / gap) * 8 + p % gap + sub * gap;
                            const long long o = base < rows ? poff[base + row] : -1;
                            x[u][0] = o >= 0 && k0 >= 0 ? __ldg(src + o + k0) : 0.0;
                            x[u][1] = o >= 0 && k1 >= 0 ? __ldg(src + o + k1) : 0.0;
                        }
                        /* the planes are free once the MMAs that read them are done */
                        if (p0 == 0 && !(ok = warp_wait(pfree, (np & 1) ^ 1))) break;
                        if (base >= rows) break;
#pragma unroll
                        for (int u = 0; u < 4; u += 2) {
                            const int p = p0 + u, r = (p / gap) * 8 + p % gap + sub * gap;
                            const int t = ((p + 1) / gap) * 8 + (p + 1) % gap + sub * gap;
                            const int2 e = z_slice(x[u][0], x[u][1], x[u + 1][0], x[u + 1][1], lpr,
                                                   sm + umma::kmajor_off(base + r, k, 0),
                                                   sm + umma::kmajor_off(base + t, k, 0), kZPlane,
                                                   several ? ep[r] : -1, several ? ep[t] : -1);
                            if (!several && kl == 0) { ep[r] = e.x; ep[t] = e.y; }
                        }
                    }
                }
                if (!ok) break;
                umma::fence_async_smem();
                arrive(pfull);
                /* Q: 16 rows per step, four per warp of the step's group (two or
                 * one pass for short k); the group's next step is loaded as this
                 * one is sliced */
                const int g8 = (wg >> 1) * 8 + (wg & 1) * (4 / rpp), r0 = g8 + sub * gap, passes = 4 / rpp;
                const double *const src = ti.q;
                const long long k0 = k < kc ? kq[c0 + k] : -1, k1 = k + 1 < kc ? kq[c0 + k + 1] : -1;
                auto load = [&](uint32_t a, int p, double (&x)[4][2]) {   /* passes p, p + 1 of accumulator a's step */
                    const ZRow *const rq = rows_of(a);
#pragma unroll
                    for (int u = p; u < p + 2; u++) {
                        const long long o = u < passes ? rq[r0 + u].src : -1;
                        x[u][0] = o >= 0 && k0 >= 0 ? __ldg(src + o + k0) : 0.0;
                        x[u][1] = o >= 0 && k1 >= 0 ? __ldg(src + o + k1) : 0.0;
                    }
                };
                int eg[4] = {-1, -1, -1, -1};
                double x[4][2];
                const int st0 = (int)((nq & 1) ^ (uint32_t)grp);   /* the group's first step */
                if (st0 < steps) {
                    const uint32_t a0 = na + (uint32_t)st0;
                    if (!(ok = warp_wait(rfull(a0), rturn(a0)))) break;
                    load(a0, 0, x);
                    load(a0, 2, x);
                }
                if (several && st0 < steps) {
                    const ZRow *const rq = rows_of(na);
#pragma unroll
                    for (int p = 0; p < 4; p++) {
                        /* this lane's row of the slicing pass p */
                        const long long o = p < passes ? rq[r0 + p].src : -1;
                        int h = 0;
                        for (int kk = kl; o >= 0 && kk < kn; kk += lpr)
                            h = max(h, z_top(__ldg(src + o + kq[kk])));
                        __syncwarp();
                        eg[p] = z_exp(h, lpr);
                    }
                }
                for (int st = st0; st < steps; st += 2) {
                    const uint32_t n = nq + (uint32_t)st, a = na + (uint32_t)st;
                    const bool more = st + 2 < steps;
                    ok = warp_wait(qfree(grp), ((n >> 1) & 1) ^ 1) && (!more || warp_wait(rfull(a + 2), rturn(a + 2)));
                    if (!ok) break;
                    unsigned char *const dst = sm + kZOffQ + (uint32_t)grp * kZQBuf;
                    ZRow *const rq = rows_of(a);
#pragma unroll
                    for (int p = 0; p < 4; p += 2) {
                        if (p >= passes) break;
                        /* one pass: the second row is the first again */
                        const bool two = passes > 1;
                        const int u = r0 + p, v = two ? u + 1 : u;
                        const int2 e = z_slice(x[p][0], x[p][1], two ? x[p + 1][0] : x[p][0], two ? x[p + 1][1] : x[p][1],
                                               lpr, dst + umma::kmajor_off(u, k, 0), dst + umma::kmajor_off(v, k, 0),
                                               kZQ * kZK * 2, eg[p], two ? eg[p + 1] : eg[p]);
                        if (kl == 0) { rq[u].e = e.x; rq[v].e = e.y; }
                        if (more) load(a + 2, p, x);
                    }
                    umma::fence_async_smem();
                    arrive(qfull(grp));
                }
                nq += (uint32_t)steps;
            }
            na += (uint32_t)steps;
            arrive(dfree(slot));
            next_slot();
        }
    } else if (warp == kZProd + 1) {
        /* ---- descriptors: tiles, and the rows of Q, a row per lane (of 16) ---- */
        uint32_t na = 0;
        bool ok = true;
        for (long long tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
            const ZTile ti = z_tile(tile, tasks, tile_start, tile_task);
            const GemmTask &T = *ti.task;
            const ZSide A = z_side_a(T), B = z_side_b(T), Cr = z_side_c_rows(T), Cc = z_side_c_cols(T);
            const ZSide P = ti.wide ? A : B, Q = ti.wide ? B : A, Op = ti.wide ? Cr : Cc, Oq = ti.wide ? Cc : Cr;
            if (!(ok = warp_wait(dfree(slot), turn ^ 1))) break;
            long long *const poff = reinterpret_cast<long long *>(desc() + 128), *const pout = poff + kZP;
            long long *const kp = pout + kZP, *const kq = kp + kZGroup;
#pragma unroll
            for (int r = lane; r < kZP; r += 32) {
                poff[r] = P.row(ti.p0 + r);
                pout[r] = Op.row(ti.p0 + r);
            }
            for (int k = lane; k < ti.kn; k += 32) {
                kp[k] = P.k(ti.k0 + k);
                kq[k] = Q.k(ti.k0 + k);
            }
            if (lane == 0) *reinterpret_cast<ZTile *>(desc()) = ti;
            arrive(dfull(slot));
            next_slot();
            for (int st = 0; st < ti.steps; st++, na++) {
                const long long i = ti.q0 + (long long)st * kZQ + lane, src = Q.row(i), off = Oq.row(i);
                if (!(ok = warp_wait(rfree(na), rturn(na) ^ 1))) break;
                if (lane < kZQ) {
                    ZRow &r = rows_of(na)[lane];
                    r.src = src;
                    r.off = off;
                }
                arrive(rfull(na));
            }
        }
    } else if (warp == kZProd) {
        /* ---- MMA issue: one thread ---- */
        uint32_t np = 0, nq = 0, na = 0;   /* slices of P, steps, drained accumulators so far */
        uint32_t last_bar = 0, last_par = 0;
        bool any = false, ok = true;
        for (long long tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
            if (!(ok = warp_wait(dfull(slot), turn))) break;
            const ZTile &td = *reinterpret_cast<const ZTile *>(desc());
            const int kn = td.kn, steps = td.steps;
            arrive(dfree(slot));
            next_slot();
            for (int c0 = 0; ok && c0 < kn; c0 += kZK, np++) {
                const uint32_t nkk = (uint32_t)(min(kZK, kn - c0) + 15) / 16;
                const bool last = c0 + kZK >= kn;   /* a later chunk adds to the same accumulator */
                ok = warp_wait(pfull, np & 1);
                for (int st = 0; ok && st < steps; st++, nq++) {
                    const uint32_t b = nq & 1, ab = na & 1;
                    ok = warp_wait(qfull(b), (nq >> 1) & 1) && (c0 > 0 || warp_wait(afree(ab), ((na >> 1) & 1) ^ 1));
                    if (!ok) break;
                    if (lane == 0) {
                        umma::fence_after_sync();
                        const uint64_t ad = umma::sdesc(sbase, 16, 1024), bd = umma::sdesc(sbase + kZOffQ + (uint32_t)b * kZQBuf, 16, 1024);
#pragma unroll 1   /* short code: the roles share the instruction cache */
                        for (uint32_t kk = 0; kk < nkk; kk++) {
                            uint32_t idesc = umma::idesc_bf16(kZP, kZQ * kZD, 0, 0);
#pragma unroll 1
                            for (uint32_t i = 0; i < kZD; i++) {
                                umma::mma_bf16(tmem + 256u * ab + kZQ * i, ad + ((i * kZPlane + kk * 32u) >> 4), bd + kk * 2u, idesc,
                                               c0 > 0 || kk > 0 || i > 0);
                                idesc -= (uint32_t)(kZQ / 8) << 17;   /* 16 columns fewer */
                            }
                        }
                        umma::mma_commit(qfree(b));
                        last_bar = qfree(b);
                        last_par = (nq >> 1) & 1;
                        if (st + 1 == steps) umma::mma_commit(pfree);
                        if (last) umma::mma_commit(afull(ab));
                        any = true;
                    }
                    __syncwarp();
                    if (last) na++;
                }
            }
        }
        /* after an expiry, MMAs may still be in flight: wait (bounded) for the last commit */
        if (lane == 0 && *dead && any) (void)z_wait(last_bar, last_par);
    } else {
        /* ---- epilogue: lane quarter warp % 4, kZCols of the step's 16 rows of Q ---- */
        const int w = warp - kZProd - 2, q = warp & 3, part = kZCols * (w >> 2);
        uint32_t nt = 0, na = 0;
        bool ok = true;
        for (long long tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, nt++) {
            if (!(ok = warp_wait(dfull(slot), turn))) break;
            const ZTile &ti = *reinterpret_cast<const ZTile *>(desc());
            const long long *const poff = reinterpret_cast<const long long *>(desc() + 128);
            const long long *const kp = poff + 2 * kZP, *const kq = kp + kZGroup;
            const long long pout = poff[kZP + 32 * q + lane];
            double *const mine = ti.out + pout;
            const int steps = ti.steps;
            const bool live = 32 * q < ti.rows;
            for (int st = 0; st < steps; st++, na++) {
                const int b = (int)(na & 1);
                if (!(ok = warp_wait(afull(b), (na >> 1) & 1))) break;
                umma::fence_after_sync();
                const int ep = eP[(nt & 3) * kZP + 32 * q + lane], es = ep - 2 * 1022 - 86;
                const ZRow *const rq = rows_of(na) + part;
                const uint32_t tb = tmem + (uint32_t)(256 * b + part) + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
                for (int c0 = 0; live && c0 < kZCols && rq[c0].off >= 0; c0 += 4) {
                    uint32_t r[kZD][4];
#pragma unroll
                    for (int l = 0; l < kZD; l++)
                        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                                     : "=r"(r[l][0]), "=r"(r[l][1]), "=r"(r[l][2]), "=r"(r[l][3])
                                     : "r"(tb + (uint32_t)(kZQ * l + c0))
                                     : "memory");
                    umma::tmem_wait_ld();
                    unsigned redo[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const long long qo = rq[c0 + c].off;
                        const int eq = rq[c0 + c].e;
                        uint32_t lv[kZD];
#pragma unroll
                        for (int l = 0; l < kZD; l++) lv[l] = r[l][c];
                        bool sure;
                        const double v = z_combine(lv, es + eq, sure);
                        /* a row of zeros (exponent 0) adds nothing to finite ones */
                        const bool finite = max(ep, eq) < kZBadExp, out = pout >= 0 && qo >= 0 && (min(ep, eq) > 0 || !finite);
                        sure = sure && finite;
                        redo[c] = __ballot_sync(0xffffffffu, out && !sure);
                        if (out && sure) red_global(mine + qo, v);
                    }
                    if ((redo[0] | redo[1] | redo[2] | redo[3]) == 0) continue;
#pragma unroll 1
                    for (int c = 0; c < 4; c++) {
                        const ZRow &rc = rq[c0 + c];
                        const double *const bq = ti.q + rc.src;
                        unsigned m = c == 0 ? redo[0] : c == 1 ? redo[1] : c == 2 ? redo[2] : redo[3];
                        while (m != 0) {   /* rows times the column in FP64, lanes along k, four rows at a time */
                            int j[4];
                            double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                j[u] = m ? __ffs(m) - 1 : -1;
                                m &= m - 1;
                            }
                            for (int k = lane; k < ti.kn; k += 32) {
                                const double y = __ldg(bq + kq[k]);
                                const double *const a = ti.p + kp[k];
#pragma unroll
                                for (int u = 0; u < 4; u++)
                                    if (j[u] >= 0) t[u] = fma(__ldg(a + poff[32 * q + j[u]]), y, t[u]);
                            }
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                                for (int u = 0; u < 4; u++) t[u] += __shfl_xor_sync(0xffffffffu, t[u], o);
#pragma unroll
                            for (int u = 0; u < 4; u++)
                                if (lane == j[u]) red_global(mine + rc.off, t[u]);
                        }
                    }
                }
                umma::fence_before_sync();
                arrive(afree(b));
                arrive(rfree(na));
            }
            arrive(dfree(slot));
            next_slot();
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kZProd) umma::tmem_dealloc(tmem, 512);
}

}  // namespace h2g

#endif
