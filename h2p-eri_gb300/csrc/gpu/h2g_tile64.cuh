/*
 * FP64-mode tile kernel: the products of a stored matrix with FP64 vectors,
 * in 60-bit fixed point on the integer pipe.
 *
 * What bounds it. GB300 runs 2 FP64 FMAs (or conversions) per clock and SM
 * (measured), so a bi-product of FP64 FMAs takes 1 clock per stored element
 * and SM, 2.7 times what HBM needs to deliver it (21 bytes per clock and SM).
 * 32 x 32 + 64 bit integer multiply-adds run at 54 per clock and SM (measured),
 * so the stored entries are two signed limbs in the 8 bytes of the double,
 *   a = (ah 2^30 + al) 2^(e - 60), e the exponent of the largest entry of the
 *       matrix row in the 128-column strip (|a| < 2^e), |ah| <= 2^30, |al| <= 2^29;
 * the inputs become
 *   x = (xh 2^30 + xl) 2^(E - 58), E the exponent of the largest input of the
 *       tile (N side: of its columns; T side: of its rows, each times its
 *       2^e), |xh| <= 2^28, |xl| <= 2^29;
 * and a x is ah xh 2^60 + (ah xl + al xh) 2^30, three multiply-adds; al xl (below
 * 2^-60 of the largest product) is left out. Eight products fit in 64 bits; the
 * sums beyond that are kept in 96 bits (T side, a warp's 128 rows) or 64 + 32 bits
 * (N side, over the lanes). So a tile's sums are exact but for the entries'
 * rounding to 2^-61 and the inputs' to 2^-59 of the largest, against a
 * rounding to 2^-53 of the running sum at every step of an FP64 chain. (With
 * two bits less on each side nothing has to be folded inside a tile, 7 %
 * faster, but the error of J on C30H62 rose from 1.9e-16 to 3.8e-16, above
 * that of FP64 FMAs, 2.3e-16.)
 *
 * A tile whose inputs hold an infinity or a NaN, or with a row that does (its
 * strip keeps the doubles), takes FP64 FMAs on the decoded entries instead.
 *
 * Layout: four warps multiply; a fifth copies one row of the tile per lane
 * (bulk copies of up to 1 KB) into a ring of three 16 KB stages, with an
 * mbarrier per stage and direction (bounded waits). Four CTAs per SM. NV
 * vectors share a tile's copies. (Eight warps and two CTAs per SM: 650
 * against 531 us for the C30H62 J build, at the same arithmetic; a CTA's
 * serial part weighs less with four.)
 *
 * Measured, C30H62 (QR 1e-8, 1.84 GB stored): 1170 us per J build with FP64
 * FMAs (1.6 TB/s), 482 us (3.8 TB/s) here; five vectors on C13H28 1742 and
 * 763 us.
 */
#ifndef H2G_TILE64_CUH
#define H2G_TILE64_CUH

namespace h2g {

constexpr int kFxWarps = 4;                                  /* multiplying warps, 4 rows of a stage each */
constexpr int kFxRows = 4 * kFxWarps;                        /* rows per stage */
constexpr int kFxStages = 3;
constexpr int kFxStageBytes = kFxRows * kTileCols * 8;
constexpr int kFxMath = 32 * kFxWarps, kFxThreads = kFxMath + 32;
constexpr int kFxQ = kChunkRows / kFxMath;
constexpr int kFxBits = 60, kFxInBits = 58, kFxLimb = 30;
constexpr int16_t kFxBadExp = 32767;
constexpr int kFxNone = -30000;                              /* exponent of all-zero inputs */

template <int NV> struct FxSmem {
    unsigned char ring[kFxStages][kFxStageBytes];
    int top0[NV][4], top1[NV][4];    /* exponents of the largest inputs, per warp */
    int2 x0[NV][kTileCols];          /* inputs: xh, xl */
    int2 x1[NV][kChunkRows];
    int16_t rexp[kChunkRows];
    unsigned long long full[kFxStages], empty[kFxStages];
    int slow, dead;
};

/* |x| < 2^fx_exp (1025 for infinities and NaN) */
__device__ __forceinline__ int fx_exp(double x)
{
    return max((int)(((unsigned)__double2hiint(x) & 0x7fffffffu) >> 20), 1) - 1022;
}
/* x 2^s to the nearest integer, |x 2^s| < 2^60 */
__device__ __forceinline__ long long fx_fixed(double x, int s)
{
    const long long b = __double_as_longlong(x);
    const int e = (int)((unsigned long long)b >> 52) & 0x7ff;
    long long m = (b & 0xfffffffffffffLL) | (e ? 1LL << 52 : 0LL);
    const int sh = max(e, 1) - 1075 + s;   /* <= 7 */
    if (sh >= 0) m <<= sh;
    else if (sh >= -62) m = (m + (1LL << (-sh - 1))) >> -sh;
    else m = 0;
    return b < 0 ? -m : m;
}
__device__ __forceinline__ int2 fx_limbs(long long v)
{
    const int h = (int)((v + (1LL << (kFxLimb - 1))) >> kFxLimb);
    return make_int2(h, (int)v - (int)((unsigned)h << kFxLimb));
}
/* x 2^s, the exponent added in place where the result is a normal number */
__device__ __forceinline__ double fx_scale(double x, int s)
{
    const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
    if (e + s >= 1 && e + s <= 2046 && e != 0) return __hiloint2double(hi + (int)((unsigned)s << 20), __double2loint(x));
    return scalbn(x, s);
}

/* One 128-column strip of a stored matrix: doubles to limbs in place, and the
 * exponent of every row. */
struct FxStrip {
    uint64_t a;
    int32_t ld, nrow, nc;
    uint32_t e_off;
};
__global__ void __launch_bounds__(256) k_to_fixed(const FxStrip *__restrict__ strips, int n, double *__restrict__ arena,
                                                  int16_t *__restrict__ rexp)
{
    if ((int)blockIdx.x >= n) return;
    const FxStrip s = strips[blockIdx.x];
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < s.nrow; r += 8) {
        double *row = arena + s.a + (size_t)r * s.ld;
        double v[4];
        int e = -1021;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = lane + 32 * k < s.nc ? row[lane + 32 * k] : 0.0;
            e = max(e, fx_exp(v[k]));
        }
        e = __reduce_max_sync(0xffffffffu, e);
        if (lane == 0) rexp[s.e_off + r] = e == 1025 ? kFxBadExp : (int16_t)e;
        if (e == 1025) continue;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (lane + 32 * k < s.nc)
                reinterpret_cast<int2 *>(row)[lane + 32 * k] = fx_limbs(fx_fixed(v[k], kFxBits - e));
    }
}

__device__ __forceinline__ void fx_bulk(unsigned dst, const void *src, unsigned bytes, unsigned bar, bool once)
{
    if (once) {
        unsigned long long pol;
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                     ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(pol)
                     : "memory");
    } else {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                     : "memory");
    }
}

__device__ __forceinline__ void fx_mad(long long &s, int a, int x)   /* s += a x */
{
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s) : "r"(a), "r"(x));
}

/* Sum of four values per lane over the warp by recursive halving: lane l ends
 * with the sum of value fx_sum4_row(l). */
__device__ __forceinline__ int fx_sum4_row(int lane) { return ((lane & 16) ? 2 : 0) + ((lane & 8) ? 1 : 0); }
template <typename T>
__device__ __forceinline__ T fx_sum4(const T (&s)[4], int lane)
{
    const bool b16 = lane & 16, b8 = lane & 8;
    const T a = (b16 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, b16 ? s[0] : s[2], 16);
    const T b = (b16 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, b16 ? s[1] : s[3], 16);
    T v = (b8 ? b : a) + __shfl_xor_sync(0xffffffffu, b8 ? a : b, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

/* 96-bit accumulator w += h 2^30 + m */
__device__ __forceinline__ void fx_add96(unsigned (&w)[3], long long h, long long m)
{
    const unsigned h0 = (unsigned)h, h1 = (unsigned)(h >> 32);
    asm("{.reg .u32 a0, a1, a2, m0, m1, m2;\n\t"
        "shl.b32 a0, %3, 30;\n\tshf.l.wrap.b32 a1, %3, %4, 30;\n\tshr.s32 a2, %4, 2;\n\t"
        "mov.b64 {m0, m1}, %5;\n\tshr.s32 m2, m1, 31;\n\t"
        "add.cc.u32 a0, a0, m0;\n\taddc.cc.u32 a1, a1, m1;\n\taddc.u32 a2, a2, m2;\n\t"
        "add.cc.u32 %0, %0, a0;\n\taddc.cc.u32 %1, %1, a1;\n\taddc.u32 %2, %2, a2;}"
        : "+r"(w[0]), "+r"(w[1]), "+r"(w[2])
        : "r"(h0), "r"(h1), "l"(m));
}

/* CTA (g, y): tile y with vectors g NV .. g NV + NV - 1. Warp w multiplies
 * rows [4 w, 4 w + 4) of a stage; a lane owns columns 2 l, 2 l + 1, 64 + 2 l,
 * 65 + 2 l. */
template <int NV>
__global__ void __launch_bounds__(kFxThreads, NV == 1 ? 4 : 3)
k_tile_fx(const Tile *__restrict__ tiles, const double *__restrict__ arena, const int16_t *__restrict__ rexp,
          const __grid_constant__ VecArgs va, int nvec, unsigned *err)
{
    extern __shared__ __align__(128) unsigned char fx_raw[];
    FxSmem<NV> &sm = *reinterpret_cast<FxSmem<NV> *>(fx_raw);
    const Tile t = tiles[blockIdx.y];
    const int v0 = blockIdx.x * NV, nv = min(NV, nvec - v0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nr = t.nr, nc = t.nc, nstage = (nr + kFxRows - 1) / kFxRows;
    volatile int *dead = &sm.dead;

    if (tid == 0) {
        for (int i = 0; i < kFxStages; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.full[i])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&sm.empty[i])), "n"(kFxWarps) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sm.slow = 0;
        sm.dead = 0;
    }
    __syncthreads();

    if (warp == kFxWarps) {
        /* ---- copies ---- */
        const unsigned rb = (unsigned)((nc * 8 + 15) & ~15);
        const double *row = arena + t.a + (size_t)lane * t.ld;
        int issued = 0;
        for (int k = 0; k < nstage; k++) {
            const int slot = k % kFxStages;
            if (k >= kFxStages && !mbar_wait(smem_addr(&sm.empty[slot]), (unsigned)((k / kFxStages - 1) & 1))) {
                atomicOr(err, 1u);
                *dead = 1;
            }
            if (__shfl_sync(0xffffffffu, *dead, 0)) break;
            const unsigned bar = smem_addr(&sm.full[slot]);
            const int rows = min(kFxRows, nr - k * kFxRows);
            if (lane == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(rb * rows) : "memory");
            __syncwarp();
            if (lane < rows)
                fx_bulk(smem_addr(sm.ring[slot]) + lane * (kTileCols * 8), row, rb, bar, gridDim.x == 1);
            row += (size_t)kFxRows * t.ld;
            issued = k + 1;
        }
        /* no copy may be in flight when the CTA ends */
        if (*dead)
            for (int k = max(0, issued - kFxStages); k < issued; k++)
                (void)mbar_wait(smem_addr(&sm.full[k % kFxStages]), (unsigned)((k / kFxStages) & 1));
        return;
    }

    const bool opN = t.k_out0 != VK_NONE, opT = t.k_out1 != VK_NONE;
    const int col[4] = {2 * lane, 2 * lane + 1, 64 + 2 * lane, 65 + 2 * lane};

    /* ---- inputs to fixed point: thread i takes column i (N side) and rows
     * i, i + kFxMath, .. (T side) ---- */
    int2 xn[NV][4];
    int en[NV], et[NV];
    {
        static_assert(kFxMath == kTileCols, "a thread per column");
        bool bad = false;
        double x0[NV], x1[NV][kFxQ];
        int er[kFxQ];
#pragma unroll
        for (int v = 0; v < NV; v++) {
            x0[v] = opN && v < nv && tid < nc ? vec_ptr(va, t.k_in0, t.in0, v0 + v)[tid] : 0.0;
#pragma unroll
            for (int q = 0; q < kFxQ; q++) {
                const int r = tid + q * kFxMath;
                x1[v][q] = opT && v < nv && r < nr ? vec_ptr(va, t.k_in1, t.in1, v0 + v)[r] : 0.0;
            }
        }
#pragma unroll
        for (int q = 0; q < kFxQ; q++) {
            const int r = tid + q * kFxMath;
            er[q] = r < nr ? (int)rexp[t.e_off + r] : 0;
            sm.rexp[r] = (int16_t)er[q];
            bad |= er[q] == kFxBadExp;
        }
#pragma unroll
        for (int v = 0; v < NV; v++) {
            int e = fx_exp(x0[v]);
            bad |= e == 1025;
            e = __reduce_max_sync(0xffffffffu, x0[v] != 0.0 ? e : kFxNone);
            int top = kFxNone;
#pragma unroll
            for (int q = 0; q < kFxQ; q++) {
                const int f = fx_exp(x1[v][q]);
                bad |= f == 1025;
                if (x1[v][q] != 0.0) top = max(top, f + er[q]);
            }
            top = __reduce_max_sync(0xffffffffu, top);
            if (lane == 0) { sm.top0[v][warp] = e; sm.top1[v][warp] = top; }
        }
        if (bad) sm.slow = 1;
        asm volatile("bar.sync 1, %0;" ::"n"(kFxMath) : "memory");
#pragma unroll
        for (int v = 0; v < NV; v++) {
            const int4 a = *reinterpret_cast<const int4 *>(sm.top0[v]), b = *reinterpret_cast<const int4 *>(sm.top1[v]);
            en[v] = max(max(a.x, a.y), max(a.z, a.w));
            et[v] = max(max(b.x, b.y), max(b.z, b.w));
            if (opN) sm.x0[v][tid] = fx_limbs(x0[v] != 0.0 ? fx_fixed(x0[v], kFxInBits - en[v]) : 0LL);
            if (opT) {
#pragma unroll
                for (int q = 0; q < kFxQ; q++)
                    if (warp * 32 + q * kFxMath < nr)   /* the warp has rows that are read */
                        sm.x1[v][tid + q * kFxMath] =
                            fx_limbs(x1[v][q] != 0.0 ? fx_fixed(x1[v][q], er[q] + kFxInBits - et[v]) : 0LL);
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kFxMath) : "memory");
#pragma unroll
        for (int v = 0; v < NV; v++)
#pragma unroll
            for (int k = 0; k < 4; k++) xn[v][k] = opN ? sm.x0[v][col[k]] : make_int2(0, 0);
    }
    const bool slow = *reinterpret_cast<volatile int *>(&sm.slow) != 0;

    auto wait_full = [&](int k) -> bool {
        const unsigned bar = smem_addr(&sm.full[k % kFxStages]), par = (unsigned)((k / kFxStages) & 1);
        if (*dead) return false;
        if (mbar_try(bar, par) || mbar_wait(bar, par)) return true;
        atomicOr(err, 1u);
        *dead = 1;
        return false;
    };
    auto release = [&](int k) {
        __syncwarp();
        if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&sm.empty[k % kFxStages])) : "memory");
    };

    /* a warp that gives up a wait still meets the others at the barriers below */
    if (!slow) {
        long long th[NV][4], tm[NV][4];   /* T side: column sums of the warp's rows, two stages */
        unsigned tw[NV][4][3];            /* of which are added up in 64 bits, then in 96      */
        long long nh[NV];                 /* N side: row sums of up to 8 stages, those of */
        unsigned nl[NV];                  /* stage k on the lanes with lane % 8 = k % 8   */
#pragma unroll
        for (int v = 0; v < NV; v++) {
            nh[v] = 0;
            nl[v] = 0;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                th[v][c] = tm[v][c] = 0;
                tw[v][c][0] = tw[v][c][1] = tw[v][c][2] = 0;
            }
        }
        for (int k = 0; k < nstage; k++) {
            if (!wait_full(k)) break;
            const int r0 = k * kFxRows + 4 * warp;
            if (r0 < nr) {   /* warp-uniform */
                const unsigned char *buf = sm.ring[k % kFxStages] + 4 * warp * (kTileCols * 8) + 16 * lane;
                int a[4][8];   /* (ah, al) of the four columns */
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    *reinterpret_cast<int4 *>(&a[i][0]) = *reinterpret_cast<const int4 *>(buf + i * (kTileCols * 8));
                    *reinterpret_cast<int4 *>(&a[i][4]) = *reinterpret_cast<const int4 *>(buf + i * (kTileCols * 8) + 512);
                }
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    if (opN) {
                        long long hi[4];
                        unsigned lo[4];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            long long h = 0, m = 0;
#pragma unroll
                            for (int c = 0; c < 4; c++) {
                                fx_mad(h, a[i][2 * c], xn[v][c].x);
                                fx_mad(m, a[i][2 * c], xn[v][c].y);
                                fx_mad(m, a[i][2 * c + 1], xn[v][c].x);
                            }
                            /* the row's sum, 16 hi + lo 2^-22 in units of 2^60 */
                            h += m >> kFxLimb;
                            hi[i] = h >> 4;
                            lo[i] = __funnelshift_r((unsigned)m << 2, (unsigned)h, 4) >> 6;
                        }
                        const long long sh = fx_sum4(hi, lane);
                        const unsigned sl = fx_sum4(lo, lane);
                        if ((lane & 7) == (k & 7)) { nh[v] = sh; nl[v] = sl; }
                    }
                    if (opT) {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const int2 x = sm.x1[v][r0 + i];
#pragma unroll
                            for (int c = 0; c < 4; c++) {
                                fx_mad(th[v][c], a[i][2 * c], x.x);
                                fx_mad(tm[v][c], a[i][2 * c], x.y);
                                fx_mad(tm[v][c], a[i][2 * c + 1], x.x);
                            }
                        }
                    }
                }
            }
            release(k);
            if ((k & 1) || k + 1 == nstage) {
#pragma unroll
                for (int v = 0; v < NV; v++)
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        fx_add96(tw[v][c], th[v][c], tm[v][c]);
                        th[v][c] = tm[v][c] = 0;
                    }
            }
            if (opN && ((k & 7) == 7 || k + 1 == nstage)) {
                const int row = ((k & ~7) + (lane & 7)) * kFxRows + 4 * warp + fx_sum4_row(lane);
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    if ((lane & 7) > (k & 7) || row >= nr || v >= nv) continue;
                    const double s = fma((double)nl[v], 0x1p-26, (double)nh[v]);   /* units of 2^64 */
                    atomicAdd(vec_ptr(va, t.k_out0, t.out0, v0 + v) + row,
                              fx_scale(s, sm.rexp[row] + en[v] + 2 * kFxLimb + 4 - kFxBits - kFxInBits));
                }
            }
        }
        if (opT) {
            /* over the warps, through the ring (every copy has landed): a
             * sum, in units of 2^30, is 2^36 h + 2^4 l */
            asm volatile("bar.sync 1, %0;" ::"n"(kFxMath) : "memory");
            long long (*rh)[kFxWarps][kTileCols] = reinterpret_cast<long long (*)[kFxWarps][kTileCols]>(sm.ring[0]);
            unsigned (*rl)[kFxWarps][kTileCols] = reinterpret_cast<unsigned (*)[kFxWarps][kTileCols]>(sm.ring[1]);
#pragma unroll
            for (int v = 0; v < NV; v++)
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const unsigned *w = tw[v][c];
                    rh[v][warp][col[c]] = (long long)(((unsigned long long)w[2] << 32) | w[1]) >> 4;
                    rl[v][warp][col[c]] = __funnelshift_r(w[0], w[1], 4);
                }
            asm volatile("bar.sync 1, %0;" ::"n"(kFxMath) : "memory");
#pragma unroll
            for (int v = 0; v < NV; v++) {
                if (v >= nv || tid >= nc) continue;
                long long h = 0;
                unsigned long long l = 0;
#pragma unroll
                for (int w = 0; w < kFxWarps; w++) {
                    h += rh[v][w][tid];
                    l += rl[v][w][tid];
                }
                const double s = fma((double)l, 0x1p-32, (double)h);   /* units of 2^66 */
                atomicAdd(vec_ptr(va, t.k_out1, t.out1, v0 + v) + tid,
                          fx_scale(s, et[v] + kFxLimb + 36 - kFxBits - kFxInBits));
            }
        }
    } else {
        for (int k = 0; k < nstage; k++) {
            if (!wait_full(k)) break;
            const int r0 = k * kFxRows + 4 * warp;
            const unsigned char *buf = sm.ring[k % kFxStages] + 4 * warp * (kTileCols * 8);
            for (int i = 0; i < 4 && r0 + i < nr; i++) {
                const int e = sm.rexp[r0 + i];
                double a[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int2 p = reinterpret_cast<const int2 *>(buf + i * (kTileCols * 8))[col[c]];
                    a[c] = e == kFxBadExp ? __hiloint2double(p.y, p.x)
                                          : scalbn(fma((double)p.x, 0x1p30, (double)p.y), e - kFxBits);
                    if (col[c] >= nc) a[c] = 0.0;
                }
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    if (v >= nv) continue;
                    if (opN) {
                        const double *in0 = vec_ptr(va, t.k_in0, t.in0, v0 + v);
                        double s = 0.0;
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (col[c] < nc) s = fma(a[c], in0[col[c]], s);
                        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                        if (lane == 0) atomicAdd(vec_ptr(va, t.k_out0, t.out0, v0 + v) + r0 + i, s);
                    }
                    if (opT) {
                        const double x = vec_ptr(va, t.k_in1, t.in1, v0 + v)[r0 + i];
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if (col[c] < nc) atomicAdd(vec_ptr(va, t.k_out1, t.out1, v0 + v) + col[c], a[c] * x);
                    }
                }
            }
            release(k);
        }
    }
}

}  // namespace h2g

#endif
