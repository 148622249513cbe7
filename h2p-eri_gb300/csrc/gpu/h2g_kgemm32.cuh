/*
 * The mixed mode's exchange products on the tensor cores, persistent form (the
 * default; arithmetic as k_gemm_tc: exact bf16 thirds of every FP32 value, six
 * products, h h and the corrections in accumulators of their own, full K in
 * order before one addition to C).
 *
 * What bounds it. An MMA step (128 x 128 x 64, six products) takes 1500 clocks
 * of the tensor pipe; gathering and slicing its 16384 values is most of the
 * rest. With a thread per row every load touched 32 lines, 16 thousand L1 tag
 * accesses per step, 13 thousand clocks; so the lanes of a producer warp run
 * along k (8, 16 or 32 lanes per row, by the step's length): two loads of three
 * lines and three 128-byte stores per row. The code per row has to be short (a
 * version that loaded the next step while it stored this one took 125
 * instructions per row and 26 ms for the coupling products of 8 CH4, 15 before,
 * 11 now), so everything with dependent loads (tile -> task -> index lists ->
 * offsets) is done by one warp ahead of the others: a descriptor per tile (row
 * addresses of both sides, offsets in C) and the offsets of k per step, in
 * rings. Rows and columns past the tile's end are not sliced, multiplied (in
 * steps of 16) or drained. Waits are suspended, not spun (z_wait), and bounded.
 *
 * Roles: warps 0-15 producers, 16 MMA issue (one thread), 17 descriptors, 18-21
 * epilogue on one of two TMEM buffers (256 columns: h h, corrections). Two
 * 96 KB stages.
 * Measured: mixed K of C30H62 199 -> 133 ms, of 8 CH4 19.9 -> 15.2 ms.
 */
#ifndef H2G_KGEMM32_CUH
#define H2G_KGEMM32_CUH

namespace h2g {

constexpr int kMProd = 16, kMEpi = 4, kMThreads = 32 * (kMProd + 2 + kMEpi);
constexpr int kMSlots = 4, kMRing = 4;                         /* tile descriptors, steps of k offsets */
constexpr uint32_t kMStage = 6 * kTcSlice;
constexpr uint32_t kMDesc = 64 + 4 * kTcRows * 8;
constexpr uint32_t kMOffD = 2 * kMStage;
constexpr uint32_t kMOffK = kMOffD + kMSlots * kMDesc;         /* [ring][side][64] */
constexpr uint32_t kMOffBar = kMOffK + kMRing * 2 * kTcK * 8;
constexpr uint32_t kMSmem = kMOffBar + 208;
constexpr uint32_t kMSmemLaunch = kMSmem + 1024;
static_assert(kMSmemLaunch <= 227 * 1024, "shared memory of the mixed exchange kernel");

/* What the roles need of a tile; behind it [4][128]: addresses of P's rows in
 * their operand (the first row's past the end: what those give is not drained)
 * and offsets in C (-1 past the end), Q's the same. */
struct MTile {
    void *out;
    int K, prows, qrows, c64;
};
static_assert(sizeof(MTile) <= 64, "tile descriptor");

/* A producer warp's part of a step: 8 rows of both sides (byte addresses of the
 * rows at rows[r] and rows[2 * 128 + r]; byte offsets of k at
 * kr[k] and kr[64 + k], negative past the end), RPP rows per pass with 32 / RPP
 * lanes along k, two values per lane: a side's loads, then, when the stage is
 * free, its slices into the 8-row swizzle atom at `atom` of the side's planes. The
 * rows of a pass are 8 / RPP apart, so that their halves or quarters of the 128-
 * byte line meet different banks. */
template <int RPP, typename Free>
__device__ __forceinline__ bool m_step(const unsigned long long *rows, const long long *kr, unsigned char *atom, int lane,
                                       bool pin, bool qin, Free free_slot)
{
    constexpr int GAP = 8 / RPP, LPR = 32 / RPP;
    const int kl = lane & (LPR - 1), sub = lane / LPR;
    const uint32_t in = (uint32_t)(kl >> 2) * 16u + (uint32_t)(kl & 3) * 4u;
    bool waited = false;
#pragma unroll 1
    for (int side = pin ? 0 : 1; side < (qin ? 2 : 1); side++) {
        const long long o0 = kr[side * kTcK + 2 * kl], o1 = kr[side * kTcK + 2 * kl + 1];
        const bool in0 = o0 >= 0, in1 = o1 >= 0;
        float x[GAP][2];
#pragma unroll
        for (int p = 0; p < GAP; p++) {
            const unsigned long long a = rows[side * 2 * kTcRows + p + sub * GAP];
            x[p][0] = in0 ? __ldg(reinterpret_cast<const float *>(a + o0)) : 0.f;
            x[p][1] = in1 ? __ldg(reinterpret_cast<const float *>(a + o1)) : 0.f;
        }
        if (!waited && !free_slot()) return false;
        waited = true;
#pragma unroll
        for (int p = 0; p < GAP; p++) {
            const uint32_t r = p + sub * GAP;
            uint32_t h, m, l;
            tc_split2(x[p][0], x[p][1], h, m, l);
            unsigned char *const dst = atom + side * 3u * kTcSlice + r * 128u + (in ^ (r * 16u));
            *reinterpret_cast<uint32_t *>(dst) = h;
            *reinterpret_cast<uint32_t *>(dst + kTcSlice) = m;
            *reinterpret_cast<uint32_t *>(dst + 2 * kTcSlice) = l;
        }
    }
    if (!waited && !free_slot()) return false;
    return true;
}

__global__ void __launch_bounds__(kMThreads, 1) k_gemm_tcp(const GemmTask *__restrict__ tasks,
                                                           const long long *__restrict__ tile_start, int n_task,
                                                           const int *__restrict__ tile_task, unsigned *err)
{
    extern __shared__ __align__(16) unsigned char m_raw[];
    unsigned char *sm = m_raw + ((1024u - (umma::smem_u32(m_raw) & 1023u)) & 1023u);
    const uint32_t sbase = umma::smem_u32(sm), bar0 = sbase + kMOffBar;
    auto full = [&](uint32_t s) { return bar0 + 8u * (s & 1); };
    auto empty = [&](uint32_t s) { return bar0 + 16u + 8u * (s & 1); };
    auto afull = [&](uint32_t b) { return bar0 + 32u + 8u * (b & 1); };
    auto afree = [&](uint32_t b) { return bar0 + 48u + 8u * (b & 1); };
    auto dfull = [&](uint32_t t) { return bar0 + 64u + 8u * (t & 3); };
    auto dfree = [&](uint32_t t) { return bar0 + 96u + 8u * (t & 3); };
    auto kfull = [&](uint32_t n) { return bar0 + 128u + 8u * (n & 3); };
    auto kfree = [&](uint32_t n) { return bar0 + 160u + 8u * (n & 3); };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + kMOffBar + 192);
    volatile int *dead = reinterpret_cast<volatile int *>(sm + kMOffBar + 196);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long ntiles = tile_start[n_task];

    if (tid == 0) {
        auto init = [](uint32_t b, int n) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(n) : "memory");
        };
        for (uint32_t i = 0; i < 2; i++) {
            init(full(i), kMProd);
            init(empty(i), 1);
            init(afull(i), 1);
            init(afree(i), kMEpi);
        }
        for (uint32_t i = 0; i < 4; i++) {
            init(dfull(i), 1);
            init(dfree(i), kMProd + 1 + kMEpi);
            init(kfull(i), 1);
            init(kfree(i), kMProd);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *dead = 0;
    }
    if (warp == kMProd) umma::tmem_alloc(tmem_slot, 512);
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
    auto desc = [&](uint32_t t) -> unsigned char * { return sm + kMOffD + (t & 3) * kMDesc; };
    auto offs = [&](uint32_t t, int a) { return reinterpret_cast<long long *>(desc(t) + 64) + a * kTcRows; };

    uint32_t nt = 0, ns = 0;   /* tiles, k steps so far */
    bool ok = true;
    if (warp < kMProd) {
        /* ---- producers: 8 rows of each side per warp ---- */
        for (long long tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, nt++) {
            if (!(ok = warp_wait(dfull(nt), (nt >> 2) & 1))) break;
            const MTile &ti = *reinterpret_cast<const MTile *>(desc(nt));
            const int K = ti.K;
            const bool pin = 8 * warp < ti.prows, qin = 8 * warp < ti.qrows;
            const unsigned long long *const rows = reinterpret_cast<const unsigned long long *>(offs(nt, 0)) + 8 * warp;
            for (int k0 = 0; k0 < K; k0 += kTcK, ns++) {
                if (!(ok = warp_wait(kfull(ns), (ns >> 2) & 1))) break;
                const long long *const kr = reinterpret_cast<const long long *>(sm + kMOffK) + (ns & 3) * 2 * kTcK;
                unsigned char *const atom = sm + (ns & 1) * kMStage + (uint32_t)warp * 1024u;
                const int kc = K - k0;
                auto free_slot = [&]() { return warp_wait(empty(ns), ((ns >> 1) & 1) ^ 1); };
                ok = kc > 32 ? m_step<1>(rows, kr, atom, lane, pin, qin, free_slot)
                   : kc > 16 ? m_step<2>(rows, kr, atom, lane, pin, qin, free_slot)
                             : m_step<4>(rows, kr, atom, lane, pin, qin, free_slot);
                if (!ok) break;
                umma::fence_async_smem();
                arrive(full(ns));
                arrive(kfree(ns));
            }
            if (!ok) break;
            arrive(dfree(nt));
        }
    } else if (warp == kMProd + 1) {
        /* ---- descriptors ---- */
        for (long long tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, nt++) {
            const int task = tile_task[tile];
            const GemmTask &T = tasks[task];
            const bool swap = T.swap != 0;
            ZSide P = z_side_a(T), Q = z_side_b(T), Op = z_side_c_rows(T), Oq = z_side_c_cols(T);
            if (swap) {
                const ZSide s = P, o = Op;
                P = Q; Q = s;
                Op = Oq; Oq = o;
            }
            const long long tn = (Q.rows + kTcRows - 1) / kTcRows, loc = tile - tile_start[task];
            const long long p0 = (loc / tn) * kTcRows, q0 = (loc - (loc / tn) * tn) * kTcRows;
            if (!(ok = warp_wait(dfree(nt), ((nt >> 2) & 1) ^ 1))) break;
            for (int r = lane; r < kTcRows; r += 32) {
                const long long p = P.row(p0 + r < P.rows ? p0 + r : p0), q = Q.row(q0 + r < Q.rows ? q0 + r : q0);
                offs(nt, 0)[r] = (long long)(reinterpret_cast<const float *>(P.p) + p);
                offs(nt, 1)[r] = Op.row(p0 + r);
                offs(nt, 2)[r] = (long long)(reinterpret_cast<const float *>(Q.p) + q);
                offs(nt, 3)[r] = Oq.row(q0 + r);
            }
            if (lane == 0) {
                MTile &t = *reinterpret_cast<MTile *>(desc(nt));
                t.out = const_cast<void *>(T.c.p);
                t.K = T.K;
                t.prows = (int)min(P.rows - p0, (long long)kTcRows);
                t.qrows = (int)min(Q.rows - q0, (long long)kTcRows);
                t.c64 = T.c64;
            }
            arrive(dfull(nt));
            for (int k0 = 0; k0 < T.K; k0 += kTcK, ns++) {
                if (!(ok = warp_wait(kfree(ns), ((ns >> 2) & 1) ^ 1))) break;
                long long *const kr = reinterpret_cast<long long *>(sm + kMOffK) + (ns & 3) * 2 * kTcK;
                for (int k = lane; k < kTcK; k += 32) {
                    kr[k] = k0 + k < T.K ? 4 * P.k(k0 + k) : -1;
                    kr[kTcK + k] = k0 + k < T.K ? 4 * Q.k(k0 + k) : -1;
                }
                arrive(kfull(ns));
            }
        }
    } else if (warp == kMProd) {
        /* ---- MMA issue: one thread ---- */
        uint32_t last_bar = 0, last_par = 0;
        bool any = false;
        const int pa[6] = {2, 1, 0, 1, 0, 0}, pb[6] = {0, 1, 2, 0, 1, 0};
        for (long long tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, nt++) {
            if (!(ok = warp_wait(dfull(nt), (nt >> 2) & 1))) break;
            const int K = reinterpret_cast<const MTile *>(desc(nt))->K, nq = reinterpret_cast<const MTile *>(desc(nt))->qrows;
            arrive(dfree(nt));
            const uint32_t acc = tmem + (nt & 1) * 256u, idesc = umma::idesc_bf16(kTcRows, (nq + 15) & ~15, 0, 0);
            ok = warp_wait(afree(nt), ((nt >> 1) & 1) ^ 1);
            for (int k0 = 0; ok && k0 < K; k0 += kTcK, ns++) {
                if (!(ok = warp_wait(full(ns), (ns >> 1) & 1))) break;
                if (lane == 0) {
                    umma::fence_after_sync();
                    const uint32_t a0 = sbase + (ns & 1) * kMStage, b0 = a0 + 3u * kTcSlice;
                    const int nkk = min(kTcK / 16, (K - k0 + 15) / 16);
                    for (int kk = 0; kk < nkk; kk++)
#pragma unroll
                        for (int q = 0; q < 6; q++) {
                            const uint64_t ad = umma::sdesc(a0 + (uint32_t)pa[q] * kTcSlice + (uint32_t)kk * 32u, 16, 1024);
                            const uint64_t bd = umma::sdesc(b0 + (uint32_t)pb[q] * kTcSlice + (uint32_t)kk * 32u, 16, 1024);
                            /* q = 5 (h h) into columns [0, 128), the corrections into [128, 256) */
                            umma::mma_bf16(q == 5 ? acc : acc + kTcRows, ad, bd, idesc, k0 > 0 || kk > 0 || (q > 0 && q < 5));
                        }
                    umma::mma_commit(empty(ns));
                    if (k0 + kTcK >= K) umma::mma_commit(afull(nt));
                    last_bar = empty(ns);
                    last_par = (ns >> 1) & 1;
                    any = true;
                }
                __syncwarp();
            }
        }
        /* after an expiry, MMAs may still be in flight: wait (bounded) for the last commit */
        if (lane == 0 && *dead && any) (void)z_wait(last_bar, last_par);
    } else {
        /* ---- epilogue: lane quarter warp % 4 ---- */
        const int q = warp & 3;
        for (long long tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, nt++) {
            if (!(ok = warp_wait(dfull(nt), (nt >> 2) & 1))) break;
            const MTile ti = *reinterpret_cast<const MTile *>(desc(nt));
            const long long po = offs(nt, 1)[32 * q + lane];
            const long long *const qo = offs(nt, 3);
            const int n = 32 * q < ti.prows ? ti.qrows : 0;   /* columns to drain */
            if (!(ok = warp_wait(afull(nt), (nt >> 1) & 1))) break;
            umma::fence_after_sync();
            const uint32_t taddr = tmem + (nt & 1) * 256u + ((uint32_t)(32 * q) << 16);
            /* the columns past the end have offset -1 in C */
            auto drain = [&](auto *out) {
#pragma unroll 1
                for (int j0 = 0; j0 < n; j0 += 16) {
                    uint32_t rr[16], rc[16];
                    umma::tmem_ld16(taddr + (uint32_t)j0, rr);
                    umma::tmem_ld16(taddr + (uint32_t)(kTcRows + j0), rc);
                    umma::tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; e++) {
                        const long long o = qo[j0 + e];
                        const float v = __uint_as_float(rr[e]) + __uint_as_float(rc[e]);
                        if ((po | o) >= 0) red_global(out + po + o, (std::remove_reference_t<decltype(*out)>)v);
                    }
                    __syncwarp();
                }
            };
            if (ti.c64) drain(reinterpret_cast<double *>(ti.out));
            else drain(reinterpret_cast<float *>(ti.out));
            umma::fence_before_sync();
            arrive(afree(nt));
            arrive(dfree(nt));
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kMProd) umma::tmem_dealloc(tmem, 512);
}

}  // namespace h2g

#endif
