// rad_lw3.cuh -- the LW column solve as kernels over chunks of columns (mixed precision, sm_100a).
//
// The single-kernel LW (rad_lw2.cuh) holds a column's gas optics (taug, fracs: 140 g x 61 layers x 2 floats,
// 68 KB) in shared memory, so two CTAs fit an SM and the latency-bound table gathers and sweep recurrences
// run with ten warps per SM.  Here the gas optics go through HBM instead:
//
//   lw3_optics_kernel  one CTA (256 threads) per column: phases A and B of lw_setup_core (absorber amounts,
//                      cldprop, setcoef, Planck functions, taugb01..16 by pairs of g-points, the max-random overlap
//                      factors of rtrnmr), with taug / fracs and the sweep inputs written straight to the chunk's
//                      scratch.  Shared memory is the set-up data, the species keys of bands 3, 4, 5, 7 and 9 and
//                      the layers' packed words (LwSetupK, ~54 KB).
//   lw3_sweep_kernel   one warp per column, the two sweeps with the g-points in packed pairs (rad_f32x2.cuh), reading
//                      each layer's row of the scratch staged through shared memory by asynchronous copies.  Per
//                      layer each g-point's radiance CHANGE across the layer is formed directly (source minus
//                      radiance x absorptance) and summed over g-points in float64; the heating rates come from
//                      those changes, not from differences of ~300 W/m^2 level fluxes.
//   lw3_fp64_kernel    the plain float64 LW column (lw_column_body<double>) for the columns the optics kernel
//                      flags: a cloudy layer thinner than LW3_THIN hPa.  Such a layer (a cloud in the 0.1 hPa
//                      top layer of the precision-stress request) cools at thousands of K/day, and 1e-5 of
//                      that is already above 0.01 K/day: float optical depths put some g-points on the
//                      neighbouring entry of the 10,001-entry transmittance table, and float radiances
//                      carry ~1e-6 through the column.  Other columns exit at once.
//
// Scratch block of one column (floats, 128-byte aligned): a head record for the surface, then per layer (surface
// first) one row: the 140 optical depths, the 140 Planck fractions and an 80-word record holding everything else the
// sweeps read at that layer, so a layer step reads one contiguous run of 1,440 bytes.  The recurrences are those of
// rad_lw2.cuh (rtrnmr, phys_rrtm_lw_rtrnmr_body.cuh:130-330; rtrnmc, phys_rrtm_lw_rtrnmc.cu:85-310; rtrn,
// phys_rrtm_lw_rtrn.cu:94-330).
#pragma once
#include "rad_f32x2.cuh"
#include "rad_lw2.cuh"

namespace rad {

constexpr int LW3_SWEEP_WARPS = 16;                      // warps of a sweep CTA (one CTA per SM)
constexpr int LW3_REC = 80;                              // words per layer record
constexpr int LW3_ROW = 2 * LW_NGPT + LW3_REC;           // words per layer row: depths, fractions, record
constexpr int LW3_HEAD = 96;                             // words before the first row (the head record)
static_assert(LW3_ROW % 4 == 0 && LW_NGPT % 4 == 0 && LW3_HEAD % 4 == 0, "16-byte pieces");
// layer record k (1..nlay)
constexpr int R_PKLAY = 0;      // [16] pklay[k]
constexpr int R_PKLEVU = 16;    // [16] pklev[k]
constexpr int R_PKLEVD = 32;    // [16] pklev[k - 1]
constexpr int R_TAUCLD = 48;    // [16] cloud optical depth of layer k
constexpr int R_CLDFRC = 64;    // cldfrc[k]
constexpr int R_LSTU = 65;      // int lstu[k]
constexpr int R_LSTD = 66;      // int lstd[k]
constexpr int R_FACD = 67;      // [6] downward factors at k - 1: clr1 cld1 cmb1 cmb2 clr2 cld2
constexpr int R_FACU = 73;      // [6] upward factors at k + 1, same order
// head record
constexpr int H_PKLAY0 = 0;     // [16] pklay[0] (surface)
constexpr int H_SECDIFF = 16;   // [16]
constexpr int H_SEMISS = 32;    // [16]

constexpr float LW3_THIN = LW_THIN;   // hPa: a cloudy layer thinner than this sends the column to float64

__host__ __device__ constexpr int64_t lw3_block_floats(int nlay) { return (LW3_HEAD + (int64_t)nlay * LW3_ROW + 31) / 32 * 32; }

// Optics CTA: 8 warps, 3 CTAs per SM (24 warps, 80 registers a thread, no spills).  The CTAs per SM set how many
// columns share an SM's L1 for the table gathers, and more than 3 cost more than they gain; more warps per CTA share a
// column's tasks and hide the gathers' latency, until the registers run out.  Bound: the L1 data pipe (68 % of its peak
// wavefronts: every task's gathers touch a line per layer of the warp) and phase A's barriers.  Measured per 131,072
// columns of 61 layers: one g-point per task 17.4 ms; pairs 13.2 (288 x 3: 13.3, 224 x 4: 14.9, 320 x 3: 14.4, 384 x 2
// 14.1, 448 x 2: 14.1); phase A and the records spread out 12.6; packed layer words 12.35 (288 x 3: 12.5, 192 x 4: 13.5);
// no load of a species point of weight zero 12.16.  Same bits for every shape.
constexpr int LW3_OPT_THREADS = 256;
constexpr int LW3_OPT_MINB = 3;        // CTAs per SM the optics kernel is compiled for

__global__ void __launch_bounds__(LW3_OPT_THREADS, LW3_OPT_MINB) lw3_optics_kernel(const __grid_constant__ LwBatch bt, int64_t c0,
                                                                   float* __restrict__ scr, int* fp64list, int* err)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LwSetupK<float>& s = *reinterpret_cast<LwSetupK<float>*>(smem_raw);
    const int64_t gc = c0 + blockIdx.x;
    const int rq = bt.find(gc);
    const LwIn& a = bt.req[rq];
    const int nlay = a.nlay;
    const int64_t col = gc - bt.off[rq];
    const int tid = threadIdx.x;
    if (nlay > NLAY_MAX || col >= a.ncol) {
        if (tid == 0 && nlay > NLAY_MAX) atomicExch(err, RAD_DEV_NLAY);
        return;
    }
    float* blk = scr + (int64_t)blockIdx.x * lw3_block_floats(nlay);
    float* row = blk + LW3_HEAD;
    float* aux = row + 2 * LW_NGPT;                // layer k's record at aux + (k - 1) LW3_ROW
    lw_setup_core<float, LW3_OPT_THREADS>(
        s, a, col, tid,
        [&](int g, int k0, P2 tg, P2 fr) {
            *reinterpret_cast<float2*>(row + k0 * LW3_ROW + g) = make_float2(tg.x, tg.y);
            *reinterpret_cast<float2*>(row + k0 * LW3_ROW + LW_NGPT + g) = make_float2(fr.x, fr.y);
        },
        // the records' Planck functions and cloud depths, and the head
        [&]() {
            for (int i = tid; i < nlay * 64; i += LW3_OPT_THREADS) {
                const int k = 1 + (i >> 6), w = i & 63, b = w & 15;
                aux[(k - 1) * LW3_ROW + w] = w < 16 ? s.pklay[k][b] : w < 32 ? s.pklev[k][b] : w < 48 ? s.pklev[k - 1][b] : s.taucld[b][k - 1];
            }
            if (tid < 16) {
                blk[H_PKLAY0 + tid] = s.pklay[0][tid];
                blk[H_SECDIFF + tid] = s.secdiff[tid];
                blk[H_SEMISS + tid] = s.semiss[tid];
            }
        },
        // the records' cloud fractions and overlap factors, and the float64 flag
        [&](int lane) {
            bool thin = false;
            for (int k = 1 + lane; k <= nlay; k += 32) {
                float* r = aux + (k - 1) * LW3_ROW;
                r[R_CLDFRC] = s.cldfrc[k];
                r[R_LSTU] = __int_as_float(s.lstu[k]);
                r[R_LSTD] = __int_as_float(s.lstd[k]);
                const float fd[6] = {s.facclr1d[k - 1], s.faccld1d[k - 1], s.faccmb1d[k - 1], s.faccmb2d[k - 1],
                                     s.facclr2d[k - 1], s.faccld2d[k - 1]};
                const float fu[6] = {s.facclr1u[k + 1], s.faccld1u[k + 1], s.faccmb1u[k + 1], s.faccmb2u[k + 1],
                                     s.facclr2u[k + 1], s.faccld2u[k + 1]};
                for (int f = 0; f < 6; ++f) { r[R_FACD + f] = fd[f]; r[R_FACU + f] = fu[f]; }
                thin = thin || (s.delp[k - 1] < LW3_THIN && s.cldfrc[k] > 1.0e-6f);
            }
            // the chunk's list for lw3_fp64_kernel
            if (__any_sync(0xffffffffu, thin) && lane == 0) fp64list[1 + atomicAdd(fp64list, 1)] = blockIdx.x;
        });
}

// The flagged columns of a chunk in float64: list = [count, chunk-local columns...] appended by the optics
// kernel; a grid of one CTA per SM walks it (the float64 layout's shared memory allows one CTA per SM, so the CTA has
// as many warps as its registers allow: the gas optics' tasks spread over them, the sweeps take the first five).
constexpr int LW3_FP64_THREADS = 512;
__global__ void __launch_bounds__(LW3_FP64_THREADS) lw3_fp64_kernel(const __grid_constant__ LwBatch bt, int64_t c0,
                                                              const int* __restrict__ list, LwLut<double> lutd,
                                                              int* err)
{
    const int n = list[0];
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        lw_column_body<double, LW3_FP64_THREADS>(bt, lutd, err, c0 + list[1 + i]);
        __syncthreads();                          // shared memory is reused by the next column
    }
}

// The entry of rtrnmr's transmittance / Planck-fraction tables for optical depth od: position 10^4 od / (bpade + od) +
// 1/2, its integer part taken by adding 2^23 rounded down (entry number in the sum's low bits; clamped, so a NaN depth
// reads the last entry).  lut[i] = {exp, tfn}, one 8-byte load.  The quotient takes a Newton step: a depth's rounding
// decides which of two entries, 3e-4 apart, it gets.  The divisor is scaled (F2_DOWN), so that every finite depth has its
// entry; an infinite one (cloud times diffusivity past the largest float) has a NaN position, the last entry.
constexpr float LW3_TWO23 = 8388608.0f;
template <class V>
__device__ __forceinline__ V lw3_pos(V od)
{
    const V d = fma2(od, vset<V>(F2_DOWN), vset<V>(F2_DOWN * (1.0f / 0.278f)));
    return f2_add_rm(fma2(quot2(od, d, rcp2(d)), vset<V>(10000.0f * F2_DOWN), vset<V>(0.5f)), vset<V>(LW3_TWO23));
}
__device__ __forceinline__ float2 lw3_entry(const float2* lut, float pr)
{
    return lut[min(__float_as_uint(pr) - 0x4b000000u, 10000u)];
}
__device__ __forceinline__ void lw3_lookup(const float2* lut, F2 pr, F2& ex, F2& tfn)
{
    const float2 a = lw3_entry(lut, pr.x), b = lw3_entry(lut, pr.y);
    ex = F2{a.x, b.x};
    tfn = F2{a.y, b.y};
}
__device__ __forceinline__ void lw3_lookup(const float2* lut, float pr, float& ex, float& tfn)
{
    const float2 a = lw3_entry(lut, pr);
    ex = a.x;
    tfn = a.y;
}
// The optical depth of table entry it (lw_lut's tau: bpade it / (10^4 - it), 1e10 for the last).
template <class V>
__device__ __forceinline__ V lw3_entry_tau(V it)
{
    const V d = vset<V>(10000.0f) - it, t = quot2(it, d, rcp2(d)) * vset<V>(1.0f / 0.278f);
    return sel2(le2(d, 0.0f), vset<V>(1.0e10f), t);
}

// One layer of one g-point, or of a pair of neighbouring ones (V = float, F2; a pair shares its band), in one direction:
// the terms (phys_rrtm_lw_rtrnmr_body.cuh:130-190; branch-free, so that the g-points' table loads are all in flight
// together) and the recurrences of rtrnmr, rtrnmc and rtrn (OVR, the LW_OVR_* transfer) on the state.
// Returns the total-sky radiance change across the layer formed directly -- source - radiance x absorptance, per
// overlap part -- so it keeps its relative precision however small it is beside the radiance; incc = the clear-sky one.
template <class V>
struct Lw3State {
    V tot, clr, trad, crad, rad;   // radtot, radclr and, with the max-random overlap, totrad, clrrad, rad
};
struct Lw3Layer {                  // what a layer's g-points share (uniform over the warp)
    float clfr;
    bool lst;
    float f[6];                    // the six max-random overlap factors clr1 cld1 cmb1 cmb2 clr2 cld2
};
template <int OVR, class V, class M>
__device__ __forceinline__ V lw3_step(Lw3State<V>& s, const float2* lut, V taug, V plfrac, float blay, float plev, float tcb,
                                      float sdif, bool cl, M bit, const Lw3Layer& L, V& incc)
{
    const float rec_6 = 0.166667f, c06 = 0.06f;
    const float dpl = plev - blay;
    const V od0 = max2(taug * vset<V>(sdif), 0.0f);
    const V pr = lw3_pos(od0);
    V ex, tfn;
    lw3_lookup(lut, pr, ex, tfn);
    const auto thin = le2(od0, c06);
    const V one = vset<V>(1.0f);
    const V a1 = nma2(od0 * vset<V>(0.5f), od0, od0);
    const V atr = sel2(thin, a1, one - ex), trn = sel2(thin, one - a1, ex);
    const V gf = sel2(thin, od0 * vset<V>(rec_6), tfn);
    const V src = (plfrac * fma2(vset<V>(dpl), gf, vset<V>(blay))) * atr;
    const V prev = s.tot, pclr = s.clr;
    V inc = nma2(prev, atr, src);
    incc = nma2(pclr, atr, src);
    s.clr = fma2(pclr, trn, src);
    if (OVR == LW_OVR_MAXRAN && L.lst) {
        s.trad = prev * vset<V>(L.clfr);
        s.crad = prev - s.trad;
        s.rad = vset<V>(0.0f);
    }
    if (!cl) {                     // no cloud in the layer (McICA: in none of the warp's sub-columns)
        s.tot = fma2(prev, trn, src);
        return inc;
    }
    // the cloudy part: gas (its table entry's depth) plus cloud
    const float x = sdif * tcb;
    const V ot = fma2(vset<V>(sdif), vset<V>(tcb), sel2(thin, od0, lw3_entry_tau(pr - vset<V>(LW3_TWO23))));
    const V pc = lw3_pos(ot);
    V exc, tfc;
    lw3_lookup(lut, pc, exc, tfc);
    const auto thinc = lt2(ot, c06);
    const V a2 = nma2(ot * vset<V>(0.5f), ot, ot);
    const V att = sel2(thinc, a2, one - exc), tft = sel2(thinc, ot * vset<V>(rec_6), tfc);
    const V tsrc = (plfrac * fma2(vset<V>(dpl), tft, vset<V>(blay))) * att;
    if (OVR == LW_OVR_MAXRAN) {
        const V trt = sel2(thinc, one - a2, exc);
        const V cs = tsrc * vset<V>(L.clfr), gs = src * vset<V>(1.0f - L.clfr);
        inc = (cs + gs) - fma2(s.trad, att, s.crad * atr);
        const V tt = fma2(s.trad, trt, cs), cc = fma2(s.crad, trn, gs);
        s.tot = tt + cc;
        const V rm = fma2(s.rad, fma2(vset<V>(L.f[0]), trn, trt * vset<V>(L.f[1])),
                          nma2(vset<V>(L.f[2]), src, tsrc * vset<V>(L.f[3])));
        const V r = fma2(vset<V>(L.f[4]), cc + rm, nma2(vset<V>(L.f[5]), tt - rm, vset<V>(0.0f) - rm));
        s.rad = r;
        s.trad = tt + r;
        s.crad = cc - r;
    } else {
        // rtrnmc is rtrn with a cloud fraction of 1 in its cloudy sub-columns
        const float cf = OVR == LW_OVR_MCICA ? 1.0f : L.clfr;
        const V S = fma2(vset<V>(cf), tsrc - src, src);
        const float ef = 1.0f - (1.0f - rexp(-x)) * cf;
        const float ca = -expm1(-x) * cf;                     // 1 - ef without the cancellation
        const V ctot = fma2(prev * trn, vset<V>(ef), S);
        const V cinc = nma2(prev, nma2(atr, vset<V>(ca), atr + vset<V>(ca)), S);
        if (OVR == LW_OVR_MCICA) {
            s.tot = sel2(bit, ctot, fma2(prev, trn, src));
            inc = sel2(bit, cinc, inc);
        } else {
            s.tot = ctot;
            inc = cinc;
        }
    }
    return inc;
}

// The sweeps stream each layer's row (1,440 bytes) through a LW3_NSTAGE-stage ring in shared memory with asynchronous
// 16-byte copies (cp.async.cg: L2 to shared, no L1 allocation), LW3_NSTAGE - 1 layers ahead of the one being computed,
// so the scratch's DRAM latency overlaps the arithmetic.  (Bulk copies completed on an mbarrier per slot were 2.5 %
// slower: lane 0 alone issues and waits, where the 16-byte copies spread over the warp.)
constexpr int LW3_NSTAGE = 3;

__device__ __forceinline__ void lw3_stage_row(float* st, const float* row, int lane)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(st) + 16u * (unsigned)lane;
    const float* src = row + 4 * lane;
#pragma unroll
    for (int c = 0; c < LW3_ROW / 4; c += 32)
        if (c + 32 <= LW3_ROW / 4 || c + lane < LW3_ROW / 4)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16u * c), "l"(src + 4 * c) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// Per-g-point profiles of one column for lwrad's optional outputs (DIAG sweeps): [nlay + 1][LW3_PGQ][LW_NGPT]
// floats: at level L (surface first) the upward and downward radiance, total sky then clear sky (q 0..3); at
// layer L (1..nlay) the radiance changes across it formed directly, upward pass U(L) - U(L-1) and downward
// pass D(L-1) - D(L), total sky then clear sky (q 4..7).
constexpr int LW3_PGQ = 8;
__host__ __device__ constexpr int64_t lw3_pg_floats(int nlay) { return (int64_t)(nlay + 1) * LW3_PGQ * LW_NGPT; }

// Shared memory of a sweep CTA: the {exp, tfn} table, then per warp its ring and its level sums.
struct Lw3Warp {
    float ring[LW3_NSTAGE][LW3_ROW];
    double fup[NLAY_MAX + 1], fdn[NLAY_MAX + 1];
};
constexpr int LW3_LUT_N = 10001;
constexpr size_t LW3_LUT_BYTES = (LW3_LUT_N * sizeof(float2) + 15) / 16 * 16;
constexpr size_t lw3_sweep_smem() { return LW3_LUT_BYTES + LW3_SWEEP_WARPS * sizeof(Lw3Warp); }

// The two sweeps of the chunk's column lc by one warp.
template <int OVR, bool DIAG>
__device__ __forceinline__ void lw3_sweep_column(Lw3Warp& W, const float2* lut, const LwBatch& bt, int64_t c0, int64_t lc,
                                                 const float* __restrict__ scr, float* __restrict__ pg, int lane)
{
    const int64_t gc = c0 + lc;
    const int rq = bt.find(gc);
    const LwIn& a = bt.req[rq];
    const int nlay = a.nlay;
    const int64_t col = gc - bt.off[rq];
    const int64_t N = a.ncol;
    if (nlay > NLAY_MAX || col >= N) return;    // the optics kernel has flagged a bad nlay
    const float* head = scr + lc * lw3_block_floats(nlay);
    const float* rows = head + LW3_HEAD;
    if (DIAG) pg += lc * lw3_pg_floats(nlay);
    // sweep steps: s = 0 .. nlay-1 downward (layer nlay - s), s = nlay .. 2 nlay - 1 upward (layer s - nlay + 1)
    const int nstep = 2 * nlay;
    auto layer_of = [&](int st) { return st < nlay ? nlay - st : st - nlay + 1; };
#pragma unroll
    for (int q = 0; q < LW3_NSTAGE - 1; ++q) lw3_stage_row(W.ring[q], rows + (size_t)(layer_of(q) - 1) * LW3_ROW, lane);
    const float eps = 1.0e-6f;
    const bool val = lane < LW_NGPT - 128;                          // the single g-point is real
    const int g0 = 2 * lane, g1 = 64 + 2 * lane, g2 = val ? 128 + lane : LW_NGPT - 1;
    const int b0 = c_lw_band[g0], b1 = c_lw_band[g1], b2 = c_lw_band[g2];
    const float sd0 = __ldg(head + H_SECDIFF + b0), sd1 = __ldg(head + H_SECDIFF + b1), sd2 = __ldg(head + H_SECDIFF + b2);
    Lw3State<F2> s0, s1;
    Lw3State<float> s2;
    s0.tot = s0.clr = s0.trad = s0.crad = s0.rad = f2(0.0f);
    s1 = s0;
    s2.tot = s2.clr = s2.trad = s2.crad = s2.rad = 0.0f;
    auto ld2 = [](const float* p) { const float2 v = *reinterpret_cast<const float2*>(p); return F2{v.x, v.y}; };
    auto st2 = [](float* p, F2 v) { *reinterpret_cast<float2*>(p) = make_float2(v.x, v.y); };
    // One layer of the sweep for the lane's g-points; returns the warp's float64 sum of the radiance changes.
    auto layer = [&](const float* st, int k, bool down) -> double {
        const float* r = st + 2 * LW_NGPT;
        const float* pl = r + (down ? R_PKLEVD : R_PKLEVU);
        Lw3Layer L;
        L.clfr = r[R_CLDFRC];
        L.lst = __float_as_int(r[down ? R_LSTD : R_LSTU]) != 0;
        bool cl = L.clfr >= eps;
        B2 m0{false, false}, m1{false, false};
        bool m2 = false;
        if (OVR == LW_OVR_MCICA) {   // word j of a layer holds g-points 32 j .. 32 j + 31
            auto word = [&](int j) { return __ldg(a.mask + ((size_t)j * nlay + (k - 1)) * N + col); };
            const unsigned w0 = word(g0 >> 5) >> (g0 & 31), w1 = word(g1 >> 5) >> (g1 & 31), w2 = word(g2 >> 5) >> (g2 & 31);
            m0 = B2{(w0 & 1u) != 0, (w0 & 2u) != 0};
            m1 = B2{(w1 & 1u) != 0, (w1 & 2u) != 0};
            m2 = (w2 & 1u) != 0;
            cl = __any_sync(0xffffffffu, m0.x || m0.y || m1.x || m1.y || m2);
        }
        if (OVR == LW_OVR_MAXRAN && cl) {
#pragma unroll
            for (int i = 0; i < 6; ++i) L.f[i] = r[(down ? R_FACD : R_FACU) + i];
        }
        F2 c0_, c1_;
        float c2_;
        const F2 i0 = lw3_step<OVR>(s0, lut, ld2(st + g0), ld2(st + LW_NGPT + g0), r[R_PKLAY + b0], pl[b0], r[R_TAUCLD + b0],
                                    sd0, cl, m0, L, c0_);
        const F2 i1 = lw3_step<OVR>(s1, lut, ld2(st + g1), ld2(st + LW_NGPT + g1), r[R_PKLAY + b1], pl[b1], r[R_TAUCLD + b1],
                                    sd1, cl, m1, L, c1_);
        const float i2 = lw3_step<OVR>(s2, lut, st[g2], st[LW_NGPT + g2], r[R_PKLAY + b2], pl[b2], r[R_TAUCLD + b2], sd2, cl,
                                       m2, L, c2_);
        if (DIAG) {
            // the radiance changes across the layer; the radiances at the level the step ends on (k - 1 going down, k
            // going up)
            float* p = pg + ((size_t)k * LW3_PGQ + (down ? 5 : 4)) * LW_NGPT;
            float* q = pg + ((size_t)(down ? k - 1 : k) * LW3_PGQ + (down ? 1 : 0)) * LW_NGPT;
            st2(p + g0, i0); st2(p + 2 * LW_NGPT + g0, c0_); st2(q + g0, s0.tot); st2(q + 2 * LW_NGPT + g0, s0.clr);
            st2(p + g1, i1); st2(p + 2 * LW_NGPT + g1, c1_); st2(q + g1, s1.tot); st2(q + 2 * LW_NGPT + g1, s1.clr);
            if (val) { p[g2] = i2; p[2 * LW_NGPT + g2] = c2_; q[g2] = s2.tot; q[2 * LW_NGPT + g2] = s2.clr; }
        }
        const double sum = ((double)i0.x + (double)i0.y) + ((double)i1.x + (double)i1.y) + (val ? (double)i2 : 0.0);
        return warp_sum(sum);
    };
    // float64 sum over the column's g-points of one field of the states
    auto total = [&](F2 x, F2 y, float z) {
        return warp_sum(((double)x.x + (double)x.y) + ((double)y.x + (double)y.y) + (val ? (double)z : 0.0));
    };
    // ---- the sweeps: downward, the surface, upward; layer s + LW3_NSTAGE - 1 is copied in while layer s computes
    double s_tu = 0, s_cu = 0, s_td = 0, s_cd = 0;
    int slot = 0;                                                    // st % LW3_NSTAGE
    for (int st = 0; st < nstep; ++st) {
        const int nx = st + LW3_NSTAGE - 1, nslot = slot == 0 ? LW3_NSTAGE - 1 : slot - 1;
        if (nx < nstep) lw3_stage_row(W.ring[nslot], rows + (size_t)(layer_of(nx) - 1) * LW3_ROW, lane);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        // this lane's copies of step st have landed (the LW3_NSTAGE - 1 later groups may still be in flight)
        asm volatile("cp.async.wait_group %0;" ::"n"(LW3_NSTAGE - 1) : "memory");
        __syncwarp();                                            // ... and every lane's
        if (st == nlay) {
            // surface: emission and reflection
            s_td = total(s0.tot, s1.tot, s2.tot);
            s_cd = total(s0.clr, s1.clr, s2.clr);
            auto surface = [&](auto& s, auto fr, int b) {
                using V = decltype(s.tot);
                const float semi = __ldg(head + H_SEMISS + b);
                const V rad0 = fr * vset<V>(semi) * vset<V>(__ldg(head + H_PKLAY0 + b));
                s.tot = fma2(vset<V>(1.0f - semi), s.tot, rad0);
                s.clr = fma2(vset<V>(1.0f - semi), s.clr, rad0);
                s.trad = s.crad = s.rad = vset<V>(0.0f);
            };
            const float* fr = rows + LW_NGPT;
            surface(s0, F2{__ldg(fr + g0), __ldg(fr + g0 + 1)}, b0);
            surface(s1, F2{__ldg(fr + g1), __ldg(fr + g1 + 1)}, b1);
            surface(s2, __ldg(fr + g2), b2);
            s_tu = total(s0.tot, s1.tot, s2.tot);
            s_cu = total(s0.clr, s1.clr, s2.clr);
            if (DIAG) {   // the upward radiances leaving the surface; nothing comes down at the top
                float* top = pg + ((size_t)nlay * LW3_PGQ + 1) * LW_NGPT;
                st2(pg + g0, s0.tot); st2(pg + 2 * LW_NGPT + g0, s0.clr); st2(top + g0, f2(0.0f)); st2(top + 2 * LW_NGPT + g0, f2(0.0f));
                st2(pg + g1, s1.tot); st2(pg + 2 * LW_NGPT + g1, s1.clr); st2(top + g1, f2(0.0f)); st2(top + 2 * LW_NGPT + g1, f2(0.0f));
                if (val) { pg[g2] = s2.tot; pg[2 * LW_NGPT + g2] = s2.clr; top[g2] = 0.0f; top[2 * LW_NGPT + g2] = 0.0f; }
            }
        }
        const bool down = st < nlay;
        const int k = layer_of(st);
        const double v = layer(W.ring[slot], k, down);
        if (lane == 0) {
            if (down) W.fdn[k - 1] = v;           // D(k-1) - D(k), summed over g
            else W.fup[k] = v;                    // U(k) - U(k-1), summed over g
        }
        slot = slot == LW3_NSTAGE - 1 ? 0 : slot + 1;
        __syncwarp();                                 // the stage is free for the copy two steps on
    }
    const double t_tu = total(s0.tot, s1.tot, s2.tot), t_cu = total(s0.clr, s1.clr, s2.clr);
    __syncwarp();
    // ---- outputs: fluxes x flxfac; heating rates from the per-layer net-flux changes (rtrnmr post)
    const double pi = 3.14159265358979323846;
    const double flxfac = 0.5 * pi * 2.0e4;
    const double heatfac = 9.80665 * 1.0e-2 / 1.0046e3;
    for (int k = lane; k < nlay; k += 32) {
        // layer k + 1 (surface first): (U(k) - D(k)) - (U(k+1) - D(k+1)) = -(dU + dD)
        const double du = W.fup[k + 1], dd = W.fdn[k];
        const int kin = nlay - 1 - k;
        const double dl = (double)__ldg(a.plvl + (size_t)(kin + 1) * N + col) - (double)__ldg(a.plvl + (size_t)kin * N + col);
        a.htlw[(size_t)kin * N + col] = (float)(-(du + dd) * flxfac * (heatfac / dl));
    }
    if (lane == 0) {
        a.topflw[col] = (float)(t_tu * flxfac);
        a.topflw[N + col] = (float)(t_cu * flxfac);
        a.sfcflw[col] = (float)(s_tu * flxfac);
        a.sfcflw[N + col] = (float)(s_cu * flxfac);
        a.sfcflw[2 * N + col] = (float)(s_td * flxfac);
        a.sfcflw[3 * N + col] = (float)(s_cd * flxfac);
    }
}

// One warp per column, warps striding over the chunk's columns (grid: at most one CTA per SM).  Lane l carries the
// pairs of g-points 2 l, 2 l + 1 and 64 + 2 l, 65 + 2 l, in packed arithmetic, and lanes 0..11 the single g-points
// 128..139.  Bound: the random 8-byte table gathers and issue slots.  Measured per 131,072 columns of 61 layers: 12.4 ms
// with one g-point per slot, branches and three 4-byte gathers per entry; branch-free pairs with the table through L1
// 9.4 ms at 5 CTAs of 4 warps per SM (10.0 at 6, 7.05 at 4: the more warps, the less L1 is left for the 80 KB table);
// with the table in shared memory 6.2 ms at 16 warps per SM (12: 6.7, 14: 7.1, 20: 9.4, 24: 9.6 -- from 20 on the
// registers no longer hold two pairs' chains side by side), 6.5 ms with the Newton step on the entry positions.
template <int OVR, bool DIAG = false>
__global__ void __launch_bounds__(LW3_SWEEP_WARPS * 32, 1)
lw3_sweep_kernel(const __grid_constant__ LwBatch bt, int64_t c0, int64_t nc, const float* __restrict__ scr,
                 const float2* __restrict__ lutg, float* __restrict__ pg0 = nullptr)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* lut = reinterpret_cast<float2*>(smem_raw);
    for (int i = threadIdx.x; i < LW3_LUT_N; i += LW3_SWEEP_WARPS * 32) lut[i] = __ldg(lutg + i);
    __syncthreads();                                // the only barrier: the warps go their own ways from here
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Lw3Warp& W = reinterpret_cast<Lw3Warp*>(smem_raw + LW3_LUT_BYTES)[warp];
    for (int64_t lc = blockIdx.x + (int64_t)gridDim.x * warp; lc < nc; lc += (int64_t)gridDim.x * LW3_SWEEP_WARPS)
        lw3_sweep_column<OVR, DIAG>(W, lut, bt, c0, lc, scr, pg0, lane);
}

// Optional-output pointers of a launch's requests: hlw0, hlwb, lwflxprf, hsw0, htswb, swflxprf (null = not wanted).
struct DiagOuts {
    float* p[RAD_MAXREQ][6];
};
// lwrad's optional outputs of a chunk from the DIAG sweeps' profiles: one CTA per column, a warp per level.  The level's
// eight fields (4,480 contiguous bytes) go to shared memory, lane q of each half warp sums band q of one field at a time
// over its g-points in float64, and the totals are summed over the bands' lanes: hlwb (htrb of rtrnmr's lhlwb block)
// from a band's per-layer changes, hlw0 from the total clear-sky changes, lwflxprf the level fluxes x flxfac; heating as
// the sweeps form htlw: -(dU + dD) flxfac heatfac / delp.  Bound: the profile's bytes (278 KB per column); 5.0 -> 0.57 ms
// per 7,632 columns against one lane per band over strided words.
constexpr int LW3_DIAG_WARPS = 4;
__global__ void __launch_bounds__(LW3_DIAG_WARPS * 32) k_lw_diag(const __grid_constant__ LwBatch bt, int64_t c0,
                                                                 const float* __restrict__ pg, const __grid_constant__ DiagOuts outs)
{
    constexpr int ROW = LW3_PGQ * LW_NGPT;
    __shared__ __align__(16) float sm[LW3_DIAG_WARPS][ROW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 15, half = lane >> 4;
    const int64_t gc = c0 + blockIdx.x;
    const int rq = bt.find(gc);
    const LwIn& a = bt.req[rq];
    const int nlay = a.nlay;
    const int64_t col = gc - bt.off[rq], N = a.ncol;
    if (nlay > NLAY_MAX || col >= N) return;
    float* hlw0 = outs.p[rq][0];
    float* hlwb = outs.p[rq][1];
    float* flx = outs.p[rq][2];
    const float4* p = reinterpret_cast<const float4*>(pg + blockIdx.x * lw3_pg_floats(nlay));
    const double flxfac = 0.5 * 3.14159265358979323846 * 2.0e4;
    const double heatfac = 9.80665 * 1.0e-2 / 1.0046e3;
    const int g0 = c_lw_ns[q], g1 = c_lw_ns[q + 1];
    float* w = sm[warp];
    for (int L = warp; L <= nlay; L += LW3_DIAG_WARPS) {
        __syncwarp();                              // the previous level's sums have been read
        for (int i = lane; i < ROW / 4; i += 32) reinterpret_cast<float4*>(w)[i] = __ldg(p + (size_t)L * (ROW / 4) + i);
        __syncwarp();
        double v[4], t[4];                         // band q of field 2 i + half, and the field's total
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* f = w + (2 * i + half) * LW_NGPT;
            double x = 0.0;
            for (int g = g0; g < g1; ++g) x += (double)f[g];
            v[i] = x;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            t[i] = x;
        }
        const int kin = nlay - L;                  // top-first index of layer L and of level L
        if (flx && q == 0) {
            flx[((size_t)half * (nlay + 1) + kin) * N + col] = (float)(t[0] * flxfac);
            flx[((size_t)(2 + half) * (nlay + 1) + kin) * N + col] = (float)(t[1] * flxfac);
        }
        const double db = v[2] + __shfl_xor_sync(0xffffffffu, v[2], 16);      // fields 4 + 5 of the band
        const double dc = t[3] + __shfl_xor_sync(0xffffffffu, t[3], 16);      // fields 6 + 7 in total
        if (L > 0 && half == 0) {
            const double dl = (double)__ldg(a.plvl + (size_t)(kin + 1) * N + col) - (double)__ldg(a.plvl + (size_t)kin * N + col);
            const double rf = flxfac * (heatfac / dl);
            if (hlwb) hlwb[((size_t)q * nlay + kin) * N + col] = (float)(-db * rf);
            if (hlw0 && q == 0) hlw0[(size_t)kin * N + col] = (float)(-dc * rf);
        }
    }
}

}  // namespace rad
