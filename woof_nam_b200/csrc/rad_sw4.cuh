// rad_sw4.cuh -- the chunked SW of rad_solve (mixed precision): set-up and gas optics, the layer reflectances
// and transmittances, their float64 fix-ups and recomputes, and the adding sweeps in five kernels per chunk of sunlit
// columns.
//
// Same statements as sw2_column (rad_sw2.cuh), split where the work changes shape, and each kernel small enough
// that the CTAs resident on an SM run out of the instruction cache (one kernel with all three phases spent most
// of its stalls waiting for instructions):
//  * sw4_gas_kernel, one CTA (128 threads) per sunlit column, six per SM: set-up and cloud optics
//    (sw2_setup), gas and Rayleigh optical depths per (g-point pair, layer); writes the column image (the part of the
//    shared-memory layout the later phases read, taug included).
//  * sw4_rt_kernel, one CTA per column: loads the image, then the layer R/T of the clear pass and, in the
//    layers with cloud, of the cloudy pass (spcvrtc.cu:112-173, 330-460) in float without branches, a task a pair
//    of neighbouring g-points in packed float2 arithmetic (rad_f32x2.cuh), lanes on 32 consecutive (layer, pair)
//    tasks so that a warp shares the cloudy branch.  A g-point whose R/T needs a float64 step (the resonance, or an
//    exp-table argument near an entry bound whose neighbouring entry matters) is queued.  Output per column: a
//    header (solar source per g-point, albedos, overlap fractions, heating factors, the cloudy-pass slot of each
//    layer), the R/T as [layer][field][g-point] (a warp of the sweep kernel reads 28 consecutive pairs of g-points of
//    one field and layer, 224 contiguous bytes: half a row) and the queue.
//  * sw4_fix_kernel, over the tile's queues: sw2_layer (the single-kernel SW's own function) for the queued g-points,
//    cut into items.  Taking the queue out of the R/T kernel left that 80 registers and 6 CTAs per SM instead of 128 and
//    4, no CTA waits for its slowest float64 lane any more, and the columns at a resonance (thousands of entries; up to
//    2,000,000 cycles in one CTA when a fixed queue of 527 overflowed) spread over the grid.
//  * sw4_exact_kernel (tiles of SW4_EXACT_MIN columns or more), over per-band lists: the g-points whose R/T are
//    recomputed in float64 from the column's inputs.
//    Measured per 131,072 columns (65,536 sunlit, 61 layers): 12.76 ms for the R/T as one kernel with one g-point per
//    thread and the queue formed by the same CTA; 9.48 with pairs; 4.30 + 3.35 as R/T and fix-up; 4.30 + 1.70 + 0.23 with
//    the recomputes apart.
//  * sw4_sweep_kernel, one CTA per column: the adding method alone (swflux, spcvrtc.cu:178-215) -- the upward
//    sweep with segment checkpoints, the downward sweep re-reading each segment's R/T, float64 level sums and
//    the swrad epilogue.
// The outputs agree with sw2_column's to float rounding (tests/test_gpu_sw_split.py).
#pragma once
#include <type_traits>
#include "rad_f32x2.cuh"
#include "rad_sw2.cuh"

namespace rad {

constexpr int SW4_FIELDS = 6;                       // rb, rd, tb, td, e3 (delta-scaled beam), e4 (unscaled beam)
constexpr int SW4_LAYER = SW4_FIELDS * SW_NGPT;     // floats per layer and pass, [field][g]
// CTA shapes of the kernels, swept on the B200 (same bits): the gas-optics kernel at 128 threads x 6 CTAs
// per SM against 160 x 5, 192 x 4, 256 x 3, 320 x 2, 384 x 2 (SW +0.2 to +9.8 %).
constexpr int SW4_RT_THREADS = 128;                 // threads of an R/T CTA
constexpr int SW4_OPT_MINB = 6;                     // CTAs per SM the R/T kernel is compiled for (4: 4.62, 5: 4.41, 6: 4.30 ms)
constexpr int SW4_SWEEP_WARPS = 4;                   // warps of a sweep CTA (one column)
constexpr int SW4_SWEEP_THREADS = 32 * SW4_SWEEP_WARPS;
constexpr int SW4_SWEEP_MINB = 5;                    // CTAs per SM it is compiled for (4: 5.64, 5: 5.06, 6: 5.89, 7: 6.78 ms)
constexpr int SW4_GAS_THREADS = 128;               // threads of a gas-optics CTA
constexpr int SW4_GAS_MINB = 6;                     // ... and the gas-optics kernel
constexpr bool SW4_L2PF = true;                     // the sweeps prefetch the R/T rows two segments ahead into L2

struct Sw4Hdr {
    double rdelp[NLAY_MAX];          // heatfac / delp, float64
    float zsolar[SW_NGPT];           // ssolar * sfluxzen of each g-point
    float albbm[2], albdf[2], zcf0, zcf1, pad0[2];
    int cloudy;                      // the cloudy pass runs
    int ncl;                         // layers with a cloudy-pass R/T
    int clr5;                        // the clear rows hold no e4 (it is e3: no delta scaling in the clear pass)
    int pad1;
    signed char slot[NLAY_MAX];      // cloudy-pass slot of each layer; -1: the clear R/T serve both passes
};
static_assert(sizeof(Sw4Hdr) % 16 == 0, "the header is copied in 16-byte pieces");
__host__ __device__ constexpr size_t sw4_hdr_bytes() { return (sizeof(Sw4Hdr) + 15) / 16 * 16; }
// One column's block of the chunk scratch: header, clear R/T [nlay][SW4_LAYER], cloudy R/T [nlay][SW4_LAYER]
// (the first ncl slots used), and the float64 queue of sw4_rt_kernel (16-bit entries k0 * SW_NGPT + g, the
// table-entry tests from the front, the resonance from the back).
__host__ __device__ constexpr size_t sw4_queue_offset(int nlay)
{
    return sw4_hdr_bytes() + (size_t)2 * nlay * SW4_LAYER * sizeof(float);
}
__host__ __device__ constexpr size_t sw4_block_bytes(int nlay)
{
    return sw4_queue_offset(nlay) + (size_t)nlay * SW_NGPT * sizeof(uint16_t);
}
// The tile's work lists: a head of counters, the items of sw4_fix_kernel (at most SW4_FIX_THREADS queue entries of one
// column, {column of the tile, first entry | entries << 16}), then per band the g-points left to sw4_exact_kernel
// ({column of the tile, k0 * SW_NGPT + g}; a full list's g-points are formed by sw4_fix_kernel itself).
constexpr int SW4_FIX_THREADS = 64;
constexpr int SW4_FIX_MINB = 8;                     // CTAs per SM the fix kernel is compiled for
constexpr int SW4_LIST_HEAD = 32;                   // words: [0] items, [1 + b] exact g-points of band b
__host__ __device__ constexpr int64_t sw4_max_items(int nlay) { return nlay * SW_NGPT / SW4_FIX_THREADS + 2; }
__host__ __device__ constexpr int64_t sw4_exact_cap(int64_t cols) { return cols > 256 ? cols : 256; }   // per band
struct Sw4Lists {
    int* head;                                      // [SW4_LIST_HEAD]
    int2* items;                                    // [cols * sw4_max_items]
    int2* exact;                                    // [14][cap]
    int cap;
};
__host__ __device__ constexpr int64_t sw4_list_bytes(int nlay, int64_t cols)
{
    return SW4_LIST_HEAD * (int64_t)sizeof(int) + (cols * sw4_max_items(nlay) + 14 * sw4_exact_cap(cols)) * (int64_t)sizeof(int2);
}
inline Sw4Lists sw4_lists(void* base, int nlay, int64_t cols)
{
    Sw4Lists l;
    l.head = static_cast<int*>(base);
    l.items = reinterpret_cast<int2*>(l.head + SW4_LIST_HEAD);
    l.exact = l.items + cols * sw4_max_items(nlay);
    l.cap = (int)sw4_exact_cap(cols);
    return l;
}
static_assert(sw4_hdr_bytes() % 16 == 0 && (SW4_LAYER * sizeof(float)) % 16 == 0 && SW_NGPT * sizeof(uint16_t) % 16 == 0,
              "16-byte aligned parts");

// ---- branch-free float R/T of two g-points side by side (the phase-R fast path); the float64 decisions become flags.
struct SwRT2 {
    F2 rb, rd, tb, td, e3, e4;
};
// Position of zb in the reference's exp table: ft = zb / (bpade + zb), pos = 10^4 ft + 1/2, it = floor(pos) as a float
// (adding 2^23 rounded down leaves the integer part, so no float <-> integer conversion is needed).  q = ft / F2_DOWN:
// the divisor is scaled, so that every finite zb has its entry.
struct SwPos2 {
    F2 q, pos, it;
};
__device__ __forceinline__ SwPos2 sw4_pos(F2 zb)
{
    SwPos2 p;
    p.q = div2(zb, fma2(zb, f2(F2_DOWN), f2(F2_DOWN * ((float)1.0f / (float)0.278f))));
    p.pos = fma2(p.q, f2(10000.0f * F2_DOWN), f2(0.5f));
    p.it = f2_add_rm(p.pos, f2(8388608.0f)) - 8388608.0f;
    return p;
}
__device__ __forceinline__ bool sw4_near1(float zb, float pos, float it, float m)   // sw2_near without branches
{
    const bool tbl = fabsf((pos - it) - 0.5f) > 0.5f - m;
    const bool ser = zb > 0.06f * (1.0f - SW2_ZB_EPS);
    return zb <= 0.06f * (1.0f + SW2_ZB_EPS) ? ser : tbl;
}
__device__ __forceinline__ void sw4_near(F2 zb, const SwPos2& p, bool& n0, bool& n1)
{
    const F2 m = (p.q * (10000.0f * F2_DOWN)) * fma2(nma2(p.q, f2(F2_DOWN), f2(1.0f)), f2(SW2_ZB_EPS), f2(3.0e-7f));
    n0 = sw4_near1(zb.x, p.pos.x, p.it.x, m.x);
    n1 = sw4_near1(zb.y, p.pos.y, p.it.y, m.y);
}
// The table entry exp(-bpade it / (10^4 - it)) (1e-20 for the last) and its complement, the series below 0.06
// (evaluated instead of loaded, within a few float ulps of the table's float value for the arguments that matter; bpade
// log2(e) folded into one constant).
__device__ __forceinline__ float sw4_entry(float it)
{
    const float e = ex2a(__fdividef(-5.18955054f * it, 10000.0f - it));
    return it >= 10000.0f ? 1.0e-20f : e;
}
__device__ __forceinline__ F2 sw4_tblexp(F2 zb, const SwPos2& p, F2& em)
{
    const F2 et{sw4_entry(p.it.x), sw4_entry(p.it.y)};
    const F2 h = fma2(zb * -0.5f, zb, zb), ec = 1.0f - et, es = 1.0f - h;
    const bool s0 = zb.x <= 0.06f, s1 = zb.y <= 0.06f;
    em = F2{s0 ? h.x : ec.x, s1 ? h.y : ec.y};
    return F2{s0 ? es.x : et.x, s1 ? es.y : et.y};
}
// A depth along the beam with the last entry instead of an infinite one (a NaN stays).
__device__ __forceinline__ F2 sw4_cap(F2 zb) { return F2{zb.x > 1.0e30f ? 1.0e30f : zb.x, zb.y > 1.0e30f ? 1.0e30f : zb.y}; }
// What a float R/T is left with: nothing, a neighbouring table entry to test, or the resonance in float64.
enum : int { SW4_Q_NONE = 0, SW4_Q_NEAR = 1, SW4_Q_RES = 2 };
// The float R/T of sw2_rt_mixed (prologue of two-stream mode MODE, R/T, direct transmissions) without branches; q0 / q1 say where
// sw2_rt_mixed would take a float64 step or test a neighbouring table entry (the outputs are then not used).
// ASY = false: the asymmetry is zero (the clear pass without aerosol, 85 % of the work), so delta scaling changes
// nothing and the three direct-beam exponentials are one.
template <int MODE, bool ASY>
__device__ __forceinline__ void sw4_rt(F2 t0, F2 tabs, F2 s0, F2 y0, float cz, float snt, F2 wk, F2 wf, SwRT2& r, int& q0,
                                       int& q1)
{
    const float ftiny = 1.0e-12f;
    const float cwmin = (float)(1.0 - ((double)1.0f - (double)1.0e-6f));
    // co-albedo over F2_DOWN, from a scaled divisor: the depth may be any finite float
    const F2 ts = t0 * F2_DOWN, cw = max2(quot2(tabs, ts, rcp2(ts)), cwmin / F2_DOWN);
    const F2 zssaw = nma2(cw, f2(F2_DOWN), f2(1.0f));
    F2 ztau1, zssa1, cw1, zasy1, zasy3;      // cw1 over F2_DOWN as cw
    if constexpr (ASY) {
        const F2 sm = max2(s0, ftiny) * F2_DOWN, zasyw = quot2(y0, sm, rcp2(sm)) * F2_DOWN;
        const F2 za2s = zssaw * (zasyw * zasyw);
        const F2 om = 1.0f - za2s, ro = rcp2(om);
        ztau1 = om * t0;
        zssa1 = quot2(zssaw - za2s, om, ro);
        cw1 = quot2(cw, om, ro);
        const F2 z1 = zasyw + 1.0f;
        zasy1 = quot2(zasyw, z1, rcp2(z1));
        zasy3 = zasy1 * 0.75f;
    } else {
        ztau1 = t0; zssa1 = zssaw; cw1 = cw; zasy1 = f2(0.0f); zasy3 = f2(0.0f);
    }
    F2 g1, g2, g3, gm, gp;
    if constexpr (MODE == 2) {
        g1 = ASY ? nma2(zssa1, zasy3 + 1.25f, f2(2.0f)) : fma2(zssa1, f2(-1.25f), f2(2.0f));
        g2 = ASY ? (zssa1 * 0.75f) * (1.0f - zasy1) : zssa1 * 0.75f;
        g3 = ASY ? nma2(zasy3, f2(cz), f2(0.5f)) : f2(0.5f);
        gm = cw1 * (2.0f * F2_DOWN);
        gp = ASY ? nma2(zssa1, fma2(zasy1, f2(1.5f), f2(0.5f)), f2(2.0f)) : fma2(zssa1, f2(-0.5f), f2(2.0f));
    } else if constexpr (MODE == 1) {
        g1 = nma2(zssa1, zasy3 + 1.0f, f2(1.75f));
        g2 = nma2(zssa1, 1.0f - zasy3, f2(-0.25f));
        g3 = nma2(zasy3, f2(cz), f2(0.5f));
        gm = g1 - g2;
        gp = g1 + g2;
    } else {
        const float zsr3 = 1.7320508f;
        g1 = nma2(zssa1, zasy1 + 1.0f, f2(2.0f)) * zsr3 * 0.5f;
        g2 = (zssa1 * zsr3) * (1.0f - zasy1) * 0.5f;
        g3 = nma2(zasy1 * zsr3, f2(cz), f2(1.0f)) * 0.5f;
        gm = cw1 * (zsr3 * F2_DOWN);
        gp = nma2(zssa1, zasy1, f2(1.0f)) * zsr3;
    }
    const F2 g4 = 1.0f - g3;
    const F2 zrk = sqrt2(gm * gp);
    const F2 zrp = zrk * cz;
    const F2 zrpp0 = (1.0f - zrp) * (zrp + 1.0f);
    const F2 zbd = ztau1 * snt, zb1 = min2(zrk * ztau1, 500.0f), zb2 = min2(zbd, 500.0f), zb4 = ASY ? sw4_cap(t0 * snt) : zbd;
    const SwPos2 p1 = sw4_pos(zb1), p2 = sw4_pos(zb2);
    F2 em1, em2, em;
    const F2 e1 = sw4_tblexp(zb1, p1, em1), e2 = sw4_tblexp(zb2, p2, em2);
    // exp(-ztau1 / mu0): e2's entry; past its clamp at 500 the entries underflow to 0 in float, up to the last one
    // (10^4 ft + 1/2 >= 10^4 from zb = 71,939 on), which the table sets to 1e-20
    const F2 eb{zbd.x > 500.0f ? (zbd.x >= 71939.0f ? 1.0e-20f : 0.0f) : e2.x,
                zbd.y > 500.0f ? (zbd.y >= 71939.0f ? 1.0e-20f : 0.0f) : e2.y};
    r.e3 = eb;
    bool n10, n11, n20, n21, n40, n41;
    sw4_near(zb1, p1, n10, n11);
    sw4_near(zb2, p2, n20, n21);
    if constexpr (ASY) {
        const SwPos2 p4 = sw4_pos(zb4);
        r.e4 = sw4_tblexp(zb4, p4, em);
        sw4_near(zb4, p4, n40, n41);
    } else {
        r.e4 = eb;
        n40 = n20 && zbd.x <= 500.0f;
        n41 = n21 && zbd.y <= 500.0f;
    }
    auto code = [](float zrpp, float wk, bool n12, float wf, bool n4) {
        return fabsf(zrpp) < SW2_RESONANCE ? SW4_Q_RES : (wk > 0.0f && n12) || (wf * 4.0e-4f > 1.0f && n4) ? SW4_Q_NEAR : SW4_Q_NONE;
    };
    q0 = code(zrpp0.x, wk.x, n10 || n20, wf.x, n40);
    q1 = code(zrpp0.y, wk.y, n11 || n21, wf.y, n41);
    // sw2_rt_core with the clamp and the degenerate-denominator case as selects
    const float eps1 = 1.0e-8f;
    const F2 zrpp{fabsf(zrpp0.x) < eps1 ? copysignf(eps1, zrpp0.x) : zrpp0.x,
                  fabsf(zrpp0.y) < eps1 ? copysignf(eps1, zrpp0.y) : zrpp0.y};
    const F2 za1 = fma2(g1, g4, g2 * g3), za2 = fma2(g1, g3, g2 * g4);
    const F2 e11 = e1 * e1, em11 = em1 * (2.0f - em1);
    const F2 B = fma2(zrk, e11 + 1.0f, g1 * em11);
    const F2 D = zrpp * B;
    const F2 q = quot2(zssa1, D, rcp2(D));
    const F2 m11 = em1 * em1, e1m2 = (e1 * em2) * 2.0f;
    const F2 nr = fma2(em11, nma2(zrk * g3, zrp, za2), (zrk * nma2(za2, f2(cz), g3)) * (m11 + e1m2));
    const F2 nt = nma2(e2 * em11, fma2(zrk * g4, zrp, za1), (zrk * fma2(za1, f2(cz), g4)) * nma2(e2, m11, e1m2));
    const F2 rb = clamp01(nr * q), tb = clamp01(fma2(nt, q, e2));
    const bool d0 = fabsf(D.x) <= eps1 * e1.x, d1 = fabsf(D.y) <= eps1 * e1.y;
    r.rb = F2{d0 ? eps1 : rb.x, d1 ? eps1 : rb.y};
    r.tb = F2{d0 ? e2.x : tb.x, d1 ? e2.y : tb.y};
    // td is ~1 in the thin layers, where its rounding acts as absorption that adds up down the column: the Newton step
    // halves the fluxes' error against float64 (sfcfsw 2.8e-7 -> 1.7e-7 relative)
    const F2 rB = rcp2(B);
    r.rd = clamp01(quot2(g2 * em11, B, rB));
    r.td = clamp01(quot2((zrk + zrk) * e1, B, rB));
}

// The column image handed from the gas-optics kernel to the R/T kernel: SwSh2 from colmol to its end (taug last)
// and, with aerosol, the aerosol block after it, rounded up to 16-byte units.
__host__ __device__ constexpr size_t sw4_image_begin() { return offsetof(SwSh2, colmol); }
__host__ __device__ constexpr size_t sw4_image_bytes(bool aer)
{
    return ((sizeof(SwSh2) - sw4_image_begin() + (aer ? sizeof(SwAer) : 0)) + 15) / 16 * 16;
}
static_assert(offsetof(SwSh2, colmol) % 16 == 0, "the image starts on a 16-byte boundary");
static_assert(offsetof(SwSh2, taug) + sizeof(SwSh2::taug) == sizeof(SwSh2) && sizeof(SwAer) % 16 == 0,
              "taug closes SwSh2 and the aerosol block is whole 16-byte units");
// Shared memory of the gas-optics kernel: SwSh2 up to taug (taug goes to the image directly), the aerosol block
// where taug would be.
__host__ __device__ constexpr size_t sw4_gas_smem(bool aer) { return offsetof(SwSh2, taug) + (aer ? sizeof(SwAer) : 0); }

// The image's taug part holds the gas optical depths as [layer][g-point]: the R/T kernel reads them straight from
// the image, 32 consecutive (layer, g-point) tasks per warp on one 128-byte line, instead of staging them.
static_assert((size_t)NLAY_MAX * SW_NGPT * sizeof(float) <= sizeof(SwSh2::taug), "[layer][g] fits the taug part");
__host__ __device__ inline const float* sw4_image_taug(const int4* im)
{
    return reinterpret_cast<const float*>(reinterpret_cast<const unsigned char*>(im) + (offsetof(SwSh2, taug) - sw4_image_begin()));
}

// Set-up, cloud optics and gas optics of one sunlit column (one CTA, six per SM) into its image.
__global__ void __launch_bounds__(SW4_GAS_THREADS, SW4_GAS_MINB)
sw4_gas_kernel(const __grid_constant__ SwBatch bt, int any_aer, int* err, int d0, int4* img, Sw4Lists lists)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SwSh2& s = *reinterpret_cast<SwSh2*>(smem_raw);
    if (blockIdx.x == 0 && threadIdx.x < SW4_LIST_HEAD) lists.head[threadIdx.x] = 0;   // the tile's work lists start empty
    const int d = d0 + (int)blockIdx.x;
    if (d >= *bt.req[0].nday) return;
    const int64_t gcol = bt.req[0].daycol[d];
    const int rq = bt.find(gcol);
    const SwIn& a = bt.req[rq];
    const int nlay = a.nlay;
    if (nlay > NLAY_MAX) {
        if (threadIdx.x == 0) atomicExch(err, RAD_DEV_NLAY);
        return;
    }
    SwAer* aer = a.faersw ? reinterpret_cast<SwAer*>(smem_raw + offsetof(SwSh2, taug)) : nullptr;
    const int64_t col = gcol - bt.off[rq];
    const int tid = threadIdx.x;
    int4* im = img + (size_t)blockIdx.x * (sw4_image_bytes(any_aer) / 16);
    float* img_taug = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(im) + (offsetof(SwSh2, taug) - sw4_image_begin()));
    sw2_setup<SW4_GAS_THREADS>(s, aer, a, col, d, tid);
    for_each_band_flat<2>(c_sw_ns, 14, nlay, &s.task_next, tid & 31, [&](int g, int k0, int b) {
        P2 tg, tr;
        sw_gas<float>(s, g, k0, tg, tr, b);
        *reinterpret_cast<float2*>(img_taug + k0 * SW_NGPT + g) = make_float2(tg.x, tg.y);
        if (b == 8 && k0 < s.laytrop) { s.taur24[g - 66][k0] = tr.x; s.taur24[g - 65][k0] = tr.y; }
    });
    __syncthreads();
    const int4* sm = reinterpret_cast<const int4*>(smem_raw + sw4_image_begin());
    const int n1 = (int)((offsetof(SwSh2, taug) - sw4_image_begin()) / 16);
    const int n2 = any_aer ? (int)(sizeof(SwAer) / 16) : 0;
    const int skip = (int)(sizeof(SwSh2::taug) / 16);
    for (int i = tid; i < n1 + n2; i += SW4_GAS_THREADS) im[i < n1 ? i : i + skip] = sm[i];
}

// The column image (without taug; the aerosol block where taug would be) from global memory into the CTA's shared
// memory, every 16-byte piece in flight at once (cp.async.cg: L2 to shared).  Returns the SwSh2 the shared memory
// stands for: only its part from colmol on is there, so the image starts at smem and SwSh2 itself before it.
__device__ __forceinline__ SwSh2* sw4_load_image(unsigned char* smem, const int4* im, int any_aer, int tid, int nthreads)
{
    const uint32_t sb = (uint32_t)__cvta_generic_to_shared(smem);
    const int n1 = (int)((offsetof(SwSh2, taug) - sw4_image_begin()) / 16);
    const int n2 = any_aer ? (int)(sizeof(SwAer) / 16) : 0;
    const int skip = (int)(sizeof(SwSh2::taug) / 16);
    for (int i = tid; i < n1 + n2; i += nthreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sb + 16u * (uint32_t)i), "l"(im + (i < n1 ? i : i + skip))
                     : "memory");
    return reinterpret_cast<SwSh2*>(smem - sw4_image_begin());
}
__host__ __device__ constexpr size_t sw4_rt_smem(bool aer) { return sw4_gas_smem(aer) - sw4_image_begin(); }

__global__ void __launch_bounds__(SW4_RT_THREADS, SW4_OPT_MINB)
sw4_rt_kernel(const __grid_constant__ SwBatch bt, int any_aer, int d0, const int4* img, unsigned char* scr, size_t blk_bytes,
              int* list_head, int2* items)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int d = d0 + (int)blockIdx.x;
    if (d >= *bt.req[0].nday) return;
    const int64_t gcol = bt.req[0].daycol[d];
    const int rq = bt.find(gcol);
    const SwIn& a = bt.req[rq];
    const int nlay = a.nlay;
    if (nlay > NLAY_MAX) return;                                   // flagged by the gas-optics kernel
    const int tid = threadIdx.x;
    const int4* im = img + (size_t)blockIdx.x * (sw4_image_bytes(any_aer) / 16);
    const float* tgi = sw4_image_taug(im);   // [layer][g], read from the image as the tasks need it
    if (SW4_L2PF && tid == 0) l2_prefetch(tgi, (uint32_t)(nlay * SW_NGPT * sizeof(float)));
    SwSh2& s = *sw4_load_image(smem_raw, im, any_aer, tid, SW4_RT_THREADS);
    const SwAer* aer = a.faersw ? reinterpret_cast<const SwAer*>(smem_raw + sw4_rt_smem(false)) : nullptr;
    unsigned char* blk = scr + (size_t)blockIdx.x * blk_bytes;
    Sw4Hdr& H = *reinterpret_cast<Sw4Hdr*>(blk);
    float* rtc = reinterpret_cast<float*>(blk + sw4_hdr_bytes());
    float* rto = rtc + (size_t)nlay * SW4_LAYER;
    uint16_t* queue = reinterpret_cast<uint16_t*>(blk + sw4_queue_offset(nlay));
    const bool mc = a.mask != nullptr;
    constexpr int NP = SW_NGPT / 2;
    __shared__ int qnear, qres;                    // float64 queue: entries from the front, from the back
    __shared__ unsigned qbit[NLAY_MAX][4];
    __shared__ signed char slotk[NLAY_MAX];
    __shared__ unsigned char gband[SW_NGPT];
    __shared__ __align__(8) float zsol[SW_NGPT];   // solar source of each g-point, H.zsolar
    __shared__ float rdf[NLAY_MAX];                // heatfac / delp as float
    for (int j = tid; j < NLAY_MAX * 4; j += SW4_RT_THREADS) qbit[j >> 2][j & 3] = 0u;
    if (tid == 0) { qnear = 0; qres = 0; }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const bool cloudy = mc ? s.zcf1 > 0.0f : s.zcf1 > 1.0e-6f, clr5 = a.iswmode != 1 && !aer;
    // layers with a cloudy-pass R/T, counted from the surface (every warp forms the two words of layer bits)
    unsigned cw[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int k0 = 32 * h + (tid & 31);
        cw[h] = __ballot_sync(0xffffffffu, cloudy && k0 < nlay && s.cldfrc[k0] > 1.0e-12f);
    }
    const int ncl = __popc(cw[0]) + __popc(cw[1]);
    for (int k0 = tid; k0 < nlay; k0 += SW4_RT_THREADS) {
        const unsigned below = (1u << (k0 & 31)) - 1u;
        const int sl = k0 < 32 ? __popc(cw[0] & below) : __popc(cw[0]) + __popc(cw[1] & below);
        const bool cl = (cw[k0 >> 5] >> (k0 & 31)) & 1u;
        H.slot[k0] = cl ? (signed char)sl : (signed char)-1;
        if (cl) slotk[sl] = (signed char)k0;
        H.rdelp[k0] = s.rdelp[k0];
        rdf[k0] = (float)s.rdelp[k0];
    }
    for (int g = tid; g < SW_NGPT; g += SW4_RT_THREADS) {
        gband[g] = c_sw_band[g];
        const float z = s.ssolar * s.sfluxzen[g];
        zsol[g] = z;
        H.zsolar[g] = z;
    }
    if (tid == 0) {
        H.ncl = ncl;
        H.clr5 = clr5 ? 1 : 0;
        H.cloudy = cloudy ? 1 : 0;
        H.albbm[0] = s.albbm[0]; H.albbm[1] = s.albbm[1];
        H.albdf[0] = s.albdf[0]; H.albdf[1] = s.albdf[1];
        H.zcf0 = s.zcf0; H.zcf1 = s.zcf1;
    }
    const float cz = s.cosz, snt = s.sntz;
    __syncthreads();
    // ---- layer R/T in two passes over the column; a task is a pair of neighbouring g-points of one layer (every
    // band starts at an even g-point and has an even count, so the pair shares its band's optics), lanes on 32
    // consecutive pairs of the [layer][g-point pair] order.  A g-point whose R/T needs a float64 step or a
    // table-entry test is queued once (qbit marks it) for sw4_fix_kernel
    auto enqueue = [&](int k0, int g, int code) {
        if (atomicOr(&qbit[k0][g >> 5], 1u << (g & 31)) & (1u << (g & 31))) return;   // queued already
        const int e = code == SW4_Q_NEAR ? atomicAdd(&qnear, 1) : nlay * SW_NGPT - 1 - atomicAdd(&qres, 1);
        queue[e] = (uint16_t)(k0 * SW_NGPT + g);
    };
    auto ld2 = [](const float* p) { const float2 v = *reinterpret_cast<const float2*>(p); return F2{v.x, v.y}; };
    auto st2 = [](float* p, F2 v) { *reinterpret_cast<float2*>(p) = make_float2(v.x, v.y); };
    // clear-pass inputs of the pair (g, g + 1) of layer k0
    auto inputs = [&](int k0, int g, int ib, F2& t0, F2& ab, F2& s0, F2& y0) {
        const float2 tv = __ldg(reinterpret_cast<const float2*>(tgi + k0 * SW_NGPT + g));
        const F2 tg{tv.x, tv.y};
        F2 tr;
        if (g >= 66 && g < 74 && k0 < s.laytrop) tr = F2{s.taur24[g - 66][k0], s.taur24[g - 65][k0]};
        else tr = ld2(s.raylc + g) * s.colmol[k0];
        t0 = tr + tg; s0 = tr; y0 = f2(0.0f); ab = tg;
        if (aer) {
            t0 = t0 + aer->tau[ib][k0]; s0 = s0 + aer->tasa[ib][k0]; y0 = f2(aer->tay[ib][k0]);
            ab = ab + aer->tabs[ib][k0];
        }
        t0 = max2(t0, 1.0e-12f);
    };
    auto weights = [&](int k0, int g, F2& wk, F2& wf) {
        const F2 zs = ld2(zsol + g);
        wf = zs * (1.0f / SW2_FLUX_T);
        wk = zs * (1.5f * 86400.0f / SW2_HEAT_T) * rdf[k0];
    };
    auto put = [&](float* p, const SwRT2& r, bool e4) {   // p: the pair's place in field 0 of its layer's rows
        st2(p, r.rb); st2(p + SW_NGPT, r.rd); st2(p + 2 * SW_NGPT, r.tb); st2(p + 3 * SW_NGPT, r.td);
        st2(p + 4 * SW_NGPT, r.e3);
        if (e4) st2(p + 5 * SW_NGPT, r.e4);
    };
    auto run = [&](auto mode_tag) {
        constexpr int MODE = decltype(mode_tag)::value;
        // clear pass
        auto clear = [&](auto asy_tag) {
            for (int i = tid; i < nlay * NP; i += SW4_RT_THREADS) {
                const int k0 = i / NP, g = 2 * (i - k0 * NP);
                F2 t0, ab, s0, y0, wk, wf;
                inputs(k0, g, gband[g], t0, ab, s0, y0);
                weights(k0, g, wk, wf);
                SwRT2 r;
                int q0, q1;
                sw4_rt<MODE, decltype(asy_tag)::value>(t0, ab, s0, y0, cz, snt, wk, wf, r, q0, q1);
                put(rtc + (size_t)k0 * SW4_LAYER + g, r, decltype(asy_tag)::value);
                if (q0) enqueue(k0, g, q0);
                if (q1) enqueue(k0, g + 1, q1);
            }
        };
        if (MODE == 1 || !clr5) clear(std::true_type{});
        else if constexpr (MODE != 1) clear(std::false_type{});
        __syncthreads();
        // cloudy pass: the layers with a slot, mixture R/T blended with the clear R/T (or, McICA, taken
        // unblended where the g-point's sub-column bit is set)
        for (int j = tid; j < ncl * NP; j += SW4_RT_THREADS) {
            const int sl = j / NP, g = 2 * (j - sl * NP), k0 = slotk[sl], ib = gband[g];
            F2 t0, ab, s0, y0, wk, wf;
            inputs(k0, g, ib, t0, ab, s0, y0);
            weights(k0, g, wk, wf);
            int q0, q1;
            SwRT2 m;
            sw4_rt<MODE, true>(t0 + s.taucw[ib][k0], ab + s.tabsc[ib][k0], s0 + s.ssacw[ib][k0], y0 + s.asycw[ib][k0], cz,
                               snt, wk, wf, m, q0, q1);
            const float* pc = rtc + (size_t)k0 * SW4_LAYER + g;
            const SwRT2 c{ld2(pc), ld2(pc + SW_NGPT), ld2(pc + 2 * SW_NGPT), ld2(pc + 3 * SW_NGPT), ld2(pc + 4 * SW_NGPT),
                          ld2(pc + (clr5 ? 4 : 5) * SW_NGPT)};
            if (mc) {
                const unsigned w = s.mcw[g >> 5][k0] >> (g & 31);
                const bool b0 = w & 1u, b1 = w & 2u;
                auto pick = [&](F2 x, F2 y) { return F2{b0 ? x.x : y.x, b1 ? x.y : y.y}; };
                m.rb = pick(m.rb, c.rb); m.rd = pick(m.rd, c.rd); m.tb = pick(m.tb, c.tb); m.td = pick(m.td, c.td);
                m.e3 = pick(m.e3, c.e3); m.e4 = pick(m.e4, c.e4);
                q0 = b0 ? q0 : SW4_Q_NONE;
                q1 = b1 ? q1 : SW4_Q_NONE;
            } else {
                const float zc1 = s.cldfrc[k0], zc0 = 1.0f - zc1;
                auto mix = [&](F2 x, F2 y) { return fma2(y, f2(zc0), x * zc1); };
                m.rb = mix(m.rb, c.rb); m.rd = mix(m.rd, c.rd); m.tb = mix(m.tb, c.tb); m.td = mix(m.td, c.td);
                m.e3 = mix(m.e3, c.e3); m.e4 = mix(m.e4, c.e4);
            }
            put(rto + (size_t)sl * SW4_LAYER + g, m, true);
            if (q0) enqueue(k0, g, q0);
            if (q1) enqueue(k0, g + 1, q1);
        }
    };
    if (a.iswmode == 1) run(std::integral_constant<int, 1>{});
    else if (a.iswmode == 2) run(std::integral_constant<int, 2>{});
    else run(std::integral_constant<int, 3>{});
    __syncthreads();
    // ---- the column's queue as work items of the tile
    if (tid == 0) {
        const int n1 = (qnear + SW4_FIX_THREADS - 1) / SW4_FIX_THREADS, n2 = (qres + SW4_FIX_THREADS - 1) / SW4_FIX_THREADS;
        if (n1 + n2 > 0) {
            int2* it = items + atomicAdd(list_head, n1 + n2);
            for (int j = 0; j < n1; ++j) {
                const int e = j * SW4_FIX_THREADS;
                it[j] = make_int2((int)blockIdx.x, e | min(SW4_FIX_THREADS, qnear - e) << 16);
            }
            for (int j = 0; j < n2; ++j) {
                const int e = j * SW4_FIX_THREADS;
                it[n1 + j] = make_int2((int)blockIdx.x, nlay * SW_NGPT - qres + e | min(SW4_FIX_THREADS, qres - e) << 16);
            }
        }
    }
}

// The complete layer function of queue entry i = k0 * SW_NGPT + g of column c of the tile over the float R/T that
// sw4_rt_kernel wrote.  s, aer: the column's image, in shared or global memory.  With defer, a g-point that needs the
// float64 recompute from the column's inputs (sw2_exact) is left alone and true returned.
__device__ __forceinline__ bool sw4_fix_entry(const SwIn& a, int64_t col, const SwSh2& s, const SwAer* aer, const float* taug,
                                              unsigned char* blk, const float* ex, const double* exd, int i, bool defer)
{
    const int nlay = a.nlay, k0 = i / SW_NGPT, g = i - k0 * SW_NGPT;
    const Sw4Hdr& H = *reinterpret_cast<const Sw4Hdr*>(blk);
    const float zsolar = H.zsolar[g];
    const double czd = (double)__ldg(a.coszen + col);
    int pending = 0;
    const SwExactCtx x{&a, col, s.laytrop, s.kmin8, s.kminw, a.iswmode, czd, 1.0 / czd, exd,
                       zsolar * (1.5f * 86400.0f / SW2_HEAT_T), zsolar * (1.0f / SW2_FLUX_T), defer ? &pending : nullptr};
    const SwLayerRT2 L = sw2_layer(s, aer, x, k0, g, c_sw_band[g], H.cloudy != 0, a.mask != nullptr, s.cosz, s.sntz, ex,
                                   __ldg(taug + i));
    if (pending) return true;
    float* pc = reinterpret_cast<float*>(blk + sw4_hdr_bytes()) + (size_t)k0 * SW4_LAYER + g;
    pc[0] = L.c.rb; pc[SW_NGPT] = L.c.rd; pc[2 * SW_NGPT] = L.c.tb; pc[3 * SW_NGPT] = L.c.td;
    pc[4 * SW_NGPT] = L.c.e3; pc[5 * SW_NGPT] = L.c.e4;
    const int sl = H.slot[k0];
    if (sl >= 0) {
        float* po = pc + (size_t)(nlay - k0 + sl) * SW4_LAYER;
        po[0] = L.o.rb; po[SW_NGPT] = L.o.rd; po[2 * SW_NGPT] = L.o.tb; po[3 * SW_NGPT] = L.o.td;
        po[4 * SW_NGPT] = L.o.e3; po[5 * SW_NGPT] = L.o.e4;
    }
    return false;
}

// The queued g-points of a tile.  A column has ~50 near-entry tests and, in the 1 % of columns with mu0 near a two-stream
// resonance that all strongly absorbing layers share, thousands of float64 R/T; so the tile's queue is cut into items of
// at most 64 entries of one column, which a grid of resident CTAs walks.  The ~2.5 g-points per column that need the
// recompute from the inputs go to sw4_exact_kernel (cap > 0): in here each of them holds its warp alone, half of the
// kernel's time -- 3.41 ms per 131,072 columns against 1.70 + 0.23 ms.  A small tile has warps to spare and would pay the
// second kernel's latency instead (1,024 columns: 37 us against 20 + 42 us), so from SW4_EXACT_MIN columns on.
constexpr int64_t SW4_EXACT_MIN = 4096;
__global__ void __launch_bounds__(SW4_FIX_THREADS, SW4_FIX_MINB)
sw4_fix_kernel(const __grid_constant__ SwBatch bt, int any_aer, const float* ex, const double* exd, int d0, const int4* img,
               unsigned char* scr, size_t blk_bytes, Sw4Lists lists)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = lists.head[0], tid = threadIdx.x;
    for (int w = blockIdx.x; w < n; w += gridDim.x) {
        const int2 it = lists.items[w];
        const int64_t gcol = bt.req[0].daycol[d0 + it.x];
        const int rq = bt.find(gcol);
        const SwIn& a = bt.req[rq];
        const int4* im = img + (size_t)it.x * (sw4_image_bytes(any_aer) / 16);
        const SwSh2& s = *sw4_load_image(smem_raw, im, any_aer, tid, SW4_FIX_THREADS);
        const SwAer* aer = a.faersw ? reinterpret_cast<const SwAer*>(smem_raw + sw4_rt_smem(false)) : nullptr;
        unsigned char* blk = scr + (size_t)it.x * blk_bytes;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const int e0 = it.y & 0xffff, ne = it.y >> 16;
        if (tid < ne) {
            const int i = reinterpret_cast<const uint16_t*>(blk + sw4_queue_offset(a.nlay))[e0 + tid];
            bool defer = lists.cap > 0;
            while (sw4_fix_entry(a, gcol - bt.off[rq], s, aer, sw4_image_taug(im), blk, ex, exd, i, defer)) {
                const int b = c_sw_band[i % SW_NGPT], j = atomicAdd(lists.head + 1 + b, 1);
                if (j < lists.cap) {
                    lists.exact[(size_t)b * lists.cap + j] = make_int2(it.x, i);
                    break;
                }
                defer = false;                     // the band's list is full: here after all
            }
        }
        __syncthreads();                           // shared memory is reused by the next item
    }
}

// The g-points that sw4_fix_kernel left to the float64 recompute, warp by warp from one band's list, so that the lanes
// of a warp run the same band's gas optics.
constexpr int SW4_EXACT_THREADS = 128, SW4_EXACT_MINB = 4;
__global__ void __launch_bounds__(SW4_EXACT_THREADS, SW4_EXACT_MINB)
sw4_exact_kernel(const __grid_constant__ SwBatch bt, int any_aer, const float* ex, const double* exd, int d0, const int4* img,
                 unsigned char* scr, size_t blk_bytes, Sw4Lists lists)
{
    const int lane = threadIdx.x & 31, nw = gridDim.x * (SW4_EXACT_THREADS / 32);
    int w = blockIdx.x * (SW4_EXACT_THREADS / 32) + (threadIdx.x >> 5);     // this warp's next 32 entries
    for (int b = 0; b < 14; ++b) {
        const int n = min(lists.head[1 + b], lists.cap), nt = (n + 31) >> 5;
        for (; w < nt; w += nw) {
            const int j = 32 * w + lane;
            if (j >= n) continue;
            const int2 e = lists.exact[(size_t)b * lists.cap + j];
            const int64_t gcol = bt.req[0].daycol[d0 + e.x];
            const int rq = bt.find(gcol);
            const SwIn& a = bt.req[rq];
            const unsigned char* im = reinterpret_cast<const unsigned char*>(img + (size_t)e.x * (sw4_image_bytes(any_aer) / 16));
            const SwSh2& s = *reinterpret_cast<const SwSh2*>(im - sw4_image_begin());
            const SwAer* aer = a.faersw ? reinterpret_cast<const SwAer*>(im + sizeof(SwSh2) - sw4_image_begin()) : nullptr;
            sw4_fix_entry(a, gcol - bt.off[rq], s, aer, sw4_image_taug(reinterpret_cast<const int4*>(im)),
                          scr + (size_t)e.x * blk_bytes, ex, exd, e.y, false);
        }
        w -= nt;
    }
}

// Per-g-point level fluxes of one sunlit column for swrad's optional outputs (DIAG sweeps):
// [nlay + 1][SW4_PGQ][SW_NGPT] floats at level L (surface first), each x zsolar: up, down and net (down - up) of the clear
// pass (q 0..2), then of the cloudy pass (q 3..5, written for a cloudy column).
constexpr int SW4_PGQ = 6;
__host__ __device__ constexpr int64_t sw4_pg_floats(int nlay) { return (int64_t)(nlay + 1) * SW4_PGQ * SW_NGPT; }

// One level of the DIAG profile of the pair g, g + 1 in one pass (see sw4_pg_floats).
__device__ __forceinline__ void sw4_pg_level(float* pg, int L, int g, int pass, F2 zsolar, F2 fu, F2 fd)
{
    float* p = pg + ((size_t)L * SW4_PGQ + 3 * pass) * SW_NGPT + g;
    auto one = [&](float* q, double z, double u, double d) {
        q[0] = (float)(z * u);
        q[SW_NGPT] = (float)(z * d);
        q[2 * SW_NGPT] = (float)(z * (d - u));
    };
    one(p, zsolar.x, fu.x, fd.x);
    one(p + 1, zsolar.y, fu.y, fd.y);
}

// The steps of the adding method (sw2_up, sw2_flux, sw2_down) on a pair of g-points.
__device__ __forceinline__ void sw4_up(const SwRT2& L, F2& ub, F2& ud)
{
    const F2 den = rcp2(nma2(ud, L.rd, f2(1.0f)));
    ub = fma2(L.td * fma2(L.tb - L.e3, ud, L.e3 * ub), den, L.rb);
    ud = fma2(L.td * L.td * ud, den, L.rd);
}
__device__ __forceinline__ void sw4_flux(F2 ub, F2 ud, F2 tdn, F2 rdn, F2 tdb, F2& fu, F2& fd)
{
    const F2 den = rcp2(nma2(rdn, ud, f2(1.0f))), dif = tdn - tdb, bu = tdb * ub;
    fu = fma2(dif, ud, bu) * den;
    fd = fma2(fma2(bu, rdn, dif), den, tdb);
}
__device__ __forceinline__ void sw4_down(const SwRT2& L, F2& tdn, F2& rdn, F2& tdb)
{
    const F2 den = rcp2(nma2(L.rd, rdn, f2(1.0f)));
    tdn = fma2(L.td * fma2(tdb * L.rb, rdn, tdn - tdb), den, tdb * L.tb);
    rdn = fma2(L.td * L.td * rdn, den, L.rd);
    tdb = L.e3 * tdb;
}

// Sums of four doubles over the warp: lane 8 j holds v[j]'s (a fixed tree: the four values are folded into the lanes as
// the sums halve, 12 shuffles and 6 additions instead of four warp_sum's 40 and 20).
__device__ __forceinline__ double warp_sum4(const double* v, int lane)
{
    const bool h = lane & 16, q = lane & 8;
    double a = h ? v[2] : v[0], b = h ? v[3] : v[1];
    a += __shfl_xor_sync(0xffffffffu, h ? v[0] : v[2], 16);
    b += __shfl_xor_sync(0xffffffffu, h ? v[1] : v[3], 16);
    double c = q ? b : a;
    c += __shfl_xor_sync(0xffffffffu, q ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    return c;
}

// The adding method of one sunlit column from its block (sw2_column phase C with the R/T read instead of formed).  Four
// warps per column: warps 0 and 1 run the clear pass, warps 2 and 3 the cloudy one (idle in a cloudless column), a lane
// per pair of g-points (28 lanes each), so a pass's chain of layers is not lengthened by the other's.  Bound: the latency
// of a segment's rows and of the recurrence (3.6 TB/s of R/T rows read, 44 % of the DRAM peak).  Measured per 131,072 columns (65,536 sunlit):
// 6.47 ms with both passes and one g-point per lane at 80 registers; the same with pairs and both passes in two warps
// (168 registers, 6 CTAs per SM: latency); 5.06 ms with the passes in warps of their own and the four levels of a segment
// summed together.
template <bool DIAG = false>
__global__ void __launch_bounds__(SW4_SWEEP_THREADS, SW4_SWEEP_MINB)
sw4_sweep_kernel(const __grid_constant__ SwBatch bt, int d0, int nc, const unsigned char* scr,
                 size_t blk_bytes, float* __restrict__ pg = nullptr)
{
    extern __shared__ __align__(16) float2 ckpt[];                 // [(nseg - 1) x 2][SW4_SWEEP_THREADS]
    __shared__ __align__(16) Sw4Hdr H;
    __shared__ double fn[SW4_SWEEP_WARPS][NLAY_MAX + SW2_SEG + 1];
    __shared__ double scs[SW4_SWEEP_WARPS][9];
    const int i = (int)blockIdx.x;
    const int d = d0 + i;
    if (i >= nc || d >= *bt.req[0].nday) return;
    const int64_t gcol = bt.req[0].daycol[d];
    const int rq = bt.find(gcol);
    const SwIn& a = bt.req[rq];
    const int nlay = a.nlay;
    if (nlay > NLAY_MAX) return;                                   // flagged by the optics kernel
    const int64_t N = a.ncol;
    const int64_t col = gcol - bt.off[rq];
    const int tid = threadIdx.x;
    const unsigned char* blk = scr + (size_t)i * blk_bytes;
    {
        const int4* src = reinterpret_cast<const int4*>(blk);
        int4* dst = reinterpret_cast<int4*>(&H);
        for (int j = tid; j < (int)(sizeof(Sw4Hdr) / 16); j += SW4_SWEEP_THREADS) dst[j] = __ldg(src + j);
    }
    __syncthreads();
    const float* rtc = reinterpret_cast<const float*>(blk + sw4_hdr_bytes());
    const float* rto = rtc + (size_t)nlay * SW4_LAYER;
    if (DIAG) pg += (int64_t)i * sw4_pg_floats(nlay);
    const int warp = tid >> 5, lane = tid & 31;
    constexpr int LANES = SW_NGPT / 4;
    const int pass = warp >> 1;                                    // 0 clear, 1 cloudy
    const bool act = lane < LANES;                                 // idle lanes mirror the warp's last pair
    const int g = 2 * ((warp & 1) * LANES + min(lane, LANES - 1));
    const int ib0 = c_sw_band[g];
    const int ibd = ib0 == 8 ? 0 : ((ib0 >= 9 && ib0 <= 12) ? 2 : 1);   // idxsfc
    const bool mc = a.mask != nullptr;
    const bool cloudy = H.cloudy != 0, clr5 = H.clr5 != 0;
    const double w0 = cloudy ? (mc ? 0.0 : (double)H.zcf0) : 1.0, w1 = cloudy ? (mc ? 1.0 : (double)H.zcf1) : 0.0;
    const int nseg = (nlay + SW2_SEG - 1) / SW2_SEG;
    if (pass == 0 || cloudy) {
        const F2 zsolar = act ? F2{H.zsolar[g], H.zsolar[g + 1]} : f2(0.0f);
        const F2 ab = f2(ibd ? H.albbm[ibd - 1] : 0.5f * (H.albbm[0] + H.albbm[1]));
        const F2 ad = f2(ibd ? H.albdf[ibd - 1] : 0.5f * (H.albdf[0] + H.albdf[1]));
        float2* ck = ckpt + tid;
        auto save = [&](int sg, int q, F2 v) { ck[((sg - 1) * 2 + q) * SW4_SWEEP_THREADS] = make_float2(v.x, v.y); };
        auto saved = [&](int sg, int q) { const float2 v = ck[((sg - 1) * 2 + q) * SW4_SWEEP_THREADS]; return F2{v.x, v.y}; };
        auto ld2 = [](const float* p) { const float2 v = __ldg(reinterpret_cast<const float2*>(p)); return F2{v.x, v.y}; };
        // R/T of layer k0 in this warp's pass (transparent padding above the model top)
        auto load = [&](int k0, SwRT2& c) {
            if (k0 >= nlay) {
                c.rb = c.rd = f2(0.0f);
                c.tb = c.td = c.e3 = c.e4 = f2(1.0f);
                return;
            }
            const int sl = pass ? (int)H.slot[k0] : -1;
            const float* p = (sl >= 0 ? rto + (size_t)sl * SW4_LAYER : rtc + (size_t)k0 * SW4_LAYER) + g;
            c.rb = ld2(p); c.rd = ld2(p + SW_NGPT); c.tb = ld2(p + 2 * SW_NGPT); c.td = ld2(p + 3 * SW_NGPT);
            c.e3 = ld2(p + 4 * SW_NGPT);
            c.e4 = clr5 && sl < 0 ? c.e3 : ld2(p + 5 * SW_NGPT);
        };
        // The R/T rows of segment sg into L2 ahead of its loads (one bulk prefetch per pass by its first thread): the
        // clear rows of its layers, the cloudy rows of their slots, each a contiguous run inside the column's block.
        auto prefetch = [&](int sg) {
            if (!SW4_L2PF || (tid & 63) != 0 || sg < 0 || sg >= nseg) return;
            const int k0 = sg * SW2_SEG, k1 = min(nlay, k0 + SW2_SEG);
            if (pass == 0) {
                l2_prefetch(rtc + (size_t)k0 * SW4_LAYER, (uint32_t)((k1 - k0) * SW4_LAYER * sizeof(float)));
                return;
            }
            int s0 = -1, s1 = -1;
            for (int k = k0; k < k1; ++k)
                if (H.slot[k] >= 0) { if (s0 < 0) s0 = H.slot[k]; s1 = H.slot[k]; }
            if (s0 >= 0) l2_prefetch(rto + (size_t)s0 * SW4_LAYER, (uint32_t)((s1 - s0 + 1) * SW4_LAYER * sizeof(float)));
        };
        // ---- upward sweep: reflectances of the atmosphere below each level
        F2 ub = ab, ud = ad;
        prefetch(0);
        prefetch(1);
        for (int sg = 0; sg < nseg; ++sg) {
            prefetch(sg + 2);
            if (sg > 0) { save(sg, 0, ub); save(sg, 1, ud); }
            SwRT2 L[SW2_SEG];
#pragma unroll
            for (int j = 0; j < SW2_SEG; ++j) load(sg * SW2_SEG + j, L[j]);
#pragma unroll
            for (int j = 0; j < SW2_SEG; ++j) sw4_up(L[j], ub, ud);
        }
        // ---- downward sweep, segment by segment from the top: the segment's R/T again, its upward states from the
        // checkpoint, then the walk down through it
        const double wp = pass ? w1 : w0, zx = wp * (double)zsolar.x, zy = wp * (double)zsolar.y;   // 0 in idle lanes
        auto net = [&](F2 fu, F2 fd) { return zx * ((double)fd.x - (double)fu.x) + zy * ((double)fd.y - (double)fu.y); };
        F2 tdn = f2(1.0f), rdn = f2(0.0f), tdb = f2(1.0f), tdb0 = f2(1.0f), toa = f2(0.0f);
        prefetch(nseg - 2);
        for (int sg = nseg - 1; sg >= 0; --sg) {
            prefetch(sg - 2);
            SwRT2 L[SW2_SEG];
            F2 zub[SW2_SEG + 1], zud[SW2_SEG + 1];
            zub[0] = sg ? saved(sg, 0) : ab;
            zud[0] = sg ? saved(sg, 1) : ad;
#pragma unroll
            for (int j = 0; j < SW2_SEG; ++j) load(sg * SW2_SEG + j, L[j]);
            F2 e4 = f2(1.0f);
#pragma unroll
            for (int j = 0; j < SW2_SEG; ++j) {
                e4 = e4 * L[j].e4;
                zub[j + 1] = zub[j]; zud[j + 1] = zud[j];
                sw4_up(L[j], zub[j + 1], zud[j + 1]);
            }
            double nv[SW2_SEG];
#pragma unroll
            for (int j = SW2_SEG - 1; j >= 0; --j) {
                const int lev = sg * SW2_SEG + j + 1;    // level above layer j (0 = surface); past the top: not used
                F2 fu, fd;
                sw4_flux(zub[j + 1], zud[j + 1], tdn, rdn, tdb, fu, fd);
                if (lev == nlay) toa = fu;
                nv[j] = net(fu, fd);
                if (DIAG && act && lev <= nlay) sw4_pg_level(pg, lev, g, pass, zsolar, fu, fd);
                sw4_down(L[j], tdn, rdn, tdb);
            }
            static_assert(SW2_SEG == 4, "warp_sum4 takes a segment's four levels");
            const double v = warp_sum4(nv, lane);
            if ((lane & 7) == 0) fn[warp][sg * SW2_SEG + (lane >> 3) + 1] = v;
            tdb0 = tdb0 * e4;
        }
        // ---- surface level, the per-lane scalars (zero for idle lanes)
        double o[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) o[q] = 0;
        F2 fu, fd;
        sw4_flux(ab, ad, tdn, rdn, tdb, fu, fd);
        const double v = warp_sum(net(fu, fd));
        if (lane == 0) fn[warp][0] = v;
        if (DIAG && act) sw4_pg_level(pg, 0, g, pass, zsolar, fu, fd);
        if (act) {
            // slots: 0 toa up, 1 sfc up, 2 sfc dn, 3 uv-b, 4 nir beam, 5 nir diffuse, 6 vis beam, 7 vis diffuse, 8 toa down
            auto fill = [&](float z, float tu, float su, float sd, float sdir) {
                const double zs = (double)z;
                o[0] += zs * (double)tu;
                o[1] += zs * (double)su;
                o[2] += zs * (double)sd;
                o[3] += ib0 == 11 ? zs * (double)sd : 0.0;
                const double zb1 = (double)(z * sdir), zb2 = (double)(z * (sd - sdir));
                if (ibd == 1) { o[4] += zb1; o[5] += zb2; }
                else if (ibd == 2) { o[6] += zb1; o[7] += zb2; }
                else { o[4] += 0.5 * zb1; o[5] += 0.5 * zb2; o[6] += 0.5 * zb1; o[7] += 0.5 * zb2; }
                o[8] += zs;
            };
            fill(zsolar.x, toa.x, fu.x, fd.x, tdb0.x);
            fill(zsolar.y, toa.y, fu.y, fd.y, tdb0.y);
        }
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const double t = warp_sum(o[q]);
            if (lane == 0) scs[warp][q] = t;
        }
    }
    __syncthreads();
    // ---- column end and swrad_post
    auto tot = [&](double clr, double cld) { return cloudy ? w1 * cld + w0 * clr : clr; };
    for (int k = tid; k < nlay; k += SW4_SWEEP_THREADS) {
        double f0 = fn[0][k] + fn[1][k], f1 = fn[0][k + 1] + fn[1][k + 1];
        if (cloudy) { f0 += fn[2][k] + fn[3][k]; f1 += fn[2][k + 1] + fn[3][k + 1]; }
        a.htsw[(size_t)(nlay - 1 - k) * N + col] = (float)((f1 - f0) * H.rdelp[k]);
    }
    if (tid == 0) {
        double c[9], t[9];
        for (int q = 0; q < 9; ++q) {
            c[q] = scs[0][q] + scs[1][q];
            t[q] = cloudy ? scs[2][q] + scs[3][q] : 0.0;
        }
        a.topfsw[col] = (float)tot(c[0], t[0]);
        a.topfsw[N + col] = (float)c[8];
        a.topfsw[2 * N + col] = (float)c[0];
        a.sfcfsw[col] = (float)tot(c[1], t[1]);
        a.sfcfsw[N + col] = (float)tot(c[2], t[2]);
        a.sfcfsw[2 * N + col] = (float)c[1];
        a.sfcfsw[3 * N + col] = (float)c[2];
        if (a.fdncmp) {
            a.fdncmp[col] = (float)c[3];
            a.fdncmp[N + col] = (float)tot(c[3], t[3]);
            a.fdncmp[2 * N + col] = (float)tot(c[4], t[4]);
            a.fdncmp[3 * N + col] = (float)tot(c[5], t[5]);
            a.fdncmp[4 * N + col] = (float)tot(c[6], t[6]);
            a.fdncmp[5 * N + col] = (float)tot(c[7], t[7]);
        }
    }
}

// swrad's optional outputs of a chunk from the DIAG sweeps' profiles (swrad_post's lhsw0 / lhswb / lflxprf blocks): one
// CTA per sunlit column, a warp per level, as k_lw_diag: lane q of each half warp sums band q of one field at a time in
// float64.  htswb from the band's net fluxes, hsw0 from the clear net fluxes, heating (F(k + 1) - F(k)) heatfac / delp as
// the sweeps form htsw, swflxprf the level fluxes.  2.4 -> 0.24 ms per 7,632 columns.
constexpr int SW4_DIAG_WARPS = 4;
__global__ void __launch_bounds__(SW4_DIAG_WARPS * 32) k_sw_diag(const __grid_constant__ SwBatch bt, int d0, const unsigned char* scr,
                                                                 size_t blk_bytes, const float* __restrict__ pg,
                                                                 const __grid_constant__ DiagOuts outs)
{
    constexpr int ROW = SW4_PGQ * SW_NGPT;
    __shared__ __align__(16) float sm[SW4_DIAG_WARPS][ROW];
    __shared__ double net[NLAY_MAX + 1][15];           // net flux of each band (total sky) and of the clear pass per level
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 15, half = lane >> 4;
    const int d = d0 + (int)blockIdx.x;
    if (d >= *bt.req[0].nday) return;
    const int64_t gcol = bt.req[0].daycol[d];
    const int rq = bt.find(gcol);
    const SwIn& a = bt.req[rq];
    const int nlay = a.nlay, nlp1 = nlay + 1;
    if (nlay > NLAY_MAX) return;
    const int64_t col = gcol - bt.off[rq], N = a.ncol;
    const Sw4Hdr& H = *reinterpret_cast<const Sw4Hdr*>(scr + (size_t)blockIdx.x * blk_bytes);
    const float4* p = reinterpret_cast<const float4*>(pg + (int64_t)blockIdx.x * sw4_pg_floats(nlay));
    float* hsw0 = outs.p[rq][3];
    float* htswb = outs.p[rq][4];
    float* flx = outs.p[rq][5];
    const bool cloudy = H.cloudy != 0, mc = a.mask != nullptr;
    const double w0 = cloudy ? (mc ? 0.0 : (double)H.zcf0) : 1.0, w1 = cloudy ? (mc ? 1.0 : (double)H.zcf1) : 0.0;
    const int g0 = q < 14 ? c_sw_ns[q] : 0, g1 = q < 14 ? c_sw_ns[q + 1] : 0;
    const int rows = cloudy ? ROW : ROW / 2;           // the cloudy pass's fields are written for a cloudy column only
    float* w = sm[warp];
    for (int L = warp; L < nlp1; L += SW4_DIAG_WARPS) {
        __syncwarp();                                  // the previous level's sums have been read
        for (int i = lane; i < rows / 4; i += 32) reinterpret_cast<float4*>(w)[i] = __ldg(p + (size_t)L * (ROW / 4) + i);
        __syncwarp();
        double v[3], t[3];                             // band q of field 2 i + half, and the field's total
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int f = 2 * i + half;
            double x = 0.0;
            if (f < 3 || cloudy)
                for (int g = g0; g < g1; ++g) x += (double)w[f * SW_NGPT + g];
            v[i] = x;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            t[i] = x;
        }
        // fields 0 .. 5 of the lane's band / in total: 0 = (half 0, i 0), 1 = (1, 0), 2 = (0, 1), 3 = (1, 1), 4 = (0, 2), 5 = (1, 2)
        const double v5 = __shfl_xor_sync(0xffffffffu, v[2], 16);              // half 0: the band's field 5
        const double t1 = __shfl_xor_sync(0xffffffffu, t[0], 16), t3 = __shfl_xor_sync(0xffffffffu, t[1], 16);
        if (half == 0) {
            if (q < 14) net[L][q] = cloudy ? w0 * v[1] + w1 * v5 : v[1];
            if (q == 0) {
                net[L][14] = t[1];
                if (flx) {
                    const int k = nlp1 - 1 - L;
                    flx[(size_t)k * N + col] = (float)(cloudy ? w0 * t[0] + w1 * t3 : t[0]);
                    flx[((size_t)nlp1 + k) * N + col] = (float)(cloudy ? w0 * t1 + w1 * t[2] : t1);
                    flx[((size_t)2 * nlp1 + k) * N + col] = (float)t[0];
                    flx[((size_t)3 * nlp1 + k) * N + col] = (float)t1;
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 15 * nlay; i += SW4_DIAG_WARPS * 32) {
        const int b = i / nlay, k0 = i - b * nlay;
        const float h = (float)((net[k0 + 1][b] - net[k0][b]) * H.rdelp[k0]);
        const size_t k = (size_t)(nlay - 1 - k0);
        if (b < 14) {
            if (htswb) htswb[((size_t)b * nlay + k) * N + col] = h;
        } else if (hsw0) {
            hsw0[k * N + col] = h;
        }
    }
}

}  // namespace rad
