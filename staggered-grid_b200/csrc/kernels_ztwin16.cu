// kernels_ztwin16.cu — z-marching velocity and stress updates of 16-bit
// wavefield storage (BF16 / F16, 32 x 8 tiles): planes are taken two at a
// time.
//
// Work decomposition.  A CTA of 256 threads owns a 32 x 8 tile of computed
// cells and marches along z over a chunk of planes; warp w is tile row w,
// lane l its column, and an iteration updates the thread's cells of planes z
// and z + 1.
//
// What bounds it.  16-bit storage halves the bytes, so the updates are bound
// by the work per cell: the FP32 arithmetic on read-back values float(h) *
// 2^e.  Per iteration, TMA tiled loads (4-D maps, two planes per copy, no
// multicast) bring the 16-bit field boxes with their halos into one stage;
// one pass widens every staged value once, into an FP32 work buffer that
// interleaves the two planes, so that
//   * a tap of both planes is one 8-byte shared load straight into the
//     register pair of a packed FP32x2 operation (fma.rn.f32x2), one lane per
//     plane: half the loads and half the arithmetic instructions of one plane
//     at a time;
//   * the stage is free as soon as it is widened: the next pair's copies have
//     the whole stencil to land, and one stage is enough;
//   * with two work buffers there is one block barrier per two planes (after
//     the widening); it also frees the own-cell buffer, whose copies overlap
//     the stencil.
// The z taps sit in register queues of stored values, 11 deep and moved by two
// per iteration, fed from the staged lead planes by the threads that own them
// and read back per use: half the registers of FP32 queues, which spilled at
// the 80 registers of three CTAs per SM (velocity, 266^3 with a 20-cell border:
// 0.532 ms per launch with FP32 queues, 0.493 like this).
// Measured, 50 steps: 394^3 FP16 167.2 ms one plane at a time (three-stage
// ring, one widening and two barriers per plane), 140.0 ms like this; 522^3
// BF16 356.9 to 299.0 ms.  Every packed
// lane rounds as the scalar operation does: results are bit-identical to
// kernels_half.cu, kernels_zpair.cu and the oracle's emulation.
//
// PML cells take the split-field path (cell_math.cuh) plane by plane from the
// same differences; the stress update brings their split rows into L2 one
// plane ahead.  Source injection, receivers and the scale updates run as the
// 16-bit family's own kernels (half_phase); on rescale steps the largest
// written magnitudes are reduced in shared memory and added to the global
// ones once per CTA.
#include <cuda.h>

#include <type_traits>

#include "cell_math.cuh"
#include "store16.cuh"
#include "zmarch.h"
#include "zmarch_dev.cuh"

namespace sgfd {

namespace {

using namespace zdev;

constexpr int TX = kZTileX, TY = 8, NT = 256;
constexpr int W48 = 48, W32 = 32, W36 = 36;
// values of a box's plane
constexpr int N48 = W48 * TY, N48Y = W48 * (TY + 10), N32Y = W32 * (TY + 10), N32 = W32 * TY;

constexpr int al128(int b) { return (b + 127) / 128 * 128; }

// Velocity update, byte offsets: the 16-bit stage, the own-cell buffer (vx,
// vy, vz at 16 bits, FP32 buoyancy of planes z, z+1, z+2) and one work buffer
// (float2 per staged value: planes z and z+1).
struct VelH {
    static constexpr int SXX = 0;                        // 48 x TY, 2 planes: sigma_xx, then sigma_xz
    static constexpr int SYY = SXX + 2 * 2 * N48 * 2;    // 32 x (TY+10): sigma_yy, then sigma_yz
    static constexpr int SXY = SYY + 2 * 2 * N32Y * 2;   // 48 x (TY+10): sigma_xy
    static constexpr int LXZ = SXY + 2 * N48Y * 2;       // 32 x TY: sigma_xz, sigma_yz at z+4, z+5
    static constexpr int LZZ = LXZ + 2 * 2 * N32 * 2;    // 32 x TY: sigma_zz at z+5, z+6
    static constexpr int STAGE = LZZ + 2 * N32 * 2;
    static constexpr uint32_t TXB = STAGE;
    static constexpr int OV = 0;                         // 3 x 2 x 32 x TY
    static constexpr int B = OV + 3 * 2 * N32 * 2;       // 36 x (TY+1) x 3 FP32
    static constexpr int OWN = B + al128(3 * W36 * (TY + 1) * 4);
    static constexpr uint32_t OTXB = 3 * 2 * N32 * 2 + 3 * W36 * (TY + 1) * 4;
    // work buffer, float2 units
    static constexpr int wXX = 0, wXZ = wXX + N48, wYY = wXZ + N48, wYZ = wYY + N32Y, wXY = wYZ + N32Y,
                         WORK = wXY + N48Y;
};
// Stress update: stage (vx, vy, vz and their lead planes), own-cell buffer
// (the six stresses at 16 bits, the FP32 medium), work buffer.
struct StrH {
    static constexpr int V = 0;                          // 48 x (TY+10), 2 planes: vx, vy, vz
    static constexpr int LX = V + 3 * 2 * N48Y * 2;      // 32 x TY: vx, vy at z+5, z+6
    static constexpr int LZ = LX + 2 * 2 * N32 * 2;      // 32 x TY: vz at z+4, z+5
    static constexpr int STAGE = LZ + 2 * N32 * 2;
    static constexpr uint32_t TXB = STAGE;
    static constexpr int SG = 0;                         // 6 x 2 x 32 x TY
    static constexpr int MED = SG + 6 * 2 * N32 * 2;     // 5 x 2 x 32 x TY FP32: lambda, mu, three shear moduli
    static constexpr int OWN = MED + 5 * 2 * N32 * 4;
    static constexpr uint32_t OTXB = OWN;
    static constexpr int WORK = 3 * N48Y;
};
static_assert(VelH::SYY % 128 == 0 && VelH::SXY % 128 == 0 && VelH::LXZ % 128 == 0 && VelH::LZZ % 128 == 0 &&
                  VelH::STAGE % 128 == 0 && VelH::B % 128 == 0 && StrH::LX % 128 == 0 && StrH::LZ % 128 == 0 &&
                  StrH::STAGE % 128 == 0 && StrH::MED % 128 == 0,
              "boxes start on 128-byte boundaries");
template <class L>
constexpr int smem_bytes() { return L::STAGE + L::OWN + 2 * 8 * L::WORK + 128; }
static_assert(3 * (smem_bytes<VelH>() + 1024 + 256) <= 228 * 1024 && 3 * (smem_bytes<StrH>() + 1024 + 256) <= 228 * 1024,
              "three CTAs per SM");

// A CTA's barriers (stage, own-cell buffer), its step's scales 2^e and 2^-e,
// and its largest written magnitudes on rescale steps.
struct Shared16 {
    uint64_t full, own;
    float scl[18];
    unsigned smax[9];
};
__device__ __forceinline__ void init16(Shared16 &y, const HalfState &hs) {
    if (threadIdx.x == 0) {
        mbar_init(&y.full, 1);
        mbar_init(&y.own, 1);
        fence_barrier_init();
    }
    step_wait();
    if (threadIdx.x < 9) {
        y.scl[threadIdx.x] = hs.sc[threadIdx.x];
        y.scl[9 + threadIdx.x] = hs.inv[threadIdx.x];
        y.smax[threadIdx.x] = 0u;
    }
    __syncthreads();
}

struct Tile16 {
    int cx0, cy0, xd, gx0, gy0;   // computed origin; device x; GRID origin
    int zs, ze;                   // computed z range of this CTA
};
__device__ __forceinline__ Tile16 make_tile(const Model &m, const ZGeom &g) {
    Tile16 t;
    const int tile = blockIdx.x, chunk = blockIdx.y + g.c0;
    t.cx0 = (tile % g.ntx) * TX;
    t.cy0 = (tile / g.ntx) * TY;
    t.gx0 = t.cx0 + kHalo;
    t.gy0 = t.cy0 + kHalo;
    t.xd = t.gx0 + kXOff;
    t.zs = chunk * g.zc;
    t.ze = min(t.zs + g.zc, m.nzc);
    return t;
}

__device__ __forceinline__ void vel_stage(const ZTwin16Maps &mp, const Tile16 &t, unsigned char *st, uint64_t *bar,
                                          int cz) {
    const int z = cz + kHalo;
    mbar_expect_tx(bar, VelH::TXB);
    tma4(st + VelH::SXX, &mp.v_sxx_sxz, t.xd - 8, t.gy0, z, 0, bar);
    tma4(st + VelH::SYY, &mp.v_syy_syz, t.xd, t.gy0 - 5, z, 0, bar);
    tma4(st + VelH::SXY, &mp.v_sxy, t.xd - 8, t.gy0 - 5, z, 0, bar);
    tma4(st + VelH::LXZ, &mp.v_lead_xz_yz, t.xd, t.gy0, z + 4, 0, bar);
    tma4(st + VelH::LZZ, &mp.v_lead_zz, t.xd, t.gy0, z + 5, 0, bar);
}
__device__ __forceinline__ void vel_own(const ZTwin16Maps &mp, const Tile16 &t, unsigned char *ob, uint64_t *bar,
                                        int cz) {
    const int z = cz + kHalo;
    mbar_expect_tx(bar, VelH::OTXB);
    tma4(ob + VelH::OV, &mp.v_own, t.xd, t.gy0, z, 0, bar);
    tma4(ob + VelH::B, &mp.v_b, t.xd, t.gy0, z, 0, bar);
}
__device__ __forceinline__ void str_stage(const ZTwin16Maps &mp, const Tile16 &t, unsigned char *st, uint64_t *bar,
                                          int cz) {
    const int z = cz + kHalo;
    mbar_expect_tx(bar, StrH::TXB);
    tma4(st + StrH::V, &mp.s_v, t.xd - 8, t.gy0 - 5, z, 0, bar);
    tma4(st + StrH::LX, &mp.s_lead_xy, t.xd, t.gy0, z + 5, 0, bar);
    tma4(st + StrH::LZ, &mp.s_lead_z, t.xd, t.gy0, z + 4, 0, bar);
}
__device__ __forceinline__ void str_own(const ZTwin16Maps &mp, const Tile16 &t, unsigned char *ob, uint64_t *bar,
                                        int cz) {
    const int z = cz + kHalo;
    mbar_expect_tx(bar, StrH::OTXB);
    tma4(ob + StrH::SG, &mp.s_own, t.xd, t.gy0, z, 0, bar);
    tma4(ob + StrH::MED, &mp.s_med, t.xd, t.gy0, z, 0, bar);
}

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
template <int K>
__device__ __forceinline__ float half_of(float2 v) { return K == 0 ? v.x : v.y; }

// Widen one field's box of N values per plane (two planes, N values apart)
// into dst: pairs (plane z, plane z+1) of float(h) * sc.
template <int ST, int N>
__device__ __forceinline__ void widen2(const unsigned char *src, float2 *dst, float sc) {
    static_assert(N % 2 == 0, "two values per word");
    const uint32_t *s = reinterpret_cast<const uint32_t *>(src);
    float4 *d = reinterpret_cast<float4 *>(dst);
#pragma unroll
    for (int i = threadIdx.x; i < N / 2; i += NT) {
        const uint32_t a = s[i], b = s[i + N / 2];
        const float2 lo = __fmul2_rn(make_float2(H16<ST>::h2f(a & 0xffffu), H16<ST>::h2f(b & 0xffffu)), both(sc));
        const float2 hi = __fmul2_rn(make_float2(H16<ST>::h2f(a >> 16), H16<ST>::h2f(b >> 16)), both(sc));
        d[i] = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
}
// Own values of both planes (N32 apart).
template <int ST>
__device__ __forceinline__ float2 own2(const uint16_t *p, float sc) {
    return __fmul2_rn(make_float2(H16<ST>::h2f(p[0]), H16<ST>::h2f(p[N32])), both(sc));
}

// Differences of both planes from pairs p[o * STRIDE]: forward sum c_i
// (p(1+i) - p(-i)), backward sum c_i (p(i) - p(-1-i)).
template <int STRIDE>
__device__ __forceinline__ float2 fwd2(const float2 (&c)[5], const float2 *p) {
    return dpair(c, [&](int i) { return p[(1 + i) * STRIDE]; }, [&](int i) { return p[-i * STRIDE]; });
}
template <int STRIDE>
__device__ __forceinline__ float2 bwd2(const float2 (&c)[5], const float2 *p) {
    return dpair(c, [&](int i) { return p[i * STRIDE]; }, [&](int i) { return p[(-1 - i) * STRIDE]; });
}
// z differences of plane K of the pair from the queues (taps q[5+i], q[4-i]
// of the plane's 10 values).
template <int K>
__device__ __forceinline__ float2 zdiff2(const float2 (&c)[5], const float2 (&q)[11]) {
    return dpair(c, [&](int i) { return q[K + 5 + i]; }, [&](int i) { return q[K + 4 - i]; });
}
template <int K>
__device__ __forceinline__ float zdiff(const float (&c)[5], const float (&q)[11]) {
    float d = 0.0f;
#pragma unroll
    for (int i = 0; i < 5; ++i) d = __fmaf_rn(c[i], q[K + 5 + i] - q[K + 4 - i], d);
    return d;
}
template <bool FAST>
__device__ __forceinline__ float2 by_cell2(const Physics &ph, int axis, float2 s) {
    return make_float2(by_cell<FAST>(ph, axis, s.x), by_cell<FAST>(ph, axis, s.y));
}

// The thread's column.
struct Col16 {
    int kx, ky;           // x and y PML band distances
    bool act, xy_pml;     // inside the computed region; the warp's columns touch the x or y band
    uint32_t col;         // element offset at z = 0 (inactive threads: a valid cell's, results discarded)
    PmlColumn pcol;
};
__device__ __forceinline__ Col16 make_col(const Model &m, const Tile16 &t, int lx, int warp) {
    Col16 c;
    const int gx = t.gx0 + lx, gy = t.gy0 + warp;
    c.kx = band(gx, m.nx, m.pml);
    c.ky = band(gy, m.ny, m.pml);
    c.act = t.cx0 + lx < m.nxc && t.cy0 + warp < m.nyc;
    c.xy_pml = __any_sync(0xffffffffu, c.act && (c.kx | c.ky));
    c.col = (uint32_t)pidx(m, min(gx, m.nx - 1), min(gy, m.ny - 1), 0);
    c.pcol = pml_column(m, min(t.cx0 + lx, m.nxc - 1), min(t.cy0 + warp, m.nyc - 1));
    return c;
}

// Damping factors of one PML cell (wave speed v).
template <bool FAST>
struct Damp {
    float mx = 1.f, my = 1.f, mz = 1.f;
    PDiv<FAST> px = 1, py = 1, pz = 1;
    __device__ __forceinline__ Damp(const Physics &ph, int pml, int kx, int ky, int kz, float v) {
        if (kx) damp_factors<FAST>(ph, 0, ph.dx, kx, pml, v, mx, px);
        if (ky) damp_factors<FAST>(ph, 1, ph.dy, ky, pml, v, my, py);
        if (kz) damp_factors<FAST>(ph, 2, ph.dz, kz, pml, v, mz, pz);
    }
};

// After a failed wait, thread 0: the error flag and (bounded) the copies in
// flight.  ns, no: copies issued to the stage and to the own-cell buffer.
__device__ __noinline__ void give_up(Shared16 &y, int *err, int ns, int no) {
    atomicExch(err, 1);
    mbar_wait(&y.full, (uint32_t)(ns - 1) & 1u);
    if (no > 0) mbar_wait(&y.own, (uint32_t)(no - 1) & 1u);
}

template <bool FAST, int ST>
__global__ void __launch_bounds__(NT, 3)
k_velocity_ztwin16(const __grid_constant__ ZTwin16Maps mp, const __grid_constant__ Model m,
                   const __grid_constant__ Physics ph, const __grid_constant__ ZGeom g,
                   const __grid_constant__ SourceRec sr, const __grid_constant__ HalfState hs, int it_arg) {
    using L = VelH;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) Shared16 y;
    unsigned char *st = align_smem(smem_raw), *ob = st + L::STAGE;
    float2 *work0 = reinterpret_cast<float2 *>(ob + L::OWN);
    const Tile16 t = make_tile(m, g);
    const int tid = threadIdx.x, lx = tid & 31, warp = tid >> 5;
    init16(y, hs);
    if (tid == 0) vel_stage(mp, t, st, &y.full, t.zs);
    const bool track = rescale_step16(step_index(sr, it_arg));   // note the written maxima
    const Col16 c = make_col(m, t, lx, warp);
    const uint32_t PL = (uint32_t)m.plane;
    const int gz0 = t.zs + kHalo, pairs = (t.ze - t.zs + 1) / 2;
    auto h2f = [&](uint32_t h, int f) { return H16<ST>::h2f(h) * y.scl[f]; };
    auto put = [&](uint16_t *p, int f, float v) { *p = (uint16_t)H16<ST>::f2h(v * y.scl[9 + f]); };

    // z queues: at the start of an iteration at z, sigma_xz and sigma_yz hold
    // z-5..z+3, sigma_zz z-4..z+4 in slots 0..8
    uint32_t qxy[11], qz[11];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const uint32_t o = c.col + (uint32_t)(gz0 - 5 + k) * PL;
        qxy[k] = hs.f[7][o] | (uint32_t)hs.f[8][o] << 16;
        qz[k] = hs.f[5][o + PL];
    }
    const float2 (&cX)[5] = FAST ? ph.cp[0] : ph.cr;
    const float2 (&cY)[5] = FAST ? ph.cp[1] : ph.cr;
    const float2 (&cZ)[5] = FAST ? ph.cp[2] : ph.cr;
    const float (&cz1)[5] = FAST ? ph.cs[2] : ph.c;

    bool failed = false, abort = false;
    int cz = t.zs;
    for (int i = 0; i < pairs; ++i, cz += 2) {
        const int gz = cz + kHalo;
        const bool gen = c.xy_pml || bandz(m, gz) != 0 || bandz(m, gz + 1) != 0;
        // PML cells: splits and damping speed of plane K (stored values)
        uint32_t o[2][9];
        float vd[2];
        auto load = [&](auto k_tag) {
            constexpr int K = decltype(k_tag)::value;
            if (c.act && (c.kx | c.ky | bandz(m, gz + K)) && cz + K < t.ze) {
                const uint32_t pi = pml_plane_index(m, c.pcol, cz + K);
                const uint16_t *sp = hs.split + split_base32(pi);
#pragma unroll
                for (int q = 0; q < 9; ++q) o[K][q] = sp[q * kSplitBlock];
                vd[K] = m.vd[pi];
            }
        };
        if (gen) load(std::integral_constant<int, 0>{});   // ahead of the wait, whose time they overlap

        if (!mbar_wait(&y.full, (uint32_t)i & 1u)) failed = true;
        {
            const uint16_t *l = reinterpret_cast<const uint16_t *>(st + L::LXZ) + tid;
            const uint16_t *lz = reinterpret_cast<const uint16_t *>(st + L::LZZ) + tid;
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                qxy[9 + p] = l[p * N32] | (uint32_t)l[(2 + p) * N32] << 16;
                qz[9 + p] = lz[p * N32];
            }
        }
        float2 *wk = work0 + (i & 1) * L::WORK;
        widen2<ST, N48>(st + L::SXX, wk + L::wXX, y.scl[3]);
        widen2<ST, N48>(st + L::SXX + 4 * N48, wk + L::wXZ, y.scl[7]);
        widen2<ST, N32Y>(st + L::SYY, wk + L::wYY, y.scl[4]);
        widen2<ST, N32Y>(st + L::SYY + 4 * N32Y, wk + L::wYZ, y.scl[8]);
        widen2<ST, N48Y>(st + L::SXY, wk + L::wXY, y.scl[6]);
        // the pair is widened, and every thread is done with the pair before it
        if (__syncthreads_or(failed)) {
            if (tid == 0) give_up(y, g.err, i + 1, i);
            abort = true;
            break;
        }
        if (tid == 0) {
            fence_proxy_async();
            if (i + 1 < pairs) vel_stage(mp, t, st, &y.full, cz + 2);
            vel_own(mp, t, ob, &y.own, cz);
        }

        const float2 *w48 = wk + warp * W48 + lx + 8, *w32 = wk + warp * W32 + lx;
        const float2 xX = by_cell2<FAST>(ph, 0, fwd2<1>(cX, w48 + L::wXX));
        const float2 xY = by_cell2<FAST>(ph, 1, bwd2<W48>(cY, w48 + L::wXY + 5 * W48));
        const float2 yX = by_cell2<FAST>(ph, 0, bwd2<1>(cX, w48 + L::wXY + 5 * W48));
        const float2 yY = by_cell2<FAST>(ph, 1, fwd2<W32>(cY, w32 + L::wYY + 5 * W32));
        const float2 zX = by_cell2<FAST>(ph, 0, bwd2<1>(cX, w48 + L::wXZ));
        const float2 zY = by_cell2<FAST>(ph, 1, bwd2<W32>(cY, w32 + L::wYZ + 5 * W32));
        float2 a, b, zZ;
        {
            float2 w[11];
            float wz[11];
#pragma unroll
            for (int k = 0; k < 11; ++k) {
                w[k] = __fmul2_rn(make_float2(H16<ST>::h2f(qxy[k] & 0xffffu), H16<ST>::h2f(qxy[k] >> 16)),
                                  make_float2(y.scl[7], y.scl[8]));
                wz[k] = H16<ST>::h2f(qz[k]) * y.scl[5];
            }
            a = by_cell2<FAST>(ph, 2, zdiff2<0>(cZ, w));
            b = by_cell2<FAST>(ph, 2, zdiff2<1>(cZ, w));
            zZ = by_cell2<FAST>(ph, 2, make_float2(zdiff<0>(cz1, wz), zdiff<1>(cz1, wz)));
        }
        const float2 xZ = make_float2(a.x, b.x), yZ = make_float2(a.y, b.y);
        if (gen) load(std::integral_constant<int, 1>{});

        if (!mbar_wait(&y.own, (uint32_t)i & 1u)) failed = true;
        const uint16_t *ov = reinterpret_cast<const uint16_t *>(ob + L::OV) + tid;
        const float *pb = reinterpret_cast<const float *>(ob + L::B) + warp * W36 + lx;
        constexpr int PB = W36 * (TY + 1);
        const float2 b0 = make_float2(pb[0], pb[PB]);
        const float2 bx = __fmul2_rn(__fadd2_rn(b0, make_float2(pb[1], pb[PB + 1])), both(0.5f));
        const float2 by = __fmul2_rn(__fadd2_rn(b0, make_float2(pb[W36], pb[PB + W36])), both(0.5f));
        const float2 bz = __fmul2_rn(__fadd2_rn(b0, make_float2(pb[PB], pb[2 * PB])), both(0.5f));
        const float2 dt2 = both(ph.dt);
        const float2 ax = __fmul2_rn(dt2, bx), ay = __fmul2_rn(dt2, by), az = __fmul2_rn(dt2, bz);
        const uint32_t ci = c.col + (uint32_t)gz * PL;
        const float2 v0 = __ffma2_rn(ax, __fadd2_rn(__fadd2_rn(xX, xY), xZ), own2<ST>(ov, y.scl[0]));
        const float2 v1 = __ffma2_rn(ay, __fadd2_rn(__fadd2_rn(yX, yY), yZ), own2<ST>(ov + 2 * N32, y.scl[1]));
        const float2 v2 = __ffma2_rn(az, __fadd2_rn(__fadd2_rn(zX, zY), zZ), own2<ST>(ov + 4 * N32, y.scl[2]));
        // one plane's cell: through the splits in the PML
        auto cell = [&](auto k_tag) {
            constexpr int K = decltype(k_tag)::value;
            if (!c.act || cz + K >= t.ze) return;
            float v[3] = {half_of<K>(v0), half_of<K>(v1), half_of<K>(v2)};
            if (gen) {
                const int kz = bandz(m, gz + K);
                if (c.kx | c.ky | kz) {
                    const Damp<FAST> d(ph, m.pml, c.kx, c.ky, kz, vd[K]);
                    const bool ref = ph.quirks == 0;
                    const float r[3] = {half_of<K>(ax), half_of<K>(ref ? ax : ay), half_of<K>(ref ? ax : az)};
                    const float df[3][3] = {{half_of<K>(xX), half_of<K>(xY), half_of<K>(xZ)},
                                            {half_of<K>(yX), half_of<K>(yY), half_of<K>(yZ)},
                                            {half_of<K>(zX), half_of<K>(zY), half_of<K>(zZ)}};
                    uint16_t *sp = hs.split + split_base32(pml_plane_index(m, c.pcol, cz + K));
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        float s[3];
                        s[0] = split_update<FAST>(h2f(o[K][3 * q], q), r[q], df[q][0], c.kx, d.mx, d.px);
                        s[1] = split_update<FAST>(h2f(o[K][3 * q + 1], q), r[q], df[q][1], c.ky, d.my, d.py);
                        s[2] = split_update<FAST>(h2f(o[K][3 * q + 2], q), r[q], df[q][2], kz, d.mz, d.pz);
#pragma unroll
                        for (int e = 0; e < 3; ++e) {
                            if (track) note_max16s(y.smax, q, s[e]);
                            put(sp + (3 * q + e) * kSplitBlock, q, s[e]);
                        }
                        v[q] = (s[0] + s[1]) + s[2];
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                if (track) note_max16s(y.smax, q, v[q]);
                put(hs.f[q] + ci + K * PL, q, v[q]);
            }
        };
        cell(std::integral_constant<int, 0>{});
        cell(std::integral_constant<int, 1>{});
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            qxy[j] = qxy[j + 2];
            qz[j] = qz[j + 2];
        }
    }
    if (!abort && __syncthreads_or(failed) && tid == 0) give_up(y, g.err, pairs, pairs);
    if (track) {
        __syncthreads();
        flush_max16(hs, y.smax);
    }
}

template <bool FAST, int ST>
__global__ void __launch_bounds__(NT, 3)
k_stress_ztwin16(const __grid_constant__ ZTwin16Maps mp, const __grid_constant__ Model m,
                 const __grid_constant__ Physics ph, const __grid_constant__ ZGeom g,
                 const __grid_constant__ SourceRec sr, const __grid_constant__ HalfState hs, int it_arg) {
    using L = StrH;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) Shared16 y;
    unsigned char *st = align_smem(smem_raw), *ob = st + L::STAGE;
    float2 *work0 = reinterpret_cast<float2 *>(ob + L::OWN);
    const Tile16 t = make_tile(m, g);
    const int tid = threadIdx.x, lx = tid & 31, warp = tid >> 5;
    init16(y, hs);
    if (tid == 0) str_stage(mp, t, st, &y.full, t.zs);
    const bool track = rescale_step16(step_index(sr, it_arg));
    const Col16 c = make_col(m, t, lx, warp);
    const uint32_t PL = (uint32_t)m.plane;
    const int gz0 = t.zs + kHalo, pairs = (t.ze - t.zs + 1) / 2;
    auto h2f = [&](uint32_t h, int f) { return H16<ST>::h2f(h) * y.scl[f]; };
    auto put = [&](uint16_t *p, int f, float v) { *p = (uint16_t)H16<ST>::f2h(v * y.scl[9 + f]); };

    // z queues: vx and vy hold z-4..z+4, vz z-5..z+3 in slots 0..8
    uint32_t qxy[11], qz[11];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const uint32_t o = c.col + (uint32_t)(gz0 - 5 + k) * PL;
        qxy[k] = hs.f[0][o + PL] | (uint32_t)hs.f[1][o + PL] << 16;
        qz[k] = hs.f[2][o];
    }
    const float2 (&cX)[5] = FAST ? ph.cp[0] : ph.cr;
    const float2 (&cY)[5] = FAST ? ph.cp[1] : ph.cr;
    const float2 (&cZ)[5] = FAST ? ph.cp[2] : ph.cr;
    const float (&cz1)[5] = FAST ? ph.cs[2] : ph.c;

    // PML cells of plane pz: their split rows into L2 ahead of their loads
    auto prefetch = [&](int pz) {
        if (pz >= t.ze) return;
        const int kzp = bandz(m, pz + kHalo);
        if (!c.xy_pml && kzp == 0) return;
        prefetch_split_rows(hs.split, c.act && (c.kx | c.ky | kzp), pml_plane_index(m, c.pcol, pz), S_XXX, kNumSplit,
                            lx);
    };
    prefetch(t.zs);

    bool failed = false, abort = false;
    int cz = t.zs;
    for (int i = 0; i < pairs; ++i, cz += 2) {
        const int gz = cz + kHalo;
        const bool gen = c.xy_pml || bandz(m, gz) != 0 || bandz(m, gz + 1) != 0;
        prefetch(cz + 1);
        if (!mbar_wait(&y.full, (uint32_t)i & 1u)) failed = true;
        {
            const uint16_t *l = reinterpret_cast<const uint16_t *>(st + L::LX) + tid;
            const uint16_t *lz = reinterpret_cast<const uint16_t *>(st + L::LZ) + tid;
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                qxy[9 + p] = l[p * N32] | (uint32_t)l[(2 + p) * N32] << 16;
                qz[9 + p] = lz[p * N32];
            }
        }
        float2 *wk = work0 + (i & 1) * L::WORK;
#pragma unroll
        for (int f = 0; f < 3; ++f) widen2<ST, N48Y>(st + L::V + f * 4 * N48Y, wk + f * N48Y, y.scl[f]);
        if (__syncthreads_or(failed)) {
            if (tid == 0) give_up(y, g.err, i + 1, i);
            abort = true;
            break;
        }
        if (tid == 0) {
            fence_proxy_async();
            if (i + 1 < pairs) str_stage(mp, t, st, &y.full, cz + 2);
            str_own(mp, t, ob, &y.own, cz);
        }

        const float2 *vx = wk + (warp + 5) * W48 + lx + 8, *vy = vx + N48Y, *vz = vy + N48Y;
        const uint16_t *sg = reinterpret_cast<const uint16_t *>(ob + L::SG) + tid;
        const float *md = reinterpret_cast<const float *>(ob + L::MED) + tid;
        auto med = [&](int q) { return make_float2(md[2 * q * N32], md[(2 * q + 1) * N32]); };
        const uint32_t ci = c.col + (uint32_t)gz * PL;
        const bool second = cz + 1 < t.ze;
        auto dZ = [&]() {   // vz along z
            float w[11];
#pragma unroll
            for (int k = 0; k < 11; ++k) w[k] = h2f(qz[k], 2);
            return by_cell2<FAST>(ph, 2, make_float2(zdiff<0>(cz1, w), zdiff<1>(cz1, w)));
        };
        auto dZ2 = [&](float2 &a, float2 &b) {   // vx and vy along z, per plane
            float2 w[11];
#pragma unroll
            for (int k = 0; k < 11; ++k)
                w[k] = __fmul2_rn(make_float2(H16<ST>::h2f(qxy[k] & 0xffffu), H16<ST>::h2f(qxy[k] >> 16)),
                                  make_float2(y.scl[0], y.scl[1]));
            a = by_cell2<FAST>(ph, 2, zdiff2<0>(cZ, w));
            b = by_cell2<FAST>(ph, 2, zdiff2<1>(cZ, w));
        };
        if (!gen) {
            auto store = [&](int q, float2 v) {
                if (!c.act) return;
                uint16_t *p = hs.f[3 + q] + ci;
                if (track) note_max16s(y.smax, 3 + q, v, second);
                put(p, 3 + q, v.x);
                if (second) put(p + PL, 3 + q, v.y);
            };
            auto own = [&](int q) { return own2<ST>(sg + 2 * q * N32, y.scl[3 + q]); };
            const float2 dt2 = both(ph.dt);
            // shear stresses last: their differences wait for no copy
            float2 a, b;
            dZ2(a, b);
            const float2 sxy =
                __fadd2_rn(by_cell2<FAST>(ph, 1, fwd2<W48>(cY, vx)), by_cell2<FAST>(ph, 0, fwd2<1>(cX, vy)));
            const float2 sxz = __fadd2_rn(make_float2(a.x, b.x), by_cell2<FAST>(ph, 0, fwd2<1>(cX, vz)));
            const float2 syz = __fadd2_rn(make_float2(a.y, b.y), by_cell2<FAST>(ph, 1, fwd2<W48>(cY, vz)));
            const float2 dXx = by_cell2<FAST>(ph, 0, bwd2<1>(cX, vx)), dYy = by_cell2<FAST>(ph, 1, bwd2<W48>(cY, vy)),
                         dZz = dZ();
            if (!mbar_wait(&y.own, (uint32_t)i & 1u)) failed = true;
            const float2 l = med(0), l2m = __ffma2_rn(both(2.0f), med(1), l);
            store(0, __ffma2_rn(dt2, __ffma2_rn(l2m, dXx, __fmul2_rn(l, __fadd2_rn(dYy, dZz))), own(0)));
            store(1, __ffma2_rn(dt2, __ffma2_rn(l2m, dYy, __fmul2_rn(l, __fadd2_rn(dXx, dZz))), own(1)));
            store(2, __ffma2_rn(dt2, __ffma2_rn(l2m, dZz, __fmul2_rn(l, __fadd2_rn(dXx, dYy))), own(2)));
            store(3, __ffma2_rn(__fmul2_rn(dt2, med(2)), sxy, own(3)));
            store(4, __ffma2_rn(__fmul2_rn(dt2, med(3)), sxz, own(4)));
            store(5, __ffma2_rn(__fmul2_rn(dt2, med(4)), syz, own(5)));
        } else {
            float2 a, b;
            dZ2(a, b);
            const float2 xyY = by_cell2<FAST>(ph, 1, fwd2<W48>(cY, vx)), xyX = by_cell2<FAST>(ph, 0, fwd2<1>(cX, vy));
            const float2 xzX = by_cell2<FAST>(ph, 0, fwd2<1>(cX, vz)), yzY = by_cell2<FAST>(ph, 1, fwd2<W48>(cY, vz));
            const float2 dXx = by_cell2<FAST>(ph, 0, bwd2<1>(cX, vx)), dYy = by_cell2<FAST>(ph, 1, bwd2<W48>(cY, vy)),
                         dZz = dZ();
            prefetch(cz + 2);
            if (!mbar_wait(&y.own, (uint32_t)i & 1u)) failed = true;
            // one plane after the other, one body for both, as in the velocity update
#pragma unroll
            for (int K = 0; K < 2; ++K) {
                if (!c.act || cz + K >= t.ze) continue;
                auto at = [&](float2 v) { return K ? v.y : v.x; };
                const int kz = bandz(m, gz + K);
                const float xx = at(dXx), yy = at(dYy), zz = at(dZz), dt = ph.dt;
                const float *mk = md + K * N32;
                const float lk = mk[0], l2 = __fmaf_rn(2.0f, mk[2 * N32], lk);
                const float axy = dt * mk[4 * N32], axz = dt * mk[6 * N32], ayz = dt * mk[8 * N32];
                const float hyY = at(xyY), hyX = at(xyX), hzX = at(xzX), gzY = at(yzY);
                const float hzZ = K ? b.x : a.x, gzZ = K ? b.y : a.y;
                float sn[6];
                if (!(c.kx | c.ky | kz)) {
                    auto own = [&](int q) { return h2f(sg[(2 * q + K) * N32], 3 + q); };
                    sn[0] = __fmaf_rn(dt, __fmaf_rn(l2, xx, lk * (yy + zz)), own(0));
                    sn[1] = __fmaf_rn(dt, __fmaf_rn(l2, yy, lk * (xx + zz)), own(1));
                    sn[2] = __fmaf_rn(dt, __fmaf_rn(l2, zz, lk * (xx + yy)), own(2));
                    sn[3] = __fmaf_rn(axy, hyY + hyX, own(3));
                    sn[4] = __fmaf_rn(axz, hzZ + hzX, own(4));
                    sn[5] = __fmaf_rn(ayz, gzZ + gzY, own(5));
                } else {
                    const uint32_t pi = pml_plane_index(m, c.pcol, cz + K);
                    uint16_t *sp = hs.split + split_base32(pi);
                    constexpr uint32_t N = kSplitBlock;
                    uint32_t o[15];
#pragma unroll
                    for (int q = 0; q < 15; ++q) o[q] = sp[(S_XXX + q) * N];
                    const Damp<FAST> d(ph, m.pml, c.kx, c.ky, kz, m.vd[pi]);
                    auto sput = [&](int k, int f, float v) {
                        if (track) note_max16s(y.smax, f, v);
                        put(sp + (S_XXX + k) * N, f, v);
                    };
                    // part e of normal stress q has rate dt * l2m * d_e when e = q, dt * (l * d_e) otherwise
                    const float dl = dt * l2;
                    const float df[3] = {xx, yy, zz}, ld[3] = {lk * xx, lk * yy, lk * zz};
                    const float mm[3] = {d.mx, d.my, d.mz};
                    const PDiv<FAST> pp[3] = {d.px, d.py, d.pz};
                    const int kk[3] = {c.kx, c.ky, kz};
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        float s[3];
#pragma unroll
                        for (int e = 0; e < 3; ++e) {
                            s[e] = split_update<FAST>(h2f(o[3 * q + e], 3 + q), e == q ? dl : dt,
                                                      e == q ? df[e] : ld[e], kk[e], mm[e], pp[e]);
                            sput(3 * q + e, 3 + q, s[e]);
                        }
                        sn[q] = (s[0] + s[1]) + s[2];
                    }
                    float a0, a1;
                    a0 = split_update<FAST>(h2f(o[9], 6), axy, hyX, c.kx, d.mx, d.px);
                    a1 = split_update<FAST>(h2f(o[10], 6), axy, hyY, c.ky, d.my, d.py);
                    sput(9, 6, a0); sput(10, 6, a1);
                    sn[3] = a0 + a1;
                    a0 = split_update<FAST>(h2f(o[11], 7), axz, hzX, c.kx, d.mx, d.px);
                    a1 = split_update<FAST>(h2f(o[12], 7), axz, hzZ, kz, d.mz, d.pz);
                    sput(11, 7, a0); sput(12, 7, a1);
                    sn[4] = a0 + a1;
                    a0 = split_update<FAST>(h2f(o[13], 8), ayz, gzY, c.ky, d.my, d.py);
                    a1 = split_update<FAST>(h2f(o[14], 8), ayz, gzZ, kz, d.mz, d.pz);
                    sput(13, 8, a0); sput(14, 8, a1);
                    sn[5] = a0 + a1;
                }
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    if (track) note_max16s(y.smax, 3 + q, sn[q]);
                    put(hs.f[3 + q] + ci + K * PL, 3 + q, sn[q]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            qxy[j] = qxy[j + 2];
            qz[j] = qz[j + 2];
        }
    }
    if (!abort && __syncthreads_or(failed) && tid == 0) give_up(y, g.err, pairs, pairs);
    if (track) {
        __syncthreads();
        flush_max16(hs, y.smax);
    }
}

template <bool FAST, int ST>
cudaError_t set_attrs() {
    cudaError_t e = cudaFuncSetAttribute(k_velocity_ztwin16<FAST, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem_bytes<VelH>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_stress_ztwin16<FAST, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 smem_bytes<StrH>());
    return e;
}

// One step: the source injection before the velocity update, the velocity
// receivers after it, the stress receivers and the rescale after the stress
// update (kernels_half.cu, half_phase).
template <bool FAST, int ST>
void launch(const Model &m, const Physics &ph, const SourceRec &sr, const HalfState &hs, const ZGeom &g,
            const ZTwin16Maps &tm, int it, float src_value, bool uw, cudaStream_t s, cudaEvent_t *ev) {
    const dim3 grid(g.ntx * g.nty, g.nchunks);
    half_phase(m, ph, sr, hs, it, src_value, uw, s, 0);
    if (ev) cudaEventRecord(ev[0], s);
    step_launch(k_velocity_ztwin16<FAST, ST>, grid, NT, smem_bytes<VelH>(), s, sr.overlap != 0, tm, m, ph, g, sr, hs,
                it);
    if (ev) cudaEventRecord(ev[1], s);
    half_phase(m, ph, sr, hs, it, src_value, uw, s, 1);
    if (ev) cudaEventRecord(ev[2], s);
    step_launch(k_stress_ztwin16<FAST, ST>, grid, NT, smem_bytes<StrH>(), s, sr.overlap != 0, tm, m, ph, g, sr, hs, it);
    if (ev) cudaEventRecord(ev[3], s);
    half_phase(m, ph, sr, hs, it, src_value, uw, s, 2);
}

}  // namespace

cudaError_t ztwin16_prepare(const Model &m, size_t st, const HalfState &hs, size_t st16, ZTwin16Maps *tm) {
    // the orders the merged copies rely on: the nine stored wavefields evenly
    // spaced, and lambda, mu, mxy, mxz, myz
    for (int k = 0; k < 9; ++k)
        if (hs.f[k] != reinterpret_cast<const uint16_t *>(reinterpret_cast<const char *>(hs.f[0]) + k * st16))
            return cudaErrorInvalidValue;
    const float *med[5] = {m.lam, m.mu, m.mxy, m.mxz, m.myz};
    for (int k = 0; k < 5; ++k)
        if (med[k] != reinterpret_cast<const float *>(reinterpret_cast<const char *>(m.lam) + k * st))
            return cudaErrorInvalidValue;
    bool ok = true;
    ok &= make_pool_map16(&tm->v_sxx_sxz, hs.f[3], m, 4 * st16, 2, W48, TY, 2);
    ok &= make_pool_map16(&tm->v_syy_syz, hs.f[4], m, 4 * st16, 2, W32, TY + 10, 2);
    ok &= make_pool_map16(&tm->v_sxy, hs.f[6], m, st16, 1, W48, TY + 10, 2);
    ok &= make_pool_map16(&tm->v_lead_xz_yz, hs.f[7], m, st16, 2, W32, TY, 2);
    ok &= make_pool_map16(&tm->v_lead_zz, hs.f[5], m, st16, 1, W32, TY, 2);
    ok &= make_pool_map16(&tm->v_own, hs.f[0], m, st16, 3, W32, TY, 2);
    ok &= make_pool_map(&tm->v_b, m.b, m, st, 1, W36, TY + 1, 3);
    ok &= make_pool_map16(&tm->s_v, hs.f[0], m, st16, 3, W48, TY + 10, 2);
    ok &= make_pool_map16(&tm->s_lead_xy, hs.f[0], m, st16, 2, W32, TY, 2);
    ok &= make_pool_map16(&tm->s_lead_z, hs.f[2], m, st16, 1, W32, TY, 2);
    ok &= make_pool_map16(&tm->s_own, hs.f[3], m, st16, 6, W32, TY, 2);
    ok &= make_pool_map(&tm->s_med, m.lam, m, st, 5, W32, TY, 2);
    if (!ok) return cudaErrorInvalidValue;
    cudaError_t e = set_attrs<false, SGFD_STORE_BF16>();
    if (e == cudaSuccess) e = set_attrs<true, SGFD_STORE_BF16>();
    if (e == cudaSuccess) e = set_attrs<false, SGFD_STORE_F16>();
    if (e == cudaSuccess) e = set_attrs<true, SGFD_STORE_F16>();
    return e;
}

cudaError_t ztwin16_step(const Model &m, const Physics &ph, const SourceRec &sr, const HalfState &hs, const ZGeom &g,
                         const ZTwin16Maps &tm, int it, float src_value, bool use_wavelet, cudaStream_t s,
                         cudaEvent_t *ev) {
    if (hs.storage == SGFD_STORE_BF16) {
        if (ph.fast) launch<true, SGFD_STORE_BF16>(m, ph, sr, hs, g, tm, it, src_value, use_wavelet, s, ev);
        else launch<false, SGFD_STORE_BF16>(m, ph, sr, hs, g, tm, it, src_value, use_wavelet, s, ev);
    } else {
        if (ph.fast) launch<true, SGFD_STORE_F16>(m, ph, sr, hs, g, tm, it, src_value, use_wavelet, s, ev);
        else launch<false, SGFD_STORE_F16>(m, ph, sr, hs, g, tm, it, src_value, use_wavelet, s, ev);
    }
    return cudaGetLastError();
}

}  // namespace sgfd
