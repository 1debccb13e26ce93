// Device kernels of the multislice engine (sm_100a).
//
// Data layout in HBM follows the reference (column-major, element (iy, ix) at ix*ny + iy, real
// space fft-shifted the way Grid_2d::ind_col_pbc_shift stores the potential, src/types.cuh:2229).
// A probe wave between passes is kept "hybrid": Fourier transformed along y (contiguous lines)
// and real along x. One multislice step psi <- IFFT2[P * FFT2[T * psi]] is then two passes, each
// reading and writing the wave once:
//   rows  (contiguous y-lines): S <- F_y( T * F_y^-1 S )
//   cols  (strided x-lines)   : S <- F_x^-1( P * F_x S )
// because F = F_x F_y and the two 1-D transforms commute. The annular-detector sums of the
// reference's get_psi + sum_square_over_Det (src/wave_function.cuh:96-155) are taken inside the
// column pass right after the P multiply, where the registers hold FFT2(psi)/N.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>

#include "common.hpp"
#include "fft_core.cuh"
#include "kernels.cuh"
#include "launch.cuh"

namespace mtb {

// Kernel launches issued by the calling thread (an engine runs on one host thread). A CUDA graph
// replay adds the launches it holds through add_launches.
static thread_local long long g_launches = 0;
long long launches_issued() { return g_launches; }
void note_launch() { g_launches++; }
void add_launches(long long n) { g_launches += n; }

void encode_tile_map(CUtensorMap* map, const float2* base, int nx, int ldy, int nprobe, int w, int boxr, bool swizzle) {
    static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        MTB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !fn) fail(MT_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }();
    // float32 [nprobe][nx][2*ldy]; box: 2w floats (w complex columns) x boxr rows x 1 probe
    const cuuint64_t dims[3] = {(cuuint64_t)2 * ldy, (cuuint64_t)nx, (cuuint64_t)nprobe};
    const cuuint64_t strides[2] = {(cuuint64_t)2 * ldy * sizeof(float), (cuuint64_t)2 * ldy * nx * sizeof(float)};
    const cuuint32_t box[3] = {(cuuint32_t)(2 * w), (cuuint32_t)boxr, 1};
    const cuuint32_t estride[3] = {1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float2*>(base), dims, strides, box,
                              estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              !swizzle ? CU_TENSOR_MAP_SWIZZLE_NONE
                              : w == 16 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) fail(MT_ERR_CUDA, "cuTensorMapEncodeTiled failed for the column-pass tile map");
}

// =============================================================================================
// Projected potential splat fused with the transmission function.
//
// Projected_Potential::operator() (src/projected_potential.cuh:127-156) evaluates, for every atom
// of a slice and every pixel of its footprint box (get_bn, src/cpu_fcns.hpp:1670-1684),
//   R2 = (ix*dRx + Rx_0 - x)^2 + (iy*dRy + Ry_0 - y)^2;  if R2 < R2_max:
//   V[ind_col_pbc_shift(ix, iy)] += occ * cubic(R2)   (eval_cubic_poly, src/cgpu_fcns.cuh:1498-1567)
// with an FP32 atomicAdd per contribution. Here one CTA owns a tile of 8*PX x 32 pixels of the stored
// (shifted) grid of one slice of one configuration, culls the slice's atoms against its tile, and
// sums the contributions of the surviving atoms in atom order in registers (deterministic, no atomics;
// the tile size changes no sum). The epilogue writes T = exp(i*w*V) (functor::transmission_function,
// src/cgpu_fcns.cuh:3072-3086) directly; V never goes to HBM unless asked for. Float products and sums
// use the _rn intrinsics, so that distances and knot intervals are those of the reference's host float
// path; the cubic itself takes fused multiply-adds (one rounding a step instead of two: potentials
// within 2e-8 of the separately rounded ones, as near to the 64-bit ones).
//
// Bound by instructions. A warp owns PX consecutive x of 32 consecutive y: (x - x_atom)^2 is the same
// for its 32 lanes, so an atom whose circle does not reach a row of the warp costs that row one
// uniform test, and (y - y_atom)^2 is computed once per atom. (By area, for a radius of 40 pixels: 0.6
// of the pixels visited lie inside the circle, 0.17 with a thread's pixels spread over the tile.) Two pixels are
// evaluated together with packed arithmetic, their spline interval found
// from a base-2 logarithm and two exact comparisons with one 8-byte load, the four coefficients from
// one 16-byte load. Measured on one B200 per
// configuration: Si 256^2 x 32 slices 54 -> 26 us (eight configurations in one launch), SrTiO3 512^2 x
// 50 slices 546 -> 325 us, 128^2 x 16 slices 47 -> 15 us, Au(110) 2048^2 x 30 slices 1745 -> 1129 us.
// =============================================================================================
constexpr int SPLAT_TY = 32;   // tile extent along y (contiguous index): one per lane
constexpr int SPLAT_THREADS = 256;
constexpr int SPLAT_WARPS = SPLAT_THREADS / 32;

__device__ __forceinline__ int pmod(int a, int n) {
    int r = a % n;
    return r < 0 ? r + n : r;
}

struct AtomFoot {
    float x, y, occ, R2_max;
    int ix0, nxa, iy0, nya;
    int sx, sy;  // first footprint pixel in stored (shifted) coordinates
    int type, pad;
};

__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// The interval of unrolledBinarySearch_c_nR (src/cgpu_fcns.cuh:1498-1518): the largest i in [0, nR-2]
// with knot[i] <= R2 (0 below the first knot). The knots are log-spaced in R, so the guess is linear in
// log2(R2); exact comparisons decide. Returns knot[i].
__device__ __forceinline__ float spline_interval(const float2* knot, int nR, float scale, float offset, float R2, int& i) {
    // floor of a value in [0.5, nR - 2] through the rounding of a sum with 2^23 - 0.5
    const float g = fminf(fmaxf(__fmaf_rn(__log2f(R2), scale, offset), 0.5f), (float)(nR - 2));
    i = __float_as_int(__fadd_rn(g, 8388607.5f)) - 0x4B000000;
    float2 k = knot[i];
    while (i > 0 && R2 < k.x) k = knot[--i];
    while (i < nR - 2 && !(R2 < k.y)) k = knot[++i];
    return k.x;
}

template <int PX>
__global__ void __launch_bounds__(SPLAT_THREADS) splat_kernel(SplatArgs a, int islice_0, int n_slice) {
    extern __shared__ float4 sm_coef[];  // n_types * nR coefficients (c0..c3)[i], then the knot pairs (R2[i], R2[i+1])
    __shared__ AtomFoot s_list[SPLAT_THREADS];
    __shared__ int s_warp_cnt[SPLAT_WARPS];
    __shared__ float2 s_guess[kMaxTypes];  // log2(R2) -> interval: scale, offset
    constexpr int TX = SPLAT_WARPS * PX;

    previous_done();
    const int nR = a.nR;
    float2* sm_knot = reinterpret_cast<float2*>(sm_coef + a.n_types * nR);
    for (int i = threadIdx.x; i < a.n_types * nR; i += SPLAT_THREADS) {
        const int type = i / nR, k = i - type * nR;
        const float* T = a.tab + (size_t)type * 5 * nR;
        sm_coef[i] = make_float4(T[nR + k], T[2 * nR + k], T[3 * nR + k], T[4 * nR + k]);
        sm_knot[i] = make_float2(T[k], T[k + 1 < nR ? k + 1 : k]);
        if (k == 0) {
            const float lg0 = __log2f(T[0]), scale = (float)(nR - 1) / (__log2f(T[nR - 1]) - lg0);
            s_guess[type] = make_float2(scale, -lg0 * scale);
        }
    }

    const GridDev g = a.g;
    const int iconf = blockIdx.z / n_slice, islice = islice_0 + blockIdx.z % n_slice;
    const float4* atoms = a.conf[iconf].atoms;
    const int2 rng = a.conf[iconf].slice_range[islice];
    const int tx0 = blockIdx.y * TX;
    const int ty0 = blockIdx.x * SPLAT_TY;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int jy = ty0 + lane, jx0 = tx0 + warp * PX;  // this thread's pixels: (jx0 + p, jy)
    unsigned long long V[PX / 2];  // pixels (2q, 2q + 1)
#pragma unroll
    for (int q = 0; q < PX / 2; q++) V[q] = 0ull;

    __syncthreads();
    for (int c0 = rng.x; c0 <= rng.y; c0 += SPLAT_THREADS) {
        const int ia = c0 + threadIdx.x;
        AtomFoot f;
        bool hit = false;
        if (ia <= rng.y) {
            float4 at = atoms[ia];
            f.x = at.x;
            f.y = at.y;
            f.occ = at.z;
            f.type = __float_as_int(at.w);
            const float Rm = a.R_max[f.type];
            f.R2_max = __fmul_rn(Rm, Rm);
            // get_bn (src/cpu_fcns.hpp:1670-1684), periodic
            int i0 = (int)floorf(__fdiv_rn(__fsub_rn(f.x, Rm), g.dRx));
            int ie = (int)ceilf(__fdiv_rn(__fadd_rn(f.x, Rm), g.dRx));
            f.ix0 = i0;
            f.nxa = (i0 == ie) ? 0 : ie - i0 + 1;
            i0 = (int)floorf(__fdiv_rn(__fsub_rn(f.y, Rm), g.dRy));
            ie = (int)ceilf(__fdiv_rn(__fadd_rn(f.y, Rm), g.dRy));
            f.iy0 = i0;
            f.nya = (i0 == ie) ? 0 : ie - i0 + 1;
            f.sx = (pmod(f.ix0, g.nx) + g.nxh) % g.nx;
            f.sy = (pmod(f.iy0, g.ny) + g.nyh) % g.ny;
            // circular overlap of [sx, sx+nxa) with [tx0, tx0+TX) (and y)
            bool ox = (f.nxa >= g.nx) || (pmod(tx0 - f.sx, g.nx) < f.nxa) || (pmod(f.sx - tx0, g.nx) < TX);
            bool oy = (f.nya >= g.ny) || (pmod(ty0 - f.sy, g.ny) < f.nya) || (pmod(f.sy - ty0, g.ny) < SPLAT_TY);
            hit = ox && oy && f.nxa > 0 && f.nya > 0;
        }
        // deterministic compaction in atom order
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) s_warp_cnt[warp] = __popc(m);
        __syncthreads();
        int n = 0, first = 0;
#pragma unroll
        for (int w = 0; w < SPLAT_WARPS; w++) {
            if (w == warp) first = n;
            n += s_warp_cnt[w];
        }
        if (hit) s_list[first + __popc(m & ((1u << lane) - 1u))] = f;
        __syncthreads();
        for (int k = 0; k < n; k++) {
            const AtomFoot af = s_list[k];
            const float2* knot = sm_knot + af.type * nR;
            const float4* coef = sm_coef + af.type * nR;
            const float2 guess = s_guess[af.type];
            // offset in the footprint, of the first periodic image (jy and sy are both in [0, ny))
            int offy = jy - af.sy;
            if (offy < 0) offy += g.ny;
            if (af.nxa <= g.nx && af.nya <= g.ny) {  // at most one image of the footprint at each pixel
                const float Ry = __fsub_rn(__fadd_rn(__fmul_rn((float)(af.iy0 + offy), g.dRy), g.Ry_0), af.y);
                const float Ry2 = __fmul_rn(Ry, Ry);
                const bool iny = offy < af.nya && Ry2 < af.R2_max;
                if (!__any_sync(0xffffffffu, iny)) continue;
                const unsigned long long occ = pack2(make_float2(af.occ, af.occ));
#pragma unroll
                for (int q = 0; q < PX / 2; q++) {
                    float R2[2];
                    bool in[2];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        int offx = jx0 + 2 * q + h - af.sx;
                        if (offx < 0) offx += g.nx;
                        const float Rx = __fsub_rn(__fadd_rn(__fmul_rn((float)(af.ix0 + offx), g.dRx), g.Rx_0), af.x);
                        const float Rx2 = __fmul_rn(Rx, Rx);
                        R2[h] = __fadd_rn(Rx2, Ry2);
                        in[h] = offx < af.nxa && Rx2 < af.R2_max;  // the same for every lane
                    }
                    if (!in[0] && !in[1]) continue;
                    in[0] = in[0] && iny && R2[0] < af.R2_max;
                    in[1] = in[1] && iny && R2[1] < af.R2_max;
                    if (!in[0] && !in[1]) continue;
                    int i0, i1;
                    const float d0 = __fsub_rn(R2[0], spline_interval(knot, nR, guess.x, guess.y, R2[0], i0));
                    const float d1 = __fsub_rn(R2[1], spline_interval(knot, nR, guess.x, guess.y, R2[1], i1));
                    const float4 e0 = coef[i0], e1 = coef[i1];
                    const unsigned long long d = pack2(make_float2(d0, d1));
                    unsigned long long v = fma2(pack2(make_float2(e0.w, e1.w)), d, pack2(make_float2(e0.z, e1.z)));
                    v = fma2(v, d, pack2(make_float2(e0.y, e1.y)));
                    v = fma2(v, d, pack2(make_float2(e0.x, e1.x)));
                    const float2 r = unpack2(mul2(occ, v));
                    V[q] = add2(V[q], pack2(make_float2(in[0] ? r.x : 0.0f, in[1] ? r.y : 0.0f)));
                }
            } else {  // a footprint wider than the grid: every image in order
#pragma unroll
                for (int p = 0; p < PX; p++) {
                    int offx = jx0 + p - af.sx;
                    if (offx < 0) offx += g.nx;
                    for (int ox = offx; ox < af.nxa; ox += g.nx) {
                        const float Rx = __fsub_rn(__fadd_rn(__fmul_rn((float)(af.ix0 + ox), g.dRx), g.Rx_0), af.x);
                        for (int oy = offy; oy < af.nya; oy += g.ny) {
                            const float Ry = __fsub_rn(__fadd_rn(__fmul_rn((float)(af.iy0 + oy), g.dRy), g.Ry_0), af.y);
                            const float R2 = __fadd_rn(__fmul_rn(Rx, Rx), __fmul_rn(Ry, Ry));
                            if (R2 < af.R2_max) {
                                int i;
                                const float dx = __fsub_rn(R2, spline_interval(knot, nR, guess.x, guess.y, R2, i));
                                const float4 e = coef[i];
                                float v = __fmaf_rn(e.w, dx, e.z);
                                v = __fmaf_rn(v, dx, e.y);
                                v = __fmaf_rn(v, dx, e.x);
                                v = __fmul_rn(af.occ, v);
                                float2 s = unpack2(V[p / 2]);
                                (p % 2 ? s.y : s.x) += v;
                                V[p / 2] = pack2(s);
                            }
                        }
                    }
                }
            }
        }
        __syncthreads();
    }
    const size_t base = (size_t)iconf * a.trans_stride + (size_t)islice * g.nx * g.ny;
#pragma unroll
    for (int p = 0; p < PX; p++) {
        const size_t idx = base + (size_t)(jx0 + p) * g.ny + jy;
        const float2 s = unpack2(V[p / 2]);
        const float v = p % 2 ? s.y : s.x;
        if (a.V) a.V[idx] = v;
        if (a.trans) {
            const float th = __fmul_rn(a.w, v);
            float sn, cs;
            if (a.wpo) {
                cs = 1.0f;
                sn = th;
            } else {
                sincosf(th, &sn, &cs);
            }
            a.trans[idx] = make_float2(cs, sn);
        }
    }
    next_may_start();
}

template <int PX>
static void splat_launch(const SplatArgs& a, int islice_0, int n_slice, cudaStream_t s) {
    const dim3 grid(a.g.ny / SPLAT_TY, a.g.nx / (SPLAT_WARPS * PX), n_slice * a.n_conf);
    const size_t sm = (size_t)a.n_types * a.nR * (sizeof(float4) + sizeof(float2));
    // the same limit in every launch: it is the kernel's, and other host threads launch with tables of their own size
    constexpr size_t most = (size_t)kMaxTypes * kMaxKnots * (sizeof(float4) + sizeof(float2));
    if (sm > most) fail(MT_ERR_UNSUPPORTED, "spline tables larger than the splat's shared memory");
    MTB_CUDA(cudaFuncSetAttribute(splat_kernel<PX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    launch_early(true, splat_kernel<PX>, grid, SPLAT_THREADS, sm, s, a, islice_0, n_slice);
    g_launches++;
}

// Slices islice_0 .. islice_0 + n_slice - 1 of the n_conf configurations of `a`, as many configurations per
// launch as the grid's z extent takes (65535 slices in all). Taller warps (more pixels per thread) reuse a
// lane's (y - y_atom)^2 more often; shorter ones where the tiles would leave an SM with less than four CTAs.
void launch_splat(const SplatArgs& a, int islice_0, int n_slice, cudaStream_t s) {
    if (a.g.nx % (SPLAT_WARPS * 8) || a.g.ny % SPLAT_TY) fail(MT_ERR_UNSUPPORTED, "grid must be a multiple of 64 x 32");
    const int most = std::max(1, 65535 / n_slice);
    if (a.n_conf > most) {
        for (int c = 0; c < a.n_conf; c += most) {
            SplatArgs part = a;
            part.n_conf = std::min(most, a.n_conf - c);
            std::copy(a.conf + c, a.conf + c + part.n_conf, part.conf);
            if (a.trans) part.trans = a.trans + c * a.trans_stride;
            if (a.V) part.V = a.V + c * a.trans_stride;
            launch_splat(part, islice_0, n_slice, s);
        }
        return;
    }
    const long long tiles = (long long)(a.g.nx / 64) * (a.g.ny / SPLAT_TY) * n_slice * a.n_conf;
    if (tiles >= 4 * 148) splat_launch<8>(a, islice_0, n_slice, s);
    else if (2 * tiles >= 4 * 148) splat_launch<4>(a, islice_0, n_slice, s);
    else splat_launch<2>(a, islice_0, n_slice, s);
}

// =============================================================================================
// Line passes
// =============================================================================================
template <int NY>
void rows_dispatch_mode(RowMode mode, const RowArgs& a, int grid_ctas, cudaStream_t s);
template <int NX>
void cols_dispatch_flags(int flags, const ColArgs& a, int grid_ctas, cudaStream_t s);

template <int NY>
bool rows_has_variant(int v, int nprobe, bool one_trans);
template <int NX>
bool cols_has_variant(int v);

bool rows_step_has_variant(int ny, int v, int nprobe, bool one_trans) {
    switch (ny) {
        case 64: return rows_has_variant<64>(v, nprobe, one_trans);
        case 128: return rows_has_variant<128>(v, nprobe, one_trans);
        case 256: return rows_has_variant<256>(v, nprobe, one_trans);
        case 384: return rows_has_variant<384>(v, nprobe, one_trans);
        case 512: return rows_has_variant<512>(v, nprobe, one_trans);
        case 1024: return rows_has_variant<1024>(v, nprobe, one_trans);
        case 2048: return rows_has_variant<2048>(v, nprobe, one_trans);
        default: return v == 0;
    }
}

bool cols_step_has_variant(int nx, int v) {
    switch (nx) {
        case 64: return cols_has_variant<64>(v);
        case 128: return cols_has_variant<128>(v);
        case 256: return cols_has_variant<256>(v);
        case 384: return cols_has_variant<384>(v);
        case 512: return cols_has_variant<512>(v);
        case 1024: return cols_has_variant<1024>(v);
        case 2048: return cols_has_variant<2048>(v);
        default: return v == 0;
    }
}

template <int N>
constexpr int lines_per_cta() {
    return LinePlan<N>::T / (N / LinePlan<N>::E);
}

static int lines_per_cta(int n) {
    switch (n) {
        case 64: return lines_per_cta<64>();
        case 128: return lines_per_cta<128>();
        case 256: return lines_per_cta<256>();
        case 384: return lines_per_cta<384>();
        case 512: return lines_per_cta<512>();
        case 1024: return lines_per_cta<1024>();
        case 2048: return lines_per_cta<2048>();
        default: fail(MT_ERR_UNSUPPORTED, "grid sizes must be one of 64, 128, 256, 384, 512, 1024, 2048");
    }
    return 0;
}

template <int NX>
int cols_det_width();

int col_det_width(int nx) {
    switch (nx) {
        case 64: return cols_det_width<64>();
        case 128: return cols_det_width<128>();
        case 256: return cols_det_width<256>();
        case 384: return cols_det_width<384>();
        case 512: return cols_det_width<512>();
        case 1024: return cols_det_width<1024>();
        case 2048: return cols_det_width<2048>();
        default: fail(MT_ERR_UNSUPPORTED, "nx must be one of 64, 128, 256, 384, 512, 1024, 2048");
    }
    return 0;
}

int col_tiles(int nx, int ny) {
    const int w = col_det_width(nx);
    if (ny % w != 0) fail(MT_ERR_UNSUPPORTED, "ny must be a multiple of the column-pass tile width");
    return ny / w;
}

void launch_rows(int ny, RowMode mode, const RowArgs& a, int grid_ctas, cudaStream_t s) {
    if (a.nx % lines_per_cta(ny) != 0) fail(MT_ERR_UNSUPPORTED, "nx must be a multiple of the row-pass line group");
    switch (ny) {
        case 64: rows_dispatch_mode<64>(mode, a, grid_ctas, s); break;
        case 128: rows_dispatch_mode<128>(mode, a, grid_ctas, s); break;
        case 256: rows_dispatch_mode<256>(mode, a, grid_ctas, s); break;
        case 384: rows_dispatch_mode<384>(mode, a, grid_ctas, s); break;
        case 512: rows_dispatch_mode<512>(mode, a, grid_ctas, s); break;
        case 1024: rows_dispatch_mode<1024>(mode, a, grid_ctas, s); break;
        case 2048: rows_dispatch_mode<2048>(mode, a, grid_ctas, s); break;
        default: fail(MT_ERR_UNSUPPORTED, "ny must be one of 64, 128, 256, 384, 512, 1024, 2048");
    }
}

void launch_cols(int nx, int flags, const ColArgs& a, int grid_ctas, cudaStream_t s) {
    if (a.ny % lines_per_cta(nx) != 0) fail(MT_ERR_UNSUPPORTED, "ny must be a multiple of the column-pass tile width");
    switch (nx) {
        case 64: cols_dispatch_flags<64>(flags, a, grid_ctas, s); break;
        case 128: cols_dispatch_flags<128>(flags, a, grid_ctas, s); break;
        case 256: cols_dispatch_flags<256>(flags, a, grid_ctas, s); break;
        case 384: cols_dispatch_flags<384>(flags, a, grid_ctas, s); break;
        case 512: cols_dispatch_flags<512>(flags, a, grid_ctas, s); break;
        case 1024: cols_dispatch_flags<1024>(flags, a, grid_ctas, s); break;
        case 2048: cols_dispatch_flags<2048>(flags, a, grid_ctas, s); break;
        default: fail(MT_ERR_UNSUPPORTED, "nx must be one of 64, 128, 256, 384, 512, 1024, 2048");
    }
}

// =============================================================================================
// Detector reduction: one thread per (probe, detector); tiles summed in order (deterministic).
__global__ void det_reduce_kernel(const double* partial, int nprobe, int n_tiles, int n_det,
                                  const int* scan_index, double w, double* image,
                                  int n_scan) {
    previous_done();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nprobe * n_det) return;
    const int b = i / n_det, d = i % n_det;
    double s = 0.0;
    for (int k = 0; k < n_tiles; k++) s += partial[((size_t)b * n_tiles + k) * n_det + d];
    image[(size_t)d * n_scan + scan_index[b]] += w * s;
    next_may_start();
}

void launch_det_reduce(const double* partial, int nprobe, int n_tiles, int n_det, const int* scan_index, double w,
                       double* image, int n_scan, cudaStream_t s) {
    const int n = nprobe * n_det;
    launch_early(true, det_reduce_kernel, (n + 127) / 128, 128, 0, s, partial, nprobe, n_tiles, n_det, scan_index, w, image, n_scan);
    g_launches++;
}

// =============================================================================================
__global__ void tilt_ramp_kernel(GridDev g, float gx, float gy, float rxc, float ryc, float2* __restrict__ out) {
    const int iy = blockIdx.x * blockDim.x + threadIdx.x, ix = blockIdx.y;
    if (iy >= g.ny) return;
    const float rx = __fsub_rn(__fadd_rn(__fmul_rn((float)((ix < g.nxh) ? ix + g.nxh : ix - g.nxh), g.dRx), g.Rx_0), rxc);
    const float ry = __fsub_rn(__fadd_rn(__fmul_rn((float)((iy < g.nyh) ? iy + g.nyh : iy - g.nyh), g.dRy), g.Ry_0), ryc);
    const double th = (double)__fadd_rn(__fmul_rn(gx, rx), __fmul_rn(gy, ry));
    double sn, cs;
    sincos(th, &sn, &cs);
    const double s = 1.0 / (double)g.ny;
    out[(size_t)ix * g.ny + iy] = make_float2((float)(cs * s), (float)(sn * s));
}

void launch_tilt_ramp(const GridDev& g, float gx, float gy, float rxc, float ryc, float2* out, cudaStream_t s) {
    tilt_ramp_kernel<<<dim3((unsigned)((g.ny + 127) / 128), (unsigned)g.nx), 128, 0, s>>>(g, gx, gy, rxc, ryc, out);
    g_launches++;
    MTB_CUDA(cudaGetLastError());
}

__global__ void mul_tables_kernel(float2* __restrict__ a, const float2* __restrict__ b, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        a[i] = cmul(a[i], b[i]);
}

void launch_mul_tables(float2* a, const float2* b, size_t n, cudaStream_t s) {
    mul_tables_kernel<<<(unsigned)std::min<size_t>((n + 255) / 256, 148 * 8), 256, 0, s>>>(a, b, n);
    g_launches++;
    MTB_CUDA(cudaGetLastError());
}

__global__ void sum_waves_kernel(const float2* __restrict__ src, int n, size_t nxy, float2* __restrict__ dst) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nxy; i += (size_t)gridDim.x * blockDim.x) {
        float2 acc = src[i];
        for (int j = 1; j < n; j++) {
            const float2 v = src[(size_t)j * nxy + i];
            acc = make_float2(__fadd_rn(acc.x, v.x), __fadd_rn(acc.y, v.y));
        }
        dst[i] = acc;
    }
}

// dst += w * src over nxy complex values (add_scale, src/output_multislice.hpp:770-780)
__global__ void axpy_wave_kernel(const float2* __restrict__ src, float w, size_t nxy, float2* __restrict__ dst) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nxy; i += (size_t)gridDim.x * blockDim.x) {
        const float2 v = src[i], d = dst[i];
        dst[i] = make_float2(__fadd_rn(d.x, __fmul_rn(w, v.x)), __fadd_rn(d.y, __fmul_rn(w, v.y)));
    }
}

void launch_axpy_wave(const float2* src, float w, size_t nxy, float2* dst, cudaStream_t s) {
    axpy_wave_kernel<<<(unsigned)std::min<size_t>((nxy + 255) / 256, 148 * 8), 256, 0, s>>>(src, w, nxy, dst);
    g_launches++;
    MTB_CUDA(cudaGetLastError());
}

void launch_sum_waves(const float2* src, int n, size_t nxy, float2* dst, cudaStream_t s) {
    sum_waves_kernel<<<(unsigned)std::min<size_t>((nxy + 255) / 256, 148 * 8), 256, 0, s>>>(src, n, nxy, dst);
    g_launches++;
    MTB_CUDA(cudaGetLastError());
}

// One CTA per (thickness, scan position): detector sums of |psi_coh|^2 over the grid, per-thread
// partials in FP64 reduced in a fixed order.
__global__ void coh_detect_kernel(const float2* __restrict__ coh, int n_scan, ColArgs a, double* __restrict__ image) {
    const int ithk = blockIdx.x / n_scan, iscan = blockIdx.x % n_scan;
    const size_t nxy = (size_t)a.g.nx * a.g.ny;
    const float2* c = coh + ((size_t)ithk * n_scan + iscan) * nxy;
    double acc[kMaxDet];
#pragma unroll
    for (int d = 0; d < kMaxDet; d++) acc[d] = 0.0;
    for (size_t p = threadIdx.x; p < nxy; p += blockDim.x) {
        const int ix = (int)(p / a.g.ny), iy = (int)(p % a.g.ny);
        const float2 v = c[p];
        const float v2 = __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y));
        if (a.det_mat) {
#pragma unroll
            for (int d = 0; d < kMaxDet; d++)
                if (d < a.n_det) acc[d] += (double)__fmul_rn(a.det_mat[d * nxy + p], v2);
        } else {
            const float gx = __fmul_rn((float)((ix < a.g.nxh) ? ix : ix - a.g.nx), a.g.dgx);
            const float gy = __fmul_rn((float)((iy < a.g.nyh) ? iy : iy - a.g.ny), a.g.dgy);
            const float g2 = __fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy));
#pragma unroll
            for (int d = 0; d < kMaxDet; d++)
                if (d < a.n_det && a.det_g2_min[d] <= g2 && g2 < a.det_g2_max[d]) acc[d] += (double)v2;
        }
    }
    __shared__ double red[kMaxDet][256];
#pragma unroll
    for (int d = 0; d < kMaxDet; d++) red[d][threadIdx.x] = acc[d];
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s)
#pragma unroll
            for (int d = 0; d < kMaxDet; d++) red[d][threadIdx.x] += red[d][threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x < (unsigned)a.n_det)
        image[((size_t)ithk * a.n_det + threadIdx.x) * n_scan + iscan] = red[threadIdx.x][0];
}

void launch_coh_detect(const float2* coh, int n_thk, int n_scan, const ColArgs& det, double* image_coh,
                       cudaStream_t s) {
    coh_detect_kernel<<<(unsigned)(n_thk * n_scan), 256, 0, s>>>(coh, n_scan, det, image_coh);
    g_launches++;
    MTB_CUDA(cudaGetLastError());
}

// EW output accumulation with fft-shift and crop (add_scale_crop_shift_2d /
// add_scale_square_crop_shift_2d / assign_crop_shift_2d, src/cgpu_fcns.cuh:1681-1780).
__global__ void ew_accumulate_kernel(const float2* psi, int nx, int ny, int ix0, int ix1, int iy0,
                                     int iy1, double w, int assign, double* psi_out,
                                     double* m2_out, int nwave) {
    previous_done();
    const int iy = blockIdx.x * blockDim.x + threadIdx.x;
    const int ix = blockIdx.y;
    if (iy >= ny || ix >= nx) return;
    if (ix < ix0 || ix >= ix1 || iy < iy0 || iy >= iy1) return;
    // output pixel (ix, iy) takes the stored pixel shifted by half the grid
    const int sx = (ix + nx / 2) % nx, sy = (iy + ny / 2) % ny;
    const float2 v = psi[(size_t)sx * ny + sy];
    const size_t o = (size_t)(ix - ix0) * (iy1 - iy0) + (iy - iy0);
    if (psi_out) {
        if (assign) {
            psi_out[2 * o] = v.x;
            psi_out[2 * o + 1] = v.y;
        } else {
            psi_out[2 * o] += w * v.x;
            psi_out[2 * o + 1] += w * v.y;
        }
    }
    if (m2_out) {
        double acc = 0.0;
        for (int j = 0; j < nwave; j++) {
            const float2 u = (j == 0) ? v : psi[(size_t)j * nx * ny + (size_t)sx * ny + sy];
            const float n2 = __fadd_rn(__fmul_rn(u.x, u.x), __fmul_rn(u.y, u.y));
            acc += w * (double)n2;
        }
        m2_out[o] += acc;
    }
    next_may_start();
}

void launch_ew_accumulate(const float2* psi, int nx, int ny, int ix0, int ix1, int iy0, int iy1, double w,
                          int assign, double* psi_out, double* m2_out, cudaStream_t s, int nwave) {
    dim3 grid((ny + 127) / 128, nx);
    launch_early(true, ew_accumulate_kernel, grid, 128, 0, s, psi, nx, ny, ix0, ix1, iy0, iy1, w, assign, psi_out, m2_out, nwave);
    g_launches++;
}

// 32 x 32 tiles through shared memory, both sides coalesced.
template <class T>
__global__ void __launch_bounds__(256) transpose_kernel(const T* __restrict__ src, T* __restrict__ dst, int nx, int ny, int ld) {
    __shared__ T tile[32][33];
    const size_t sp = (size_t)blockIdx.z * nx * ld, dp = (size_t)blockIdx.z * nx * ny;
    const int lx = threadIdx.x % 32, ly = threadIdx.x / 32;
    const int iy0 = blockIdx.x * 32, ix0 = blockIdx.y * 32;
    for (int r = ly; r < 32; r += 8)
        if (ix0 + r < nx && iy0 + lx < ny) tile[r][lx] = src[sp + (size_t)(ix0 + r) * ld + iy0 + lx];
    __syncthreads();
    for (int r = ly; r < 32; r += 8)
        if (iy0 + r < ny && ix0 + lx < nx) dst[dp + (size_t)(iy0 + r) * nx + ix0 + lx] = tile[lx][r];
}

void launch_transpose(const double* src, double* dst, size_t planes, int nx, int ny, int ld, int width, cudaStream_t s) {
    const size_t sn = (size_t)nx * ld * width, dn = (size_t)nx * ny * width;
    for (size_t p = 0; p < planes; p += 65535) {
        const dim3 grid((unsigned)((ny + 31) / 32), (unsigned)((nx + 31) / 32), (unsigned)std::min<size_t>(65535, planes - p));
        if (width == 2)
            transpose_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<const double2*>(src + p * sn),
                                                  reinterpret_cast<double2*>(dst + p * dn), nx, ny, ld);
        else
            transpose_kernel<<<grid, 256, 0, s>>>(src + p * sn, dst + p * dn, nx, ny, ld);
        g_launches++;
        MTB_CUDA(cudaGetLastError());
    }
}

}  // namespace mtb
