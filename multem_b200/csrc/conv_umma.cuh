// 3x3 convolutions (zero padding 1) of NCHW bf16 tensors as implicit GEMMs on the fifth-generation
// tensor cores (tcgen05, sm_100a), FP32 accumulation in tensor memory.
//
// Pixels are numbered in a padded line: image b, row y, column x is q = (b*(H+1) + y)*(W+1) + x, with
// one zero column after each row and one zero row after each image. The tap (ky, kx) of pixel q is
// then always q + (ky-1)*(W+1) + (kx-1): every neighbour outside the image falls on a zero. A tile
// of consecutive q is gathered once into shared memory as planes of 8 channels,
//
//   plane[c / 8][pixel][c % 8]      (16 bytes per pixel and plane),
//
// which is the MMA's unswizzled operand layout for either major-ness: as a K-major operand (K =
// channels) a core matrix is 8 consecutive pixels x 8 channels, as an MN-major operand (K = pixels)
// 8 channels x 8 consecutive pixels. A tap is a shift of the operand's start address by whole
// pixels, 16 bytes each, so the nine taps read the one gathered tile and nothing is expanded in
// global memory. The pixels gathered for a tile of T: the band of T + 2*(W+1) + 2 around it, or,
// where that is longer, three segments of T + 2 (one per ky).
//
// The operands come through threads (2-byte loads coalesced along the pixels, 16-byte conflict-free
// stores): a tensor copy cannot start at an odd pixel of a 2-byte type nor interleave channels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "launch.cuh"
#include "mbarrier.cuh"

namespace mtb {
namespace conv {

constexpr int THREADS = 256;
constexpr int KC = 32;          // channels per K block of the forward and data-gradient pass
constexpr int WG_PIX = 128;     // pixels per K block of the weight gradient
constexpr int WG_OC = 32;       // output channels per CTA of the weight gradient
constexpr long long kNoPixel = -1;

// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), A and B BF16 (bits 7-9,
// 10-12 = 1), A / B MN-major (bits 15, 16), N >> 3 at bits 17-22, M >> 4 at bits 24-28.
constexpr uint32_t idesc(int m, int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Shared-memory matrix descriptor without swizzle (layout type 0, version 1 at bit 46): start address,
// leading and stride byte offsets in 16-byte units at bits 0-13, 16-29, 32-45. K-major: leading = the step
// between the two 8-wide halves of K, stride = the step between groups of 8 rows. MN-major: leading =
// the step between groups of 8 along K, stride = the step between groups of 8 along M or N.
// Steps are small enough that moving the start address is an addition to the low word.
__device__ __forceinline__ uint32_t desc_lo(unsigned saddr, unsigned leading) {
    return (saddr & 0x3FFFFu) >> 4 | (leading >> 4) << 16;  // a cluster's addresses carry the CTA's rank above
}
__device__ __forceinline__ uint64_t desc(uint32_t lo, unsigned stride) {
    return (uint64_t)lo | (uint64_t)(stride >> 4 | 1u << 14) << 32;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(unsigned* slot, unsigned ncols) {  // whole warp
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(unsigned taddr, unsigned ncols) {  // whole warp
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void mma_bf16(unsigned tmem_d, uint64_t da, uint64_t db, uint32_t id, unsigned acc) {
    const unsigned z0 = 0, z1 = 0, z2 = 0, z3 = 0;  // no output lanes disabled
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(id), "r"(acc), "r"(z0), "r"(z1), "r"(z2), "r"(z3)
        : "memory");
}
// arrive on `bar` once every MMA this thread issued before has completed
__device__ __forceinline__ void mma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// The load and its wait are one statement: nothing ties the registers to a wait of its own, so arithmetic on them
// could be placed before it.
__device__ __forceinline__ void tmem_ld16(unsigned taddr, uint32_t (&r)[16]) {  // whole warp
    __syncwarp();  // the instruction needs the warp together, whatever branches came before
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n"
        " tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// Barrier over the threads of the cluster's CTAs, ordering their shared memory. Not the .aligned form: a warp's
// threads may arrive apart (after per-pixel branches), and that form would count the warp twice.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
// The 16 bytes at this CTA's shared-memory address p in the cluster's CTA `rank`.
__device__ __forceinline__ float4 peer_load4(const float* p, int rank) {
    unsigned at;
    float4 v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(at)
                 : "memory");
    return v;
}

// Tensor-memory columns of an allocation: a power of two, at least 32.
constexpr unsigned tmem_cols(unsigned n) {
    unsigned c = 32;
    while (c < n) c *= 2;
    return c;
}

struct Image {  // the padded line of a [B][C][H][W] tensor's pixels
    int B, H, W;
    uint32_t inv_w, inv_h;  // floor(2^32 / (W + 1)), floor(2^32 / (H + 1))
    __host__ __device__ long long total() const { return (long long)B * (H + 1) * (W + 1); }
};
inline Image image(int B, int H, int W) {
    return {B, H, W, (uint32_t)((1ull << 32) / (unsigned)(W + 1)), (uint32_t)((1ull << 32) / (unsigned)(H + 1))};
}

// v / d from inv = floor(2^32 / d), d >= 2: the product's high word is the quotient or one less.
__device__ __forceinline__ uint32_t quotient(uint32_t v, uint32_t d, uint32_t inv) {
    const uint32_t q = __umulhi(v, inv);
    return v - q * d >= d ? q + 1 : q;
}

// Position q of the line: its image and the position within that image's (H+1)*(W+1).
__device__ __forceinline__ void locate(const Image& im, long long q, int& b, uint32_t& r) {
    const uint32_t n = (uint32_t)(im.H + 1) * (uint32_t)(im.W + 1);  // below 2^32: H*W is at most 2^30
    if ((q >> 32) == 0) {
        b = (int)((uint32_t)q / n);
        r = (uint32_t)q - (uint32_t)b * n;
    } else {
        b = (int)(q / n);
        r = (uint32_t)(q - (long long)b * n);
    }
}

// The pixel `d` positions after position r of image b0: its offset from in[b0][0][0][0] for C channels,
// or kNoPixel for a zero. d reaches at most a row and a column back, where there are only zeros
// before the image.
__device__ __forceinline__ long long pixel_offset(const Image& im, int C, int b0, uint32_t r, int d) {
    if (d < 0 && r < (uint32_t)(-d)) return kNoPixel;
    const uint32_t v = r + (uint32_t)d, Wp = im.W + 1, Hp = im.H + 1;
    const uint32_t row = quotient(v, Wp, im.inv_w), x = v - row * Wp;
    const uint32_t b = quotient(row, Hp, im.inv_h), y = row - b * Hp;
    if ((int)b >= im.B - b0 || y >= (uint32_t)im.H || x >= (uint32_t)im.W) return kNoPixel;
    return ((long long)b * C * im.H + y) * im.W + x;
}

__device__ __forceinline__ uint16_t ld16(const __nv_bfloat16* p) {
    return *reinterpret_cast<const unsigned short*>(p);
}

// 8 channels of a pixel packed in order.
__device__ __forceinline__ uint4 pack8(const uint32_t (&v)[8]) {
    return make_uint4(__byte_perm(v[0], v[1], 0x5410u), __byte_perm(v[2], v[3], 0x5410u),
                      __byte_perm(v[4], v[5], 0x5410u), __byte_perm(v[6], v[7], 0x5410u));
}
// the halves of v where m > 0 (not for NaN), zero elsewhere
__device__ __forceinline__ uint32_t positive2(uint32_t v, uint32_t m) {
    __nv_bfloat162 h;
    *reinterpret_cast<uint32_t*>(&h) = m;
    return v & __hgt2_mask(h, __nv_bfloat162(__ushort_as_bfloat16(0), __ushort_as_bfloat16(0)));
}

struct Source {  // one image's channels of a gather: image b0 of the tensor and of its mask (or NULL)
    const __nv_bfloat16* in;
    const __nv_bfloat16* mask;
    size_t hw;
    int nc;  // channels of the tensor
};

// U items (16-byte pieces: pixel offsets off[u], channels c[u] .. c[u]+7) with every load in flight
// before the first is used; zero for kNoPixel, past nc channels and where the mask is not positive. The
// addresses of skipped values stay inside the image (its first value), so no load is branched around.
// FULL: nc is a multiple of 8.
template <int U, bool FULL, bool MASK>
__device__ __forceinline__ void gather_items(const Source& src, const long long (&off)[U], const int (&c)[U], uint4 (&out)[U]) {
    uint32_t v[U][8], m[MASK ? U : 1][8];
    bool skip[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        skip[u] = off[u] == kNoPixel || c[u] >= src.nc;
        const size_t at = skip[u] ? 0 : (size_t)off[u] + (size_t)c[u] * src.hw;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const size_t aj = FULL || (!skip[u] && c[u] + j < src.nc) ? at + j * src.hw : at;
            v[u][j] = ld16(src.in + aj);
            if constexpr (MASK) m[u][j] = ld16(src.mask + aj);
        }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        if constexpr (!FULL) {
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (c[u] + j >= src.nc) v[u][j] = 0u;
        }
        uint4 r = pack8(v[u]);
        if constexpr (MASK) {
            const uint4 k = pack8(m[u]);
            r = make_uint4(positive2(r.x, k.x), positive2(r.y, k.y), positive2(r.z, k.z), positive2(r.w, k.w));
        }
        out[u] = skip[u] ? make_uint4(0u, 0u, 0u, 0u) : r;
    }
}

// Planes dst[p][s] (p < nplane, s < npix) of the channels c0 .. c0 + 8*nplane - 1 at the pixel offsets
// s_off, by all threads; use(v, p) sees every piece.
template <bool FULL, bool MASK, class Use>
__device__ __forceinline__ void gather_planes(const Source& src, const long long* s_off, int c0, int nplane, int npix,
                                              uint4* dst, Use use) {
    constexpr int U = 2;
    int p = 0, s = threadIdx.x;
    while (s >= npix) s -= npix, p++;
    for (int e = threadIdx.x; e < nplane * npix; e += U * THREADS) {
        long long off[U];
        int c[U];
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            off[u] = p < nplane ? s_off[s] : kNoPixel;
            c[u] = c0 + 8 * p;
            s += THREADS;
            while (s >= npix) s -= npix, p++;
        }
        gather_items<U, FULL, MASK>(src, off, c, v);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int at = e + u * THREADS;
            if (at < nplane * npix) dst[at] = v[u];
            use(v[u], (c[u] - c0) / 8);
        }
    }
}
template <class Use>
__device__ __forceinline__ void gather(const Source& src, const long long* s_off, int c0, int nplane, int npix, uint4* dst,
                                       Use use) {
    if (src.nc % 8 == 0) {
        if (src.mask) gather_planes<true, true>(src, s_off, c0, nplane, npix, dst, use);
        else gather_planes<true, false>(src, s_off, c0, nplane, npix, dst, use);
    } else {
        if (src.mask) gather_planes<false, true>(src, s_off, c0, nplane, npix, dst, use);
        else gather_planes<false, false>(src, s_off, c0, nplane, npix, dst, use);
    }
}

// The 8 x 9 block of weights w[row][col .. col+7][0 .. 8] (9*Ccol values per row) as one 16-byte vector of
// 8 columns per tap; zero outside the matrix. `vec`: rows are whole 16-byte units.
__device__ __forceinline__ void weights8(const __nv_bfloat16* w, int row, int nrow, int col, int ncol, bool vec,
                                         uint4 (&out)[9]) {
    uint32_t h[36];  // 72 values, two per word
    if (row >= nrow || col >= ncol) {
#pragma unroll
        for (int i = 0; i < 36; i++) h[i] = 0u;
    } else {
        const __nv_bfloat16* p = w + ((size_t)row * ncol + col) * 9;
        if (vec) {
#pragma unroll
            for (int i = 0; i < 9; i++) {
                const uint4 u = reinterpret_cast<const uint4*>(p)[i];
                h[4 * i] = u.x, h[4 * i + 1] = u.y, h[4 * i + 2] = u.z, h[4 * i + 3] = u.w;
            }
        } else {
            const int n = (ncol - col < 8 ? ncol - col : 8) * 9;
#pragma unroll
            for (int i = 0; i < 36; i++) {
                const uint32_t lo = 2 * i < n ? ld16(p + 2 * i) : 0u, hi = 2 * i + 1 < n ? ld16(p + 2 * i + 1) : 0u;
                h[i] = lo | hi << 16;
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 9; t++) {
        uint32_t r[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int e0 = 18 * j + t, e1 = e0 + 9;  // columns 2j and 2j+1
            r[j] = __byte_perm(h[e0 >> 1], h[e1 >> 1], ((e0 & 1) ? 0x32u : 0x10u) | ((e1 & 1) ? 0x7600u : 0x5400u));
        }
        out[t] = make_uint4(r[0], r[1], r[2], r[3]);
    }
}

// whether the low (bit 0) and the high (bit 1) bf16 of a word are infinities or NaN (exponent bits all set)
__device__ __forceinline__ unsigned nonfinite(uint32_t u) {
    return ((u & 0x7F80u) == 0x7F80u ? 1u : 0u) | ((u & 0x7F800000u) == 0x7F800000u ? 2u : 0u);
}

struct ConvArgs {
    const __nv_bfloat16* in;    // [B][Cin][H][W]
    const __nv_bfloat16* mask;  // zero `in` where not positive, or NULL
    const __nv_bfloat16* w;     // [Cout][Cin][3][3], or for the data gradient [Cin][Cout][3][3]
    const float* bias;          // [Cout] or NULL
    __nv_bfloat16* out_bf;      // [B][Cout][H][W], or NULL
    float* out_f;               // the same, or NULL
    Image im;
    int Cin, Cout;
    int relu;
    int vec;                    // weight rows start on 16-byte boundaries
    int ksplit;                 // CTAs (one cluster, a power of two) that share the input channels of a tile
    int* err;
    long long wait_ns;
};

// Shared memory of one K block: the pixel planes and the weights.
template <int BN, int MT>
struct ConvTile {
    static constexpr int TM = 128 * MT;
    static constexpr int NACC = MT == 1 ? 4 : 1;  // accumulators that take the products in turn
    static constexpr unsigned COLS = tmem_cols(NACC * MT * BN);
    static __host__ __device__ int seg(int W) { return W + 1 <= TM + 2 ? W + 1 : TM + 2; }  // pixels between taps ky
    static __host__ __device__ int npix(int W) { return TM + 2 + 2 * seg(W); }
    static __host__ __device__ int nplane(int Cin) { return Cin <= 16 ? 2 : KC / 8; }
    static __host__ __device__ size_t stage_bytes(int W, int Cin) {
        return (size_t)16 * nplane(Cin) * (npix(W) + 9 * BN);
    }
    static __host__ size_t smem(int W, int Cin, int ksplit) {
        const int nkb = (Cin + KC - 1) / KC;
        size_t s = (nkb > ksplit ? 2 : 1) * stage_bytes(W, Cin);
        if (s < (size_t)4 * TM * BN) s = (size_t)4 * TM * BN;  // a split's partial sums reuse the stages
        s += 8 * (size_t)((npix(W) + 1) & ~1);
        const size_t least = (size_t)232448 / (512 / COLS + 1) + 16;  // at most 512 / COLS CTAs per SM (tensor memory)
        return s > least ? s : least;
    }
};

// Forward (DGRAD = false) or data gradient (DGRAD = true: `in` is the output gradient, the kernel
// flipped and transposed). One CTA: 128*MT pixels of the padded line x BN output channels, K blocks of
// KC input channels double buffered: while the tensor core works through the nine taps of a block,
// the threads gather the next one. Each tap multiplies 128 x BN x 16 slices, the pixels K-major;
// weights are K-major planes [k / 8][n][k % 8] for the forward pass and MN-major planes
// [n / 8][k][n % 8] for the data gradient, which are the planes that 16-byte pieces of w give without
// a transposition. Where the tiles alone leave SMs idle, a cluster of ksplit CTAs shares a tile's input
// channels and adds the partial sums through its shared memory.
//
// An accumulator loses about 1.1e-8 of the sum with every MMA that it takes in (the products are aligned to it and
// cut off), so a sum of n in a row is off by 1.1e-8 n. One pixel tile per CTA therefore spreads its products
// over four accumulators (channel group x parity of the tap; two for up to 16 channels), added in
// FP32 by the epilogue; two tiles per CTA, which large batches take, have the tensor memory for one.
//
// Bound by the chain of a CTA (about 18 k cycles: weights 3 k, gather 2-5 k, the MMAs' reads of the pixel
// operand, 40 cycles each with 32 channels, epilogue 3 k, or 7-10 k over a cluster), which three CTAs
// per SM overlap (two: 44 us, four: 37 us for the first layer below). Measured on one B200: 16 images of
// 32 -> 32 channels at 128 x 128, forward 32 us and data gradient 36 us (im2col through memory and a
// GEMM: 205 us each); 32 images of 256 -> 256 channels at 4 x 4, forward 13 us, data gradient 13 us.
template <int BN, int MT, bool DGRAD>
__global__ void __launch_bounds__(THREADS, 3) conv_kernel(const ConvArgs a) {
    using T = ConvTile<BN, MT>;
    extern __shared__ __align__(1024) unsigned char conv_smem[];
    __shared__ unsigned long long done[2];
    __shared__ unsigned s_tmem;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int W = a.im.W, Wp = W + 1;
    const size_t hw = (size_t)a.im.H * W;
    const int npix = T::npix(W), seg = T::seg(W), nplane = T::nplane(a.Cin);
    const int n0 = blockIdx.y * BN;
    const long long q0 = (long long)blockIdx.x * T::TM;
    int b0;
    uint32_t r0;
    locate(a.im, q0, b0, r0);
    long long* s_off = reinterpret_cast<long long*>(conv_smem);
    unsigned char* stage0 = conv_smem + 8 * (size_t)((npix + 1) & ~1);
    const size_t stage_bytes = T::stage_bytes(W, a.Cin);
    const size_t bbytes = (size_t)16 * nplane * npix;  // weights follow the pixel planes

    if (threadIdx.x == 0) {
        mbar_init(&done[0], 1);
        mbar_init(&done[1], 1);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&s_tmem, T::COLS);
    for (int s = threadIdx.x; s < npix; s += THREADS) {
        // position s of the tile: the band around it, or segment ky of T::TM + 2 pixels
        int ky = 0, j = s;
        if (seg != Wp) {
            ky = s / seg > 2 ? 2 : s / seg;
            j = s - ky * seg;
        }
        s_off[s] = pixel_offset(a.im, a.Cin, b0, r0, (ky - 1) * Wp - 1 + j);
    }
    tc_fence_before();
    __syncthreads();
    previous_done();
    // not before the allocation: no CTA of a later kernel may hold tensor memory that one of this kernel waits for
    next_may_start();
    const __nv_bfloat16* in = a.in + (size_t)b0 * a.Cin * hw;
    const __nv_bfloat16* mask = a.mask ? a.mask + (size_t)b0 * a.Cin * hw : nullptr;

    // this CTA's K blocks: kb0 + kb, kb < nkb (at least one: ksplit is at most the number of blocks)
    const int kw = 8 * nplane, nkb_all = (a.Cin + kw - 1) / kw;
    const int kb0 = (int)((long long)nkb_all * blockIdx.z / a.ksplit);
    const int nkb = (int)((long long)nkb_all * (blockIdx.z + 1) / a.ksplit) - kb0;
    bool ok = !err_set(a.err);
    for (int kb = 0; kb < nkb; kb++) {
        unsigned char* st = stage0 + (kb & 1) * stage_bytes;
        if (kb >= 2 && ok) ok = mbar_wait(&done[kb & 1], (unsigned)((kb >> 1) - 1) & 1u, a.err, a.wait_ns);
        uint4* wt = reinterpret_cast<uint4*>(st + bbytes);
        for (int e = threadIdx.x; e < nplane * BN; e += THREADS) {
            uint4 v[9];
            if constexpr (!DGRAD) {  // row = output channel, 8 input channels
                const int n = e % BN, p = e / BN;
                weights8(a.w, n0 + n, a.Cout, (kb0 + kb) * kw + 8 * p, a.Cin, a.vec != 0, v);
#pragma unroll
                for (int t = 0; t < 9; t++) wt[(t * nplane + p) * BN + n] = v[t];
            } else {  // row = k (the output gradient's channel), 8 output channels; the flipped tap
                const int k = e % kw, p = e / kw;
                weights8(a.w, (kb0 + kb) * kw + k, a.Cin, n0 + 8 * p, a.Cout, a.vec != 0, v);
#pragma unroll
                for (int t = 0; t < 9; t++) wt[((8 - t) * (BN / 8) + p) * kw + k] = v[t];
            }
        }
        gather({in, mask, hw, a.Cin}, s_off, (kb0 + kb) * kw, nplane, npix, reinterpret_cast<uint4*>(st), [](uint4, int) {});
        fence_proxy_async();
        __syncthreads();
        if (threadIdx.x == 0) {
            tc_fence_after();
            const unsigned tmem = s_tmem;
            constexpr uint32_t id = idesc(128, BN, false, DGRAD);
            const uint32_t da = desc_lo(smem_u32(st), 16u * npix), db = desc_lo(smem_u32(st + bbytes), DGRAD ? 128u : 16u * BN);
            const unsigned bstride = DGRAD ? 16u * kw : 128u;
            const uint32_t btap = DGRAD ? (BN / 8) * kw : nplane * BN;
#pragma unroll 1
            for (int k = 0; k < nplane / 2; k++) {
                const unsigned acc = kb > 0 || (T::NACC == 1 && k > 0);
                const unsigned tmem_k = tmem + (T::NACC == 1 ? 0 : 2 * k * BN);
                const uint32_t dak = da + 2 * k * npix, dbk = db + (DGRAD ? 16 * k : 2 * k * BN);
#pragma unroll
                for (int t = 0; t < 9; t++) {
#pragma unroll
                    for (int m = 0; m < MT; m++)
                        mma_bf16(tmem_k + (T::NACC == 1 ? m * BN : (t & 1) * BN), desc(dak + (t / 3) * seg + (t % 3) + 128 * m, 128u),
                                 desc(dbk + t * btap, bstride), id, acc | (t >= (T::NACC == 1 ? 1 : 2)));
                }
            }
            mma_commit(&done[kb & 1]);
        }
    }
    const unsigned tmem = s_tmem;
    // the last commit covers every MMA issued before it
    mbar_drain(&done[(nkb - 1) & 1], (unsigned)((nkb - 1) >> 1) & 1u);
    tc_fence_after();
    ok = ok && !err_set(a.err);

    // warp: 32 pixels (lanes) of M tile mt, every second 16-column group when both warp groups share one
    const int mt = MT == 2 ? warp / 4 : 0;
    const int row = 128 * mt + 32 * (warp % 4) + lane;
    const int cfirst = MT == 2 ? 0 : 16 * (warp / 4), cstep = MT == 2 ? 16 : 32;
    const unsigned taddr = tmem + ((unsigned)(32 * (warp % 4)) << 16) + (unsigned)(mt * BN);
    // the sum of the accumulators in use, of 16 columns from c0 on
    auto sums = [&](int c0, float (&v)[16]) {
        uint32_t r[16];
        tmem_ld16(taddr + (unsigned)c0, r);
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
        if constexpr (T::NACC > 1) {
#pragma unroll 1
            for (int i = 1; i < nplane; i++) {
                tmem_ld16(taddr + (unsigned)(i * BN + c0), r);
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] += __uint_as_float(r[j]);
            }
        }
    };
    if (a.ksplit == 1) {
        const long long o = pixel_offset(a.im, a.Cout, b0, r0, row);
        const size_t obase = (size_t)b0 * a.Cout * hw + (size_t)(o == kNoPixel ? 0 : o);
#pragma unroll 1
        for (int c0 = cfirst; c0 < BN; c0 += cstep) {
            float bias[16];
#pragma unroll
            for (int j = 0; j < 16; j++) bias[j] = a.bias && n0 + c0 + j < a.Cout ? a.bias[n0 + c0 + j] : 0.0f;
            float v[16];
            sums(c0, v);
            if (o == kNoPixel) continue;
            const size_t at = obase + (size_t)(n0 + c0) * hw;
            const int n = a.Cout - n0 - c0;
#pragma unroll
            for (int j = 0; j < 16; j++) {
                v[j] = (ok ? v[j] : 0.0f) + bias[j];
                if (a.relu) v[j] = fmaxf(v[j], 0.0f);
            }
            if (a.out_bf)
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (j < n) a.out_bf[at + j * hw] = __float2bfloat16_rn(v[j]);
            if (a.out_f)
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (j < n) a.out_f[at + j * hw] = v[j];
        }
    } else {
        // partial sums [n][pixel] of every CTA of the cluster in its own shared memory; CTA z then adds
        // its share of the columns over the cluster in rank order, four pixels at a time
        float* part = reinterpret_cast<float*>(stage0);
#pragma unroll 1
        for (int c0 = cfirst; c0 < BN; c0 += cstep) {
            float v[16];
            sums(c0, v);
#pragma unroll
            for (int j = 0; j < 16; j++) part[(c0 + j) * T::TM + row] = ok ? v[j] : 0.0f;
        }
        cluster_sync();
        const int quads = T::TM / 4, cols = BN / a.ksplit;
        for (int e = threadIdx.x; e < quads * cols; e += THREADS) {
            const int c = blockIdx.z * cols + e / quads, p = 4 * (e % quads), n = n0 + c;
            float4 q[8];
#pragma unroll
            for (int z = 0; z < 8; z++)
                if (z < a.ksplit) q[z] = peer_load4(part + c * T::TM + p, z);
            float v[4] = {q[0].x, q[0].y, q[0].z, q[0].w};
#pragma unroll
            for (int z = 1; z < 8; z++)
                if (z < a.ksplit) v[0] += q[z].x, v[1] += q[z].y, v[2] += q[z].z, v[3] += q[z].w;
            if (n >= a.Cout) continue;
            const float bias = a.bias ? a.bias[n] : 0.0f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const long long o = pixel_offset(a.im, a.Cout, b0, r0, p + j);
                if (o == kNoPixel) continue;
                const size_t at = (size_t)b0 * a.Cout * hw + (size_t)o + n * hw;
                float w = v[j] + bias;
                if (a.relu) w = fmaxf(w, 0.0f);
                if (a.out_bf) a.out_bf[at] = __float2bfloat16_rn(w);
                if (a.out_f) a.out_f[at] = w;
            }
        }
        cluster_sync();  // the peers have read this CTA's sums
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, T::COLS);
    }
}

struct WgradArgs {
    const __nv_bfloat16* in;    // [B][Cin][H][W]
    const __nv_bfloat16* dout;  // [B][Cout][H][W]
    const __nv_bfloat16* mask;  // zero dout where not positive, or NULL
    float* part;                // [split][ky][kx][Cin][Cout32], Cout32 = Cout rounded up to WG_OC
    float* bpart;               // [split][Cout32]
    unsigned* special;          // [split][Cin / 32]: bit per input channel, whether it holds an infinity or NaN
    Image im;
    int Cin, Cout;
    int nblk, blk_per_split;    // K blocks of WG_PIX pixels, and per split
    int* err;
    long long wait_ns;
};

template <int NI>
struct WgradTile {
    static constexpr unsigned COLS = tmem_cols(3 * NI);
    static __host__ __device__ int seg(int W) { return W + 1 <= WG_PIX ? W + 1 : WG_PIX; }
    static __host__ __device__ int npix(int W) { return WG_PIX + 2 * seg(W); }
    // the gradient's three shifted copies (12 planes of WG_PIX pixels), then the input's planes; the MMA's
    // 128 rows reach 4 planes past the copies, into the input's
    static __host__ __device__ size_t stage_bytes(int W) { return (size_t)16 * (12 * WG_PIX + (NI / 8) * npix(W)); }
    static __host__ size_t smem(int W) {
        size_t in = stage_bytes(W) - (size_t)16 * 12 * WG_PIX, pad = 0;
        if (in < (size_t)16 * 4 * WG_PIX) pad = (size_t)16 * 4 * WG_PIX - in;
        const size_t s = 8 * (size_t)(npix(W) + WG_PIX + 2) + 2 * stage_bytes(W) + pad;
        const size_t least = (size_t)232448 / (512 / COLS + 1) + 16;
        return s > least ? s : least;
    }
};

// Weight gradient of WG_OC output channels x NI input channels over a range of pixels: for each ky
// one 128 x NI accumulator whose rows are (kx, o), three copies of the gradient tile shifted by kx
// filling 96 of the MMA's 128 rows, so three MMAs per 16 pixels do the nine taps. Both operands
// are MN-major. The bias gradient is summed from the gathered values (input tile 0). FP32 partial
// sums per split, added in split order by wgrad_finalize_kernel. The zeros between rows and images
// take part in the products, so an infinite or NaN input beside them would reach taps that it has no
// part in: such channels are noted for the split (WgradArgs::special) and their sums taken without the padding.
// 16 images of 32 -> 32 channels at 128 x 128: 55 us with the finalize kernel (transposed im2col, GEMM and
// finalize through memory: 195 us).
template <int NI>
__global__ void __launch_bounds__(THREADS) wgrad_kernel(const WgradArgs a) {
    using T = WgradTile<NI>;
    extern __shared__ __align__(1024) unsigned char conv_smem[];
    __shared__ unsigned long long done[2];
    __shared__ unsigned s_tmem;
    __shared__ float s_bias[THREADS / 32][8];
    __shared__ unsigned s_special[(NI + 31) / 32];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int W = a.im.W, Wp = W + 1;
    const size_t hw = (size_t)a.im.H * W;
    const int npix = T::npix(W), seg = T::seg(W);
    const int i0 = blockIdx.y * NI, o0 = blockIdx.z * WG_OC;
    long long* s_off = reinterpret_cast<long long*>(conv_smem);  // input pixels
    long long* s_goff = s_off + npix;                            // gradient pixels -1 .. WG_PIX
    unsigned char* stage0 = conv_smem + 8 * (size_t)(npix + WG_PIX + 2);
    const size_t stage_bytes = T::stage_bytes(W);
    if (threadIdx.x < (NI + 31) / 32) s_special[threadIdx.x] = 0u;
    if (threadIdx.x == 0) {
        mbar_init(&done[0], 1);
        mbar_init(&done[1], 1);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&s_tmem, T::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = s_tmem;
    previous_done();
    next_may_start();  // after the allocation, as in conv_kernel

    const int blk0 = blockIdx.x * a.blk_per_split;
    const int nb = a.nblk - blk0 < a.blk_per_split ? a.nblk - blk0 : a.blk_per_split;
    bool ok = !err_set(a.err);
    float bsum[8];
#pragma unroll
    for (int j = 0; j < 8; j++) bsum[j] = 0.0f;
    for (int kb = 0; kb < nb; kb++) {
        const long long q0 = (long long)(blk0 + kb) * WG_PIX;
        int b0;
        uint32_t r0;
        locate(a.im, q0, b0, r0);
        for (int s = threadIdx.x; s < npix; s += THREADS) {
            int ky = 0, j = s;
            if (seg != Wp) {
                ky = s / seg > 2 ? 2 : s / seg;
                j = s - ky * seg;
            }
            s_off[s] = pixel_offset(a.im, a.Cin, b0, r0, (ky - 1) * Wp + j);
        }
        for (int s = threadIdx.x; s < WG_PIX + 2; s += THREADS) s_goff[s] = pixel_offset(a.im, a.Cout, b0, r0, s - 1);
        if (kb >= 2 && ok) ok = mbar_wait(&done[kb & 1], (unsigned)((kb >> 1) - 1) & 1u, a.err, a.wait_ns);
        __syncthreads();
        unsigned char* st = stage0 + (kb & 1) * stage_bytes;
        uint4* g = reinterpret_cast<uint4*>(st);
        uint4* xin = g + 12 * WG_PIX;
        // the gradient: thread t always takes plane t / 64, so its sums are of one set of channels
        {
            const int p = threadIdx.x / 64;
            const __nv_bfloat16* d = a.dout + (size_t)b0 * a.Cout * hw;
            const __nv_bfloat16* m = a.mask ? a.mask + (size_t)b0 * a.Cout * hw : nullptr;
            constexpr int U = (WG_PIX + 2 + 63) / 64;
            long long off[U];
            int c[U];
            uint4 gv[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int s = threadIdx.x % 64 + 64 * u;
                off[u] = s < WG_PIX + 2 ? s_goff[s] : kNoPixel;
                c[u] = o0 + 8 * p;
            }
            const Source src{d, m, hw, a.Cout};
            if (a.Cout % 8 == 0) {
                if (m) gather_items<U, true, true>(src, off, c, gv);
                else gather_items<U, true, false>(src, off, c, gv);
            } else {
                if (m) gather_items<U, false, true>(src, off, c, gv);
                else gather_items<U, false, false>(src, off, c, gv);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint4 v = gv[u];
                const int k = threadIdx.x % 64 + 64 * u - 1;  // pixel q0 + k; copy kx holds it at k + kx - 1
#pragma unroll
                for (int kx = 0; kx < 3; kx++) {
                    const int at = k + kx - 1;
                    if (at >= 0 && at < WG_PIX) g[(4 * kx + p) * WG_PIX + at] = v;
                }
                if (k >= 0 && k < WG_PIX) {
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        bsum[2 * j] += __uint_as_float(w[j] << 16);
                        bsum[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u);
                    }
                }
            }
        }
        const __nv_bfloat16* in = a.in + (size_t)b0 * a.Cin * hw;
        gather({in, nullptr, hw, a.Cin}, s_off, i0, NI / 8, npix, xin, [&](uint4 v, int p) {
            const unsigned bits = nonfinite(v.x) | nonfinite(v.y) << 2 | nonfinite(v.z) << 4 | nonfinite(v.w) << 6;
            if (bits) atomicOr(&s_special[p / 4], bits << 8 * (p % 4));
        });
        fence_proxy_async();
        __syncthreads();
        if (threadIdx.x == 0) {
            tc_fence_after();
            constexpr uint32_t id = idesc(128, NI, true, true);
            const uint32_t dg = desc_lo(smem_u32(g), 128u), dx = desc_lo(smem_u32(xin), 128u);
#pragma unroll
            for (int k = 0; k < WG_PIX / 16; k++)
#pragma unroll
                for (int ky = 0; ky < 3; ky++)
                    mma_bf16(tmem + ky * NI, desc(dg + 16 * k, 16u * WG_PIX), desc(dx + ky * seg + 16 * k, 16u * npix), id,
                             k > 0 || kb > 0);
            mma_commit(&done[kb & 1]);
        }
    }
    if (nb > 0) mbar_drain(&done[(nb - 1) & 1], (unsigned)((nb - 1) >> 1) & 1u);
    tc_fence_after();
    ok = ok && nb > 0 && !err_set(a.err);

    const int C32 = (a.Cout + WG_OC - 1) / WG_OC * WG_OC;
    if (warp % 4 < 3) {  // lanes of quadrant kx are its output channels
        const int kx = warp % 4;
#pragma unroll 1
        for (int c0 = 16 * (warp / 4); c0 < 3 * NI; c0 += 32) {
            uint32_t r[16];
            tmem_ld16(tmem + ((unsigned)(32 * kx) << 16) + (unsigned)c0, r);
            const int ky = c0 / NI, i = i0 + c0 % NI;
            float* dst = a.part + ((((size_t)blockIdx.x * 3 + ky) * 3 + kx) * a.Cin + i) * C32 + o0 + lane;
#pragma unroll
            for (int j = 0; j < 16; j++)
                if (i + j < a.Cin) dst[(size_t)j * C32] = ok ? __uint_as_float(r[j]) : 0.0f;
        }
    }
    // the last block's barrier came after every note
    const int words = (a.Cin + 31) / 32, w0 = i0 / 32 + threadIdx.x;
    if (blockIdx.z == 0 && threadIdx.x < (NI + 31) / 32 && w0 < words) a.special[(size_t)blockIdx.x * words + w0] = s_special[threadIdx.x];
    if (blockIdx.y == 0) {
#pragma unroll
        for (int j = 0; j < 8; j++)
            for (int o = 16; o > 0; o >>= 1) bsum[j] += __shfl_down_sync(0xffffffffu, bsum[j], o);
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < 8; j++) s_bias[warp][j] = bsum[j];
        __syncthreads();
        if (threadIdx.x < WG_OC) {
            const int p = threadIdx.x / 8, j = threadIdx.x % 8;  // warps 2p and 2p+1 summed plane p
            a.bpart[(size_t)blockIdx.x * C32 + o0 + threadIdx.x] = s_bias[2 * p][j] + s_bias[2 * p + 1][j];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, T::COLS);
    }
}

// Adds what split k sums for output channel o (a lane's), input channel i and the three taps kx of ky: the
// gradient's pixels q whose input column q + kx - 1 lies in the split's range. Returns true, early, once the sums
// of every lane are NaN.
__device__ __forceinline__ bool direct_sums(const WgradArgs& a, int i, int o, int ky, int k, float (&acc)[3]) {
    const int H = a.im.H, W = a.im.W;
    const long long q0 = (long long)k * a.blk_per_split * WG_PIX, q1 = q0 + (long long)a.blk_per_split * WG_PIX;
    const long long first = q0 > 0 ? q0 - 1 : 0;
    int b, y, x;
    uint32_t r;
    locate(a.im, first, b, r);
    y = (int)(r / (uint32_t)(W + 1));
    x = (int)(r - (uint32_t)y * (uint32_t)(W + 1));
    for (long long q = first; q <= q1 && b < a.im.B; q++) {
        if (y < H && x < W) {
            const int yy = y + ky - 1;
            const bool row = yy >= 0 && yy < H;
            const __nv_bfloat16* xi = a.in + (((size_t)b * a.Cin + i) * H + (row ? yy : 0)) * W;
            const size_t go = (((size_t)b * a.Cout + (o < a.Cout ? o : 0)) * H + y) * W + x;
            float g = __bfloat162float(a.dout[go]);
            if (a.mask && !(__bfloat162float(a.mask[go]) > 0.0f)) g = 0.0f;
#pragma unroll
            for (int t = 0; t < 3; t++) {
                const int xx = x + t - 1;
                // outside the image the input is zero (times an infinite gradient: NaN)
                if (q + t - 1 >= q0 && q + t - 1 < q1)
                    acc[t] = __fmaf_rn(g, row && xx >= 0 && xx < W ? __bfloat162float(xi[xx]) : 0.0f, acc[t]);
            }
            if (__all_sync(0xffffffffu, isnan(acc[0]) && isnan(acc[1]) && isnan(acc[2]))) return true;
        }
        if (++x > W) {
            x = 0;
            if (++y > H) y = 0, b++;
        }
    }
    return false;
}

// dw[o][i][tap] and db[o] from the splits' partial sums: one CTA per (32 output channels, input
// channel, ky); warp v adds splits v, v + 8, ... in order, then the eight warps' sums are added in
// order. The CTA row i = Cin does the bias. Where a split's input channel holds an infinity or NaN, the split's
// sum runs over its image pixels themselves, until every sum of the warp is NaN, which nothing changes
// any more.
__global__ void __launch_bounds__(256) wgrad_finalize_kernel(const WgradArgs a, int splits, float* dw, float* db) {
    __shared__ float s[8][3][32];
    previous_done();
    next_may_start();
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int o = blockIdx.x * 32 + lane, i = blockIdx.y, ky = blockIdx.z, C32 = gridDim.x * 32;
    const bool bias = i == a.Cin;
    if (bias && ky > 0) return;
    float acc[3] = {0.0f, 0.0f, 0.0f};
    const int words = (a.Cin + 31) / 32;
    auto special = [&](int k) { return a.special[(size_t)k * words + i / 32] >> (i % 32) & 1u; };
    unsigned any = 0;
    float first = 0.0f;
    const float* p = a.part + ((size_t)(3 * ky) * a.Cin + i) * C32 + o;
    const size_t tap = (size_t)a.Cin * C32, split = 9 * tap;
    if (bias) {
        for (int k = warp; k < splits; k += 8) acc[0] += a.bpart[(size_t)k * C32 + o];
    } else {
        for (int k = threadIdx.x; k < splits; k += 256) any |= special(k);
        // the line's first pixel meets the zero before it in no split: nothing, or NaN for an infinite gradient
        if (warp == 0 && o < a.Cout) {
            const size_t go = (size_t)o * a.im.H * a.im.W;
            if (!a.mask || __bfloat162float(a.mask[go]) > 0.0f) first = __bfloat162float(a.dout[go]) * 0.0f;
        }
#pragma unroll 4
        for (int k = warp; k < splits; k += 8)
#pragma unroll
            for (int t = 0; t < 3; t++) acc[t] += p[k * split + t * tap];
    }
    if (__syncthreads_or((int)any)) {
        float sum[3] = {0.0f, 0.0f, 0.0f};
        bool nan = false;
        for (int k = warp; k < splits && !nan; k += 8) {
            if (special(k)) {
                nan = direct_sums(a, i, o, ky, k, sum);
            } else {
#pragma unroll
                for (int t = 0; t < 3; t++) sum[t] += p[k * split + t * tap];
            }
        }
#pragma unroll
        for (int t = 0; t < 3; t++) acc[t] = sum[t];
    }
    acc[0] += first;
#pragma unroll
    for (int t = 0; t < 3; t++) s[warp][t][lane] = acc[t];
    __syncthreads();
    const int nt = bias ? 1 : 3;
    for (int e = threadIdx.x; e < 32 * nt; e += 256) {
        const int l = e / nt, t = e % nt;
        float v = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; k++) v += s[k][t][l];
        const int oo = blockIdx.x * 32 + l;
        if (oo < a.Cout) {
            if (bias) db[oo] = v;
            else dw[((size_t)oo * a.Cin + i) * 9 + 3 * ky + t] = v;
        }
    }
}

}  // namespace conv
}  // namespace mtb
