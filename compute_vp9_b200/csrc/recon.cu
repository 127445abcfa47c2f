/*
 * recon.cu — VP9 reconstruction kernels for sm_100a.
 *
 * Three launches per batch of frames (one frame from each of J streams):
 *
 *   k_scan_blocks   one thread per block: superblock (SB) membership, the
 *                   contiguous block range of every SB, layout checks.
 *   k_recon<A>      one CTA per SB ticket, tickets handed out in
 *                   SB-diagonal order across all streams of the batch. A CTA
 *                   predicts its SB's inter blocks and transforms every
 *                   residual, then waits (bounded) for the left / above /
 *                   above-left SBs whose samples its intra blocks read, and
 *                   predicts those level by level, four samples a thread.
 *                   The SB tile (with a one-pixel halo) lives in shared
 *                   memory; its right column and bottom row are written
 *                   first, the SB's done flag released, then the tile.
 *   k_loopfilter<A> the 4-tap deblock on 64x64 luma tiles shifted by 4 px so
 *                   every filter tap of every 8-px edge falls inside one tile
 *                   (horizontal pass then vertical pass, in place), with the
 *                   NV12 pack fused into the same tile pass.
 *
 * Arithmetic profiles (template A):
 *   CVP9_ARITH_REFCPU reproduces src/decoder/vp9_reconstruct.c:194-370
 *     bit for bit: float64 inverse DCT of the raw coefficients with the
 *     host-built basis (separately rounded products and sums, k ascending),
 *     bilinear MC, the CPU's 127 edge rules, luma-only residual.
 *   CVP9_ARITH_SPEC reproduces the shader arithmetic: dequantised integer
 *     butterflies (vp9_idct.comp.glsl), regular 8-tap MC (vp9_mc.comp.glsl)
 *     on luma and chroma, intra with the shader's availability rules
 *     (vp9_intra_pred.comp.glsl), the residual of every TX of every plane.
 *
 * No tensor cores: every sample is integer-exact and nothing here is a dense
 * contraction; the kernels are bound by memory traffic and dependency
 * latency.
 */
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "recon_job.h"
#include "vp9_tables.h"
#include "recon_launch.h"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxBlocks = 128;      /* blocks per SB (the tile parser emits at most 64) */
constexpr int kCoefStage = 6144;     /* int16 coefficients staged per SB (64x64 luma + chroma) */
constexpr int kYPitch = 72;          /* luma tile row pitch; x = 0 at byte 4 */
constexpr int kCPitch = 40;          /* chroma tile row pitch; x = 0 at byte 4 */
constexpr int kTyBytes = (65 * kYPitch + 15) / 16 * 16;
constexpr int kTcBytes = (33 * kCPitch + 15) / 16 * 16;
/* Looks at a flag before a wait gives up, and what one takes (measured, ns):
 * superblocks' flags (wait_flag) 0.9 s in all, the loop filter's rows
 * (wait_at_least) 1.1 s, its counts in shared memory (lf_wait) 2.1 s: who waits
 * for these waits for a thread that may itself be waiting for a row. */
constexpr int kFlagLooks = 1 << 22, kRowLooks = 1 << 21, kShmLooks = 1 << 24;
constexpr double kFlagLookNs = 213, kRowLookNs = 512, kShmLookNs = 128;
static_assert(kShmLooks * kShmLookNs > 1.5 * kRowLooks * kRowLookNs && kFlagLooks * kFlagLookNs > 0.5e9,
              "an inner wait outlasts the one it depends on; none gives up within half a second");

__constant__ double c_dct[16 + 64 + 256 + 1024];      /* N = 4, 8, 16, 32 */
/* The basis again in global memory: lane-varying reads are served by L1
 * instead of being serialised by the constant cache. */
__device__ __align__(16) double g_dct[16 + 64 + 256 + 1024];
__constant__ uint8_t c_tx_type[10] = CVP9_INTRA_TX_TYPE_INIT;
/* the regular filter's taps as signed bytes, taps 0-3 and 4-7 in two words, for dp4a
 * (phase 0's 128 does not fit a byte: callers take the centre sample for
 * it, which is what its filter computes); uploaded by cvp9k_configure */
__constant__ uint32_t c_subpel_pk[16][2];
/* the four VP9 filters (interp_filter 0..3) packed the same way, for the FULL profile */
__constant__ uint32_t c_subpel4_pk[4][16][2];

/* Wait for the kernel before, in a chain launched with programmatic
 * dependencies (a no-op otherwise): every kernel of such a chain starts with
 * it, so that its CTAs may be placed while the one before drains. */
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

/* Saturated and packed, the first in the low bits: one instruction for two
 * values, where clamping and shifting them in takes five. */
__device__ __forceinline__ uint32_t pack4_u8(int a, int b, int c, int d)
{
    uint32_t hi, r;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(b), "r"(a), "r"(hi));
    return r;
}
__device__ __forceinline__ uint32_t pack2_s16(int a, int b)
{
    uint32_t r;
    asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(r) : "r"(b), "r"(a));
    return r;
}
__device__ __forceinline__ uint32_t min2_s16(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("min.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t max2_s16(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("max.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
/* two 10-bit samples */
__device__ __forceinline__ uint32_t pack2_u10(int a, int b)
{
    return max2_s16(min2_s16(pack2_s16(a, b), 0x03ff03ffu), 0u);
}

__device__ __forceinline__ int dp4a_su(uint32_t taps, uint32_t px, int c)
{
    int d;
    asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(taps), "r"(px), "r"(c));
    return d;
}

/* One 8-tap output from samples s0 (samples 0-3 of the window) and s1 (4-7),
 * not clamped to a sample yet; phase 0 is the centre sample itself. */
__device__ __forceinline__ int tap8(uint32_t ta, uint32_t tb, int phase, uint32_t s0, uint32_t s1)
{
    return phase ? dp4a_su(tb, s1, dp4a_su(ta, s0, 64)) >> 7 : (int)(s0 >> 24);
}

/* t / d for 0 <= t < 4096 and 1 <= d <= 16 without an integer divide:
 * (t * ceil(2^16 / d)) >> 16 is exact in that range. */
__device__ __forceinline__ int div_small(int t, int d)
{
    return (int)(((unsigned)t * ((65536u + (unsigned)d - 1u) / (unsigned)d)) >> 16);
}

/* ── Asynchronous global -> shared copies (16 bytes, both sides aligned) ── */

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

/* 8 and 4 bytes (both sides aligned to the size) */
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem)
{
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" :: "r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem)
{
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(sa), "l"(gmem) : "memory");
}
/* all but the newest group have landed */
__device__ __forceinline__ void cp_async_wait_prev() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }


/* ── 32-bit wrap-around integer for the shader butterflies ───────────────── */
struct wi {
    using P = wi;           /* the type of a product with a Q14 multiplier */
    int v;
    __device__ __forceinline__ wi() : v(0) {}
    __device__ __forceinline__ wi(int x) : v(x) {}
};
__device__ __forceinline__ wi operator+(wi a, wi b) { return wi((int)((unsigned)a.v + (unsigned)b.v)); }
__device__ __forceinline__ wi operator-(wi a, wi b) { return wi((int)((unsigned)a.v - (unsigned)b.v)); }
__device__ __forceinline__ wi operator-(wi a) { return wi((int)(0u - (unsigned)a.v)); }
__device__ __forceinline__ wi operator*(wi a, int k) { return wi((int)((unsigned)a.v * (unsigned)k)); }
__device__ __forceinline__ wi RS(wi x) { return wi(((int)((unsigned)x.v + 8192u)) >> 14); }
__device__ __forceinline__ wi shr(wi x, int k) { return wi(x.v >> k); }

/* 64-bit integer for the same butterflies at 10 bits (profile 2): products
 * of the +-2^17 dequantised range and the Q14 multipliers need 64 bits. */
struct wl {
    using P = wl;
    long long v;
    __device__ __forceinline__ wl() : v(0) {}
    __device__ __forceinline__ wl(long long x) : v(x) {}
};
__device__ __forceinline__ wl operator+(wl a, wl b) { return wl(a.v + b.v); }
__device__ __forceinline__ wl operator-(wl a, wl b) { return wl(a.v - b.v); }
__device__ __forceinline__ wl operator-(wl a) { return wl(-a.v); }
__device__ __forceinline__ wl operator*(wl a, int k) { return wl(a.v * (long long)k); }
__device__ __forceinline__ wl RS(wl x) { return wl((x.v + 8192) >> 14); }
__device__ __forceinline__ wl shr(wl x, int k) { return wl(x.v >> k); }

/* The same butterflies on values known to fit 32 bits: 32-bit values, 64-bit
 * products and sums of products (one IMAD.WIDE a multiplier), one funnel
 * shift to round back. Every value a butterfly forms is a sum of its inputs
 * with factors below 2, so a 32-point row of |inputs| < 2^18 and the column
 * after it stay below 2^30: the results are wl's. */
struct wp {
    long long v;
    __device__ __forceinline__ wp() : v(0) {}
    __device__ __forceinline__ wp(long long x) : v(x) {}
};
struct wn {
    using P = wp;
    int v;
    __device__ __forceinline__ wn() : v(0) {}
    __device__ __forceinline__ wn(int x) : v(x) {}
};
__device__ __forceinline__ wp operator+(wp a, wp b) { return wp(a.v + b.v); }
__device__ __forceinline__ wp operator-(wp a, wp b) { return wp(a.v - b.v); }
__device__ __forceinline__ wp operator-(wp a) { return wp(-a.v); }
__device__ __forceinline__ wn operator+(wn a, wn b) { return wn(a.v + b.v); }
__device__ __forceinline__ wn operator-(wn a, wn b) { return wn(a.v - b.v); }
__device__ __forceinline__ wn operator-(wn a) { return wn(-a.v); }
__device__ __forceinline__ wp operator*(wn a, int k) { return wp((long long)a.v * k); }
__device__ __forceinline__ wn RS(wp x) { return wn((int)((x.v + 8192) >> 14)); }
__device__ __forceinline__ wn shr(wn x, int k) { return wn(x.v >> k); }

/* cos(k*pi/64) in Q14 */
enum : int {
    K1 = 16364, K2 = 16305, K3 = 16207, K4 = 16069, K5 = 15893, K6 = 15679,
    K7 = 15426, K8 = 15137, K9 = 14811, K10 = 14449, K11 = 14053, K12 = 13623,
    K13 = 13160, K14 = 12665, K15 = 12140, K16 = 11585, K17 = 11003, K18 = 10394,
    K19 = 9760, K20 = 9102, K21 = 8423, K22 = 7723, K23 = 7005, K24 = 6270,
    K25 = 5520, K26 = 4756, K27 = 3981, K28 = 3196, K29 = 2404, K30 = 1606,
    K31 = 804
};

/* 1-D inverse DCTs, in place on x[0..N). Same stage structure and rounding
 * as vp9_idct.comp.glsl:47-649. */
template <class T>
__device__ __forceinline__ void idct4(T *x)
{
    T s0 = RS((x[0] + x[2]) * K16), s1 = RS((x[0] - x[2]) * K16);
    T s2 = RS(x[1] * K24 - x[3] * K8), s3 = RS(x[1] * K8 + x[3] * K24);
    x[0] = s0 + s3; x[1] = s1 + s2; x[2] = s1 - s2; x[3] = s0 - s3;
}

template <class T>
__device__ __forceinline__ void idct8(T *x)
{
    T a[8], b[8];
    a[0] = x[0]; a[1] = x[2]; a[2] = x[4]; a[3] = x[6];
    a[4] = RS(x[1] * K28 - x[7] * K4); a[7] = RS(x[1] * K4 + x[7] * K28);
    a[5] = RS(x[5] * K12 - x[3] * K20); a[6] = RS(x[5] * K20 + x[3] * K12);
    b[0] = RS((a[0] + a[2]) * K16); b[1] = RS((a[0] - a[2]) * K16);
    b[2] = RS(a[1] * K24 - a[3] * K8); b[3] = RS(a[1] * K8 + a[3] * K24);
    b[4] = a[4] + a[5]; b[5] = a[4] - a[5]; b[6] = -a[6] + a[7]; b[7] = a[6] + a[7];
    a[0] = b[0] + b[3]; a[1] = b[1] + b[2]; a[2] = b[1] - b[2]; a[3] = b[0] - b[3];
    a[4] = b[4]; a[5] = RS((b[6] - b[5]) * K16); a[6] = RS((b[5] + b[6]) * K16); a[7] = b[7];
#pragma unroll
    for (int i = 0; i < 4; i++) { x[i] = a[i] + a[7 - i]; x[7 - i] = a[i] - a[7 - i]; }
}

template <class T>
__device__ __forceinline__ void idct16(T *x)
{
    T a[16], b[16];
    a[0] = x[0]; a[1] = x[8]; a[2] = x[4]; a[3] = x[12]; a[4] = x[2]; a[5] = x[10];
    a[6] = x[6]; a[7] = x[14]; a[8] = x[1]; a[9] = x[9]; a[10] = x[5]; a[11] = x[13];
    a[12] = x[3]; a[13] = x[11]; a[14] = x[7]; a[15] = x[15];
#pragma unroll
    for (int i = 0; i < 8; i++) b[i] = a[i];
    b[8] = RS(a[8] * K30 - a[15] * K2);   b[15] = RS(a[8] * K2 + a[15] * K30);
    b[9] = RS(a[9] * K14 - a[14] * K18);  b[14] = RS(a[9] * K18 + a[14] * K14);
    b[10] = RS(a[10] * K22 - a[13] * K10); b[13] = RS(a[10] * K10 + a[13] * K22);
    b[11] = RS(a[11] * K6 - a[12] * K26);  b[12] = RS(a[11] * K26 + a[12] * K6);
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = b[i];
    a[4] = RS(b[4] * K28 - b[7] * K4); a[7] = RS(b[4] * K4 + b[7] * K28);
    a[5] = RS(b[5] * K12 - b[6] * K20); a[6] = RS(b[5] * K20 + b[6] * K12);
    a[8] = b[8] + b[9]; a[9] = b[8] - b[9]; a[10] = -b[10] + b[11]; a[11] = b[10] + b[11];
    a[12] = b[12] + b[13]; a[13] = b[12] - b[13]; a[14] = -b[14] + b[15]; a[15] = b[14] + b[15];
    b[0] = RS((a[0] + a[1]) * K16); b[1] = RS((a[0] - a[1]) * K16);
    b[2] = RS(a[2] * K24 - a[3] * K8); b[3] = RS(a[2] * K8 + a[3] * K24);
    b[4] = a[4] + a[5]; b[5] = a[4] - a[5]; b[6] = -a[6] + a[7]; b[7] = a[6] + a[7];
    b[8] = a[8]; b[15] = a[15];
    b[9] = RS(-a[9] * K8 + a[14] * K24);   b[14] = RS(a[9] * K24 + a[14] * K8);
    b[10] = RS(-a[10] * K24 - a[13] * K8); b[13] = RS(-a[10] * K8 + a[13] * K24);
    b[11] = a[11]; b[12] = a[12];
    a[0] = b[0] + b[3]; a[1] = b[1] + b[2]; a[2] = b[1] - b[2]; a[3] = b[0] - b[3];
    a[4] = b[4]; a[5] = RS((b[6] - b[5]) * K16); a[6] = RS((b[5] + b[6]) * K16); a[7] = b[7];
    a[8] = b[8] + b[11]; a[9] = b[9] + b[10]; a[10] = b[9] - b[10]; a[11] = b[8] - b[11];
    a[12] = -b[12] + b[15]; a[13] = -b[13] + b[14]; a[14] = b[13] + b[14]; a[15] = b[12] + b[15];
#pragma unroll
    for (int i = 0; i < 4; i++) { b[i] = a[i] + a[7 - i]; b[7 - i] = a[i] - a[7 - i]; }
    b[8] = a[8]; b[9] = a[9];
    b[10] = RS((-a[10] + a[13]) * K16); b[13] = RS((a[10] + a[13]) * K16);
    b[11] = RS((-a[11] + a[12]) * K16); b[12] = RS((a[11] + a[12]) * K16);
    b[14] = a[14]; b[15] = a[15];
#pragma unroll
    for (int i = 0; i < 8; i++) { x[i] = b[i] + b[15 - i]; x[15 - i] = b[i] - b[15 - i]; }
}

template <class T>
__device__ __forceinline__ void idct32(T *x)
{
    T a[32], b[32];
    a[0] = x[0]; a[1] = x[16]; a[2] = x[8]; a[3] = x[24]; a[4] = x[4]; a[5] = x[20];
    a[6] = x[12]; a[7] = x[28]; a[8] = x[2]; a[9] = x[18]; a[10] = x[10]; a[11] = x[26];
    a[12] = x[6]; a[13] = x[22]; a[14] = x[14]; a[15] = x[30];
    a[16] = RS(x[1] * K31 - x[31] * K1);  a[31] = RS(x[1] * K1 + x[31] * K31);
    a[17] = RS(x[17] * K15 - x[15] * K17); a[30] = RS(x[17] * K17 + x[15] * K15);
    a[18] = RS(x[9] * K23 - x[23] * K9);  a[29] = RS(x[9] * K9 + x[23] * K23);
    a[19] = RS(x[25] * K7 - x[7] * K25);  a[28] = RS(x[25] * K25 + x[7] * K7);
    a[20] = RS(x[5] * K27 - x[27] * K5);  a[27] = RS(x[5] * K5 + x[27] * K27);
    a[21] = RS(x[21] * K11 - x[11] * K21); a[26] = RS(x[21] * K21 + x[11] * K11);
    a[22] = RS(x[13] * K19 - x[19] * K13); a[25] = RS(x[13] * K13 + x[19] * K19);
    a[23] = RS(x[29] * K3 - x[3] * K29);  a[24] = RS(x[29] * K29 + x[3] * K3);
    /* stage 2 */
#pragma unroll
    for (int i = 0; i < 8; i++) b[i] = a[i];
    b[8] = RS(a[8] * K30 - a[15] * K2);   b[15] = RS(a[8] * K2 + a[15] * K30);
    b[9] = RS(a[9] * K14 - a[14] * K18);  b[14] = RS(a[9] * K18 + a[14] * K14);
    b[10] = RS(a[10] * K22 - a[13] * K10); b[13] = RS(a[10] * K10 + a[13] * K22);
    b[11] = RS(a[11] * K6 - a[12] * K26);  b[12] = RS(a[11] * K26 + a[12] * K6);
#pragma unroll
    for (int i = 16; i < 32; i += 4) {
        b[i] = a[i] + a[i + 1]; b[i + 1] = a[i] - a[i + 1];
        b[i + 2] = -a[i + 2] + a[i + 3]; b[i + 3] = a[i + 2] + a[i + 3];
    }
    /* stage 3 */
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = b[i];
    a[4] = RS(b[4] * K28 - b[7] * K4); a[7] = RS(b[4] * K4 + b[7] * K28);
    a[5] = RS(b[5] * K12 - b[6] * K20); a[6] = RS(b[5] * K20 + b[6] * K12);
#pragma unroll
    for (int i = 8; i < 16; i += 4) {
        a[i] = b[i] + b[i + 1]; a[i + 1] = b[i] - b[i + 1];
        a[i + 2] = -b[i + 2] + b[i + 3]; a[i + 3] = b[i + 2] + b[i + 3];
    }
    a[16] = b[16]; a[31] = b[31];
    a[17] = RS(-b[17] * K4 + b[30] * K28);  a[30] = RS(b[17] * K28 + b[30] * K4);
    a[18] = RS(-b[18] * K28 - b[29] * K4);  a[29] = RS(-b[18] * K4 + b[29] * K28);
    a[19] = b[19]; a[20] = b[20];
    a[21] = RS(-b[21] * K20 + b[26] * K12); a[26] = RS(b[21] * K12 + b[26] * K20);
    a[22] = RS(-b[22] * K12 - b[25] * K20); a[25] = RS(-b[22] * K20 + b[25] * K12);
    a[23] = b[23]; a[24] = b[24]; a[27] = b[27]; a[28] = b[28];
    /* stage 4 */
    b[0] = RS((a[0] + a[1]) * K16); b[1] = RS((a[0] - a[1]) * K16);
    b[2] = RS(a[2] * K24 - a[3] * K8); b[3] = RS(a[2] * K8 + a[3] * K24);
    b[4] = a[4] + a[5]; b[5] = a[4] - a[5]; b[6] = -a[6] + a[7]; b[7] = a[6] + a[7];
    b[8] = a[8]; b[15] = a[15];
    b[9] = RS(-a[9] * K8 + a[14] * K24);   b[14] = RS(a[9] * K24 + a[14] * K8);
    b[10] = RS(-a[10] * K24 - a[13] * K8); b[13] = RS(-a[10] * K8 + a[13] * K24);
    b[11] = a[11]; b[12] = a[12];
#pragma unroll
    for (int i = 16; i < 32; i += 8) {
        b[i] = a[i] + a[i + 3]; b[i + 1] = a[i + 1] + a[i + 2];
        b[i + 2] = a[i + 1] - a[i + 2]; b[i + 3] = a[i] - a[i + 3];
        b[i + 4] = -a[i + 4] + a[i + 7]; b[i + 5] = -a[i + 5] + a[i + 6];
        b[i + 6] = a[i + 5] + a[i + 6]; b[i + 7] = a[i + 4] + a[i + 7];
    }
    /* stage 5 */
    a[0] = b[0] + b[3]; a[1] = b[1] + b[2]; a[2] = b[1] - b[2]; a[3] = b[0] - b[3];
    a[4] = b[4]; a[5] = RS((b[6] - b[5]) * K16); a[6] = RS((b[5] + b[6]) * K16); a[7] = b[7];
    a[8] = b[8] + b[11]; a[9] = b[9] + b[10]; a[10] = b[9] - b[10]; a[11] = b[8] - b[11];
    a[12] = -b[12] + b[15]; a[13] = -b[13] + b[14]; a[14] = b[13] + b[14]; a[15] = b[12] + b[15];
    a[16] = b[16]; a[17] = b[17];
    a[18] = RS(-b[18] * K8 + b[29] * K24);  a[29] = RS(b[18] * K24 + b[29] * K8);
    a[19] = RS(-b[19] * K8 + b[28] * K24);  a[28] = RS(b[19] * K24 + b[28] * K8);
    a[20] = RS(-b[20] * K24 - b[27] * K8);  a[27] = RS(-b[20] * K8 + b[27] * K24);
    a[21] = RS(-b[21] * K24 - b[26] * K8);  a[26] = RS(-b[21] * K8 + b[26] * K24);
    a[22] = b[22]; a[23] = b[23]; a[24] = b[24]; a[25] = b[25]; a[30] = b[30]; a[31] = b[31];
    /* stage 6 */
#pragma unroll
    for (int i = 0; i < 4; i++) { b[i] = a[i] + a[7 - i]; b[7 - i] = a[i] - a[7 - i]; }
    b[8] = a[8]; b[9] = a[9];
    b[10] = RS((-a[10] + a[13]) * K16); b[13] = RS((a[10] + a[13]) * K16);
    b[11] = RS((-a[11] + a[12]) * K16); b[12] = RS((a[11] + a[12]) * K16);
    b[14] = a[14]; b[15] = a[15];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        b[16 + i] = a[16 + i] + a[23 - i]; b[23 - i] = a[16 + i] - a[23 - i];
        b[24 + i] = -a[24 + i] + a[31 - i]; b[31 - i] = a[24 + i] + a[31 - i];
    }
    /* stage 7 */
#pragma unroll
    for (int i = 0; i < 8; i++) { a[i] = b[i] + b[15 - i]; a[15 - i] = b[i] - b[15 - i]; }
#pragma unroll
    for (int i = 16; i < 20; i++) a[i] = b[i];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        a[20 + i] = RS((-b[20 + i] + b[27 - i]) * K16);
        a[27 - i] = RS((b[20 + i] + b[27 - i]) * K16);
    }
#pragma unroll
    for (int i = 28; i < 32; i++) a[i] = b[i];
    /* output */
#pragma unroll
    for (int i = 0; i < 16; i++) { x[i] = a[i] + a[31 - i]; x[31 - i] = a[i] - a[31 - i]; }
}

/* ── Shared-memory layout of one reconstruction CTA ─────────────────────── */

struct BlkS {
    uint8_t  x, y;          /* local luma position in the SB               */
    uint8_t  w, h;          /* coded size                                  */
    uint8_t  cw, ch;        /* size clamped to the frame                   */
    uint8_t  txl;           /* luma tx_size 0..3                           */
    uint8_t  flags;         /* 1 intra, 2 skip                             */
    uint8_t  ymode, uvmode;
    uint8_t  ref0;
    uint8_t  ptxl[3];       /* residual TX log2-4 per plane                */
    uint8_t  pnx[3], pny[3];    /* residual TXs per row and column, per plane */
    uint8_t  ref1;          /* FULL: second reference of a compound block  */
    int16_t  mvx, mvy;
    int16_t  mv1x, mv1y;    /* FULL: its MV                                */
    uint32_t coeff;
};
/* BlkS.flags: 1 intra, 2 skip */

/* ── Intra wavefront inside a superblock ─────────────────────────────────
 *
 * What bounds a picture with intra blocks is a serial chain: a block is
 * predicted from reconstructed samples around it, so a superblock waits for
 * its neighbours and its blocks for one another. Everything that does not
 * read those samples is taken off the chain: the inverse transforms of the
 * intra blocks run at once, before the superblock waits, into a grid of
 * residuals, and so do its inter blocks. What is left per step of the chain
 * is "predict four samples, add their residual": the unit of prediction
 * (REFCPU, SPEC: a block's plane; FULL: a transform block) is a task, a
 * task's level is one more than the deepest task whose samples it reads, and
 * a level's samples, four in a row a thread, go out over the whole CTA with
 * one barrier after them, whatever the sizes of its tasks. The last sample
 * of each four-sample group is also kept column by column (`col`), so that a
 * left edge is read along contiguous addresses, and edges that a picture or
 * tile boundary takes away are filled into the halo once, so that the
 * prediction has no cases for them.
 * Measured (one B200), against a warp per block with transform and
 * prediction in turn and the inter blocks after the wait: 16x1080p REFCPU
 * key step with its download 3.77 -> 2.43 ms, three FULL 1080p pictures (one
 * key) 21.5 -> 2.95 ms, a step of 24 1366x768 REFCPU inter pictures with 5%
 * intra blocks 2.2 -> 0.92 ms (with the steps noted further down). */

struct ITask {           /* four words, read as one 16-byte load            */
    uint32_t xywh;       /* plane position in the SB tile; samples written   */
    uint32_t edge;       /* plane | mode << 2; last sample read of the row
                          * above, of the left column (later ones repeat it);
                          * DC: 1 counts the row above, 2 the left column    */
    uint32_t area;       /* edge lengths: the TX size (FULL), the predicted
                          * area (others: samples past it keep the tile's,
                          * the residual of a SPEC sub-8x8 block covers its
                          * whole MI)                                        */
    uint32_t inv;        /* DC: ceil(2^32 / samples counted); 0: one sample  */
    __device__ __forceinline__ int x() const { return (int)(xywh & 255u); }
    __device__ __forceinline__ int y() const { return (int)((xywh >> 8) & 255u); }
    __device__ __forceinline__ int w() const { return (int)((xywh >> 16) & 255u); }
    __device__ __forceinline__ int h() const { return (int)(xywh >> 24); }
    __device__ __forceinline__ int plane() const { return (int)(edge & 3u); }
    __device__ __forceinline__ int mode() const { return (int)((edge >> 2) & 63u); }
    __device__ __forceinline__ int acl() const { return (int)((edge >> 8) & 255u); }
    __device__ __forceinline__ int lcl() const { return (int)((edge >> 16) & 255u); }
    __device__ __forceinline__ unsigned avail() const { return edge >> 24; }
    __device__ __forceinline__ int pw() const { return (int)(area & 255u); }
    __device__ __forceinline__ int ph() const { return (int)(area >> 8); }
};

__device__ __forceinline__ ITask ld_task(const uint4 *t)
{
    const uint4 w = *t;
    return ITask{ w.x, w.y, w.z, w.w };
}

__device__ __forceinline__ void st_task(uint4 *t, int x, int y, int w, int h, int plane, int mode, int acl, int lcl,
                                        int avail, int pw, int ph, uint32_t inv)
{
    *t = make_uint4((uint32_t)(x | y << 8 | w << 16) | (uint32_t)h << 24,
                    (uint32_t)(plane | mode << 2 | acl << 8 | lcl << 16) | (uint32_t)avail << 24,
                    (uint32_t)(pw | ph << 8), inv);
}

constexpr int kMaxTasks = 384;       /* 4x4 TXs of an SB's three planes; 3 x kMaxBlocks */
constexpr uint32_t kNoQuad = 0xFFFFFFFFu;
constexpr int kResidGrid = 64 * 64 + 2 * 32 * 32;
constexpr int kMaxQuads = 2048;      /* 16 a luma row, at most 16 a chroma row */
/* A level's kind of quads fills its last warp in part, and there are no more
 * of those than tasks; full warps hold 8 (kind 2) or 32 quads. */
constexpr int kMaxJobs = kMaxTasks + kMaxQuads / 8;

struct IntraWork {
    uint2    qtab[kMaxQuads];        /* quads by level and kind (quad_word)  */
    uint32_t job[kMaxJobs];          /* a warp's quads: first | count - 1 << 11 | kind << 16 */
    uint32_t lvlq[kMaxTasks][2];     /* quads of each level and kind, then the first of each: 16 bits a kind */
    uint16_t lvlj[kMaxTasks + 1];    /* first job of each level              */
    uint4    task[kMaxTasks];        /* ITask                                */
    uint16_t lvl[kMaxTasks];
    uint16_t qat[kMaxTasks];         /* a task's first quad in its level     */
    uint16_t own[kMaxTasks];         /* FULL: task + 1 owning each 4x4 cell (luma 256, U 64, V 64);
                                      * others: task of each block's luma, 0xFFFF none */
    uint32_t prow[3][16], pcol[3][16];   /* intra_levels: cells still open, by row and by column */
    int      ntask, nlev;
};

/* A superblock's tile for the intra tasks. The planes of the tile, and the
 * left columns (luma before x = 4k at [k * 64 + y], chroma before x = 2k at
 * [k * 32 + y]), lie at fixed distances, so that a plane is an offset and not
 * a pointer picked from an array (which would go through local memory). */
template <class T>
struct IntraView {
    static constexpr int kU = sizeof(T) == 1 ? kTyBytes + kCPitch - kYPitch : 65 * kYPitch + kCPitch - kYPitch;
    static constexpr int kUV = sizeof(T) == 1 ? kTcBytes : 33 * kCPitch;
    T *tile0, *col0;                 /* luma sample (0, 0); column 0          */
    const int16_t *res;              /* residuals: 64x64 luma, 32x32 U, V    */
    __device__ __forceinline__ T *tile(int p) const { return tile0 + (p ? kU + (p - 1) * kUV : 0); }
    __device__ __forceinline__ T *col(int p) const { return col0 + (p ? 16 * 64 + (p - 1) * 16 * 32 : 0); }
};

struct ReconSmem {
    union {
        uint8_t   mc[kWarps * 4 * 608];          /* REFCPU: windows of the chunks in flight */
        int32_t   tx[kWarps][32 * 32];           /* SPEC, FULL: a warp's TXs between the passes */
        IntraWork w;                             /* then the intra tasks        */
    } temp;
    /* tiles, contiguous and 16-byte sized so they fill with vector stores */
    uint8_t  ty[kTyBytes];                       /* luma tile, row 0 = halo     */
    uint8_t  tu[kTcBytes];
    uint8_t  tv[kTcBytes];
    int16_t  coef[kCoefStage];                   /* the SB's coefficient span   */
    int16_t  res[kResidGrid];                    /* residuals of intra blocks   */
    cvp9_job_t jc;                               /* this ticket's job           */
    BlkS     blk[kMaxBlocks];
    uint8_t  cell[256];                          /* owner block + 1 per 4x4     */
    uint32_t rows[16];                           /* claimed cells, a bit each   */
    uint16_t first[kMaxBlocks];                  /* FULL: a block's first task  */
    uint16_t chunk_off[kMaxBlocks + 1];          /* inter chunks before a block */
    uint16_t tx_at[3][kMaxBlocks];               /* first TX of a block's plane in tx */
    uint8_t  chunk_blk[256];                     /* chunk -> block              */
    uint2    tx[kMaxTasks];                      /* residual TXs by size (TxRef) */
    int      ntx[4];                             /* TXs of each size            */
    uint8_t  col[16 * 64 + 2 * 16 * 32];         /* left-column copies (IntraView) */
    int      scan_tmp[2 * kWarps];
    unsigned c_lo, c_hi;                         /* coefficient span of the SB  */
    unsigned needs;                              /* intra_needs of its blocks   */
    int      ticket;
};

static_assert(sizeof(ReconSmem) <= 75 * 1024, "three CTAs per SM");

__device__ __forceinline__ uint8_t &TY(ReconSmem &s, int x, int y) { return s.ty[(y + 1) * kYPitch + x + 4]; }
__device__ __forceinline__ uint8_t &TC(ReconSmem &s, int p, int x, int y)
{
    return (p == 1 ? s.tu : s.tv)[(y + 1) * kCPitch + x + 4];
}

__device__ __forceinline__ int max_tx_for(int w, int h)
{
    int m = w < h ? w : h;
    return m >= 32 ? 3 : (m >= 16 ? 2 : (m >= 8 ? 1 : 0));
}

/* The tile parser's TX layout of one plane of a block (vp9_kf_tile.c:
 * 320-396): TX size, TXs per row and per column over the coded area clipped
 * at the MI-aligned frame edge, and the plane block width (sub-8x8 blocks
 * code a whole 8x8, chroma at least 4x4). */
template <class B>
__device__ __forceinline__ void plane_layout(const B &b, const cvp9_job_t &job, int gx, int gy, int p,
                                             int &tx, int &nx, int &ny, int &pbw)
{
    int sub8 = b.w < 8 || b.h < 8;
    int ew = sub8 ? 8 : b.w, eh = sub8 ? 8 : b.h;
    int mi_col = gx >> 3, mi_row = gy >> 3;
    int ss = p > 0;
    int pw = ss ? ew / 2 : ew, ph = ss ? eh / 2 : eh;
    pw = pw < 4 ? 4 : pw;
    ph = ph < 4 ? 4 : ph;
    tx = b.txl;
    if (ss) { int mt = max_tx_for(pw, ph); tx = sub8 ? 0 : (tx > mt ? mt : tx); }
    int t4 = 1 << tx;
    int o4x = (mi_col * 2) >> ss, o4y = (mi_row * 2) >> ss;
    int mw = pw / 4, mh = ph / 4;
    int lim_w = ((job.mi_cols * 2) >> ss) - o4x, lim_h = ((job.mi_rows * 2) >> ss) - o4y;
    if (mw > lim_w) mw = lim_w;
    if (mh > lim_h) mh = lim_h;
    nx = mw > 0 ? (mw + t4 - 1) >> tx : 0;
    ny = mh > 0 ? (mh + t4 - 1) >> tx : 0;
    pbw = pw;
}

/* Residual TX layout of one block (plane TX size, TXs per row and column).
 * REFCPU: luma only, counts from the frame-clamped size
 * (vp9_reconstruct.c:336-347). SPEC, FULL: every plane as plane_layout has it. */
template <int A>
__device__ __forceinline__ void residual_layout(BlkS &b, const cvp9_job_t &job, int gx, int gy)
{
    b.pnx[0] = b.pnx[1] = b.pnx[2] = 0;
    b.pny[0] = b.pny[1] = b.pny[2] = 0;
    b.ptxl[0] = b.ptxl[1] = b.ptxl[2] = 0;
    if (b.flags & 2) return;
    if (A == CVP9_ARITH_REFCPU) {
        const int nx = b.cw >> (2 + b.txl), ny = b.ch >> (2 + b.txl);
        b.ptxl[0] = b.txl;
        b.pnx[0] = (uint8_t)nx;
        b.pny[0] = (uint8_t)ny;
    } else {
        for (int p = 0; p < 3; p++) {
            int tx, nx, ny, pbw;
            plane_layout(b, job, gx, gy, p, tx, nx, ny, pbw);
            b.ptxl[p] = (uint8_t)tx;
            b.pnx[p] = (uint8_t)nx;
            b.pny[p] = (uint8_t)ny;
        }
    }
}

__device__ __forceinline__ int mc_chunks(int cw, int ch, int ccw, int cch);

/* Inter chunks of a block: REFCPU an 8x8 of luma with its chroma, the others
 * of one plane each (mc_chunks). */
template <int A>
__device__ __forceinline__ int block_chunks(const BlkS &b)
{
    return A == CVP9_ARITH_REFCPU ? ((b.cw + 7) >> 3) * ((b.ch + 7) >> 3)
                                  : mc_chunks(b.cw, b.ch, (b.cw + 1) >> 1, (b.ch + 1) >> 1);
}

/* 4x4 byte transpose: rows a..d (one word of four columns each) to four
 * words, one column each (its bytes in row order) */
__device__ __forceinline__ void tr4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t col[4])
{
    const uint32_t x0 = __byte_perm(a, b, 0x5140), x1 = __byte_perm(a, b, 0x7362);
    const uint32_t y0 = __byte_perm(c, d, 0x5140), y1 = __byte_perm(c, d, 0x7362);
    col[0] = __byte_perm(x0, y0, 0x5410);
    col[1] = __byte_perm(x0, y0, 0x7632);
    col[2] = __byte_perm(x1, y1, 0x5410);
    col[3] = __byte_perm(x1, y1, 0x7632);
}

/* ── 8-tap inter prediction, eight lanes a chunk (SPEC, FULL, 10-bit) ─────
 *
 * A chunk is up to 8x8 samples of one plane of an inter block. Lane k of its
 * eight runs the horizontal pass on rows k and k + 8 of the (h + 7)-row
 * window — a row comes as a few 8-byte loads, shifted into place, and a
 * sample is two dp4a (8 bits) or four dp2a (16 bits) — into shared rows, then
 * the vertical pass of output row k, the window's rows transposed by byte
 * permutes. Both passes round and clip, as vp9_mc.comp.glsl:61-110 does;
 * every fetch is clamped into the reference plane. What bounded this was
 * instructions and L1 requests, not bytes: a warp per chunk with a load per
 * sample took 50 k cycles a superblock (8 bits, SPEC), a load per tap and
 * sample 75 k (10 bits), this 21 k and 42 k. Samples are clamped and packed by
 * cvt.pack and stay packed, also where two predictions are averaged: of 29 k
 * cycles a superblock that took 4 k (FULL). */
template <class T> struct McRow;

template <> struct McRow<uint8_t> {
    static constexpr int kWords = 4, kLoads = 3;      /* 16 samples; 15 + 7 bytes */
    static constexpr uint32_t kOne = 0x01010101u;     /* 1 in every sample of a word */
    /* 8 outputs of the horizontal pass, packed as two words */
    static __device__ __forceinline__ void filter(const uint32_t (&w)[4], int f, uint32_t ta, uint32_t tb, uint8_t *d)
    {
        uint32_t *o = reinterpret_cast<uint32_t *>(d);
        if (f == 0) {
            o[0] = __funnelshift_r(w[0], w[1], 24);
            o[1] = __funnelshift_r(w[1], w[2], 24);
            return;
        }
        uint32_t s[12];
#pragma unroll
        for (int c = 0; c < 12; c++) s[c] = (c & 3) ? __funnelshift_r(w[c >> 2], w[(c >> 2) + 1], 8 * (c & 3)) : w[c >> 2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            int r[4];
#pragma unroll
            for (int c = 0; c < 4; c++) r[c] = dp4a_su(tb, s[4 * h + c + 4], dp4a_su(ta, s[4 * h + c], 64)) >> 7;
            o[h] = pack4_u8(r[0], r[1], r[2], r[3]);
        }
    }
    /* output row, packed, from the 8 rows at h (8 samples each) */
    static __device__ __forceinline__ void down(const uint8_t *h, int f, uint32_t ta, uint32_t tb, uint32_t (&v)[2])
    {
        const uint2 *r = reinterpret_cast<const uint2 *>(h);
        if (f == 0) {
            const uint2 m = r[3];
            v[0] = m.x;
            v[1] = m.y;
            return;
        }
        uint2 a[8];
#pragma unroll
        for (int t = 0; t < 8; t++) a[t] = r[t];
#pragma unroll
        for (int s = 0; s < 2; s++) {
            uint32_t lo[4], hi[4];
            tr4(s ? a[0].y : a[0].x, s ? a[1].y : a[1].x, s ? a[2].y : a[2].x, s ? a[3].y : a[3].x, lo);
            tr4(s ? a[4].y : a[4].x, s ? a[5].y : a[5].x, s ? a[6].y : a[6].x, s ? a[7].y : a[7].x, hi);
            int u[4];
#pragma unroll
            for (int c = 0; c < 4; c++) u[c] = dp4a_su(tb, hi[c], dp4a_su(ta, lo[c], 64)) >> 7;
            v[s] = pack4_u8(u[0], u[1], u[2], u[3]);
        }
    }
};

/* Two 10-bit samples (signed halves hold them) with taps 0-1 or 2-3 of a word. */
__device__ __forceinline__ int dp2a_lo_ss(uint32_t px, uint32_t taps, int c)
{
    int d;
    asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(px), "r"(taps), "r"(c));
    return d;
}
__device__ __forceinline__ int dp2a_hi_ss(uint32_t px, uint32_t taps, int c)
{
    int d;
    asm("dp2a.hi.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(px), "r"(taps), "r"(c));
    return d;
}

template <> struct McRow<uint16_t> {
    static constexpr int kWords = 8, kLoads = 5;      /* 16 samples; 30 + 6 bytes */
    static constexpr uint32_t kOne = 0x00010001u;
    static __device__ __forceinline__ int tap(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t ta, uint32_t tb)
    {
        return dp2a_hi_ss(d, tb, dp2a_lo_ss(c, tb, dp2a_hi_ss(b, ta, dp2a_lo_ss(a, ta, 64)))) >> 7;
    }
    static __device__ __forceinline__ void filter(const uint32_t (&w)[8], int f, uint32_t ta, uint32_t tb, uint16_t *d)
    {
        uint4 *o = reinterpret_cast<uint4 *>(d);
        uint32_t s[7];                                /* the words one sample on */
#pragma unroll
        for (int i = 0; i < 7; i++) s[i] = __funnelshift_r(w[i], w[i + 1], 16);
        if (f == 0) {
            *o = make_uint4(s[1], s[2], s[3], s[4]);
            return;
        }
        uint32_t r[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            r[i] = pack2_u10(tap(w[i], w[i + 1], w[i + 2], w[i + 3], ta, tb), tap(s[i], s[i + 1], s[i + 2], s[i + 3], ta, tb));
        *o = make_uint4(r[0], r[1], r[2], r[3]);
    }
    static __device__ __forceinline__ void down(const uint16_t *h, int f, uint32_t ta, uint32_t tb, uint32_t (&v)[4])
    {
        const uint4 *r = reinterpret_cast<const uint4 *>(h);
        if (f == 0) {
            const uint4 m = r[3];
            v[0] = m.x; v[1] = m.y; v[2] = m.z; v[3] = m.w;
            return;
        }
        int acc[8];
#pragma unroll
        for (int c = 0; c < 8; c++) acc[c] = 64;
#pragma unroll
        for (int t = 0; t < 4; t++) {                 /* rows 2t and 2t + 1 side by side */
            const uint4 a = r[2 * t], b = r[2 * t + 1];
            const uint32_t x[4] = { a.x, a.y, a.z, a.w }, y[4] = { b.x, b.y, b.z, b.w };
            const uint32_t tp = t < 2 ? ta : tb;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t e = __byte_perm(x[i], y[i], 0x5410), o = __byte_perm(x[i], y[i], 0x7632);
                acc[2 * i] = t & 1 ? dp2a_hi_ss(e, tp, acc[2 * i]) : dp2a_lo_ss(e, tp, acc[2 * i]);
                acc[2 * i + 1] = t & 1 ? dp2a_hi_ss(o, tp, acc[2 * i + 1]) : dp2a_lo_ss(o, tp, acc[2 * i + 1]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = pack2_u10(acc[2 * i] >> 7, acc[2 * i + 1] >> 7);
    }
};

/* 16 samples of a reference row from column X (the last may be beyond the
 * window), as words. */
template <class T>
__device__ __forceinline__ void mc_load(const T *row, int X, int pw, uint32_t (&w)[McRow<T>::kWords])
{
    constexpr int kW = McRow<T>::kWords, kL = McRow<T>::kLoads, kPer = 4 / (int)sizeof(T);
    const uintptr_t at = (uintptr_t)(row + X);
    /* every byte read is the row's, which may begin anywhere: the loads begin
     * up to 7 bytes before sample X and end up to 8 after the 16 */
    if (X * (int)sizeof(T) >= (int)(at & 7) && X + 16 + 8 / (int)sizeof(T) <= pw) {
        const uint2 *q = reinterpret_cast<const uint2 *>(at & ~(uintptr_t)7);
        uint32_t u[2 * kL];
#pragma unroll
        for (int i = 0; i < kL; i++) {
            const uint2 x = __ldg(q + i);
            u[2 * i] = x.x;
            u[2 * i + 1] = x.y;
        }
        const unsigned sh = 8u * (unsigned)(at & 3);
        const bool odd = at & 4;
        /* one word on when the row starts in the upper half of its 8 bytes */
#pragma unroll
        for (int i = 0; i < 2 * kL - 1; i++) u[i] = odd ? u[i + 1] : u[i];
#pragma unroll
        for (int i = 0; i < kW; i++) w[i] = __funnelshift_r(u[i], i + 1 < 2 * kL ? u[i + 1] : 0u, sh);
    } else {
        const int xm = pw > 0 ? pw - 1 : 0;
#pragma unroll
        for (int i = 0; i < kW; i++) {
            uint32_t x = 0;
#pragma unroll
            for (int j = 0; j < kPer; j++)
                x |= (uint32_t)__ldg(row + clampi(X + i * kPer + j, 0, xm)) << (8 * (int)sizeof(T) * j);
            w[i] = x;
        }
    }
}

/* A chunk's part of one reference: its window's origin and phases. */
struct McRef {
    const void *plane;
    int pw, ph, X, Y, fx, fy;
};

template <class T>
__device__ __forceinline__ McRef mc_ref(const cvp9_ref_t &R, int p, int gx, int gy, int mvx, int mvy)
{
    McRef m;
    const T *q = reinterpret_cast<const T *>(R.plane);
    m.pw = R.w;
    m.ph = R.h;
    if (p) {
        m.pw = (R.w + 1) >> 1;
        m.ph = (R.h + 1) >> 1;
        q += (size_t)R.w * R.h + (p == 2 ? (size_t)m.pw * m.ph : 0);
    }
    m.plane = q;
    m.X = gx + (p ? mvx >> 4 : mvx >> 3) - 3;
    m.Y = gy + (p ? mvy >> 4 : mvy >> 3) - 3;
    m.fx = p ? mvx & 15 : (mvx & 7) << 1;
    m.fy = p ? mvy & 15 : (mvy & 7) << 1;
    return m;
}

/* One chunk by lane k of its eight (`on`: they have one; all lanes of the
 * warp call it): 8 samples of row k of a w x h chunk at (lx, ly) of plane p
 * into the tile row `dst`. rows: the group's 15 rows of 8 samples in shared
 * memory, 16-byte aligned. A missing first reference predicts `mid`, a missing
 * second one leaves the single prediction. */
template <class T, bool COMPOUND, class B>
__device__ __forceinline__ void mc_chunk(const cvp9_job_t &job, const uint32_t (*P)[2], const B &b, bool on, int p, int gx,
                                         int gy, int w, int h, int mid, T *rows, T *dst, int k)
{
    constexpr int kV = 2 * (int)sizeof(T), kPer = 4 / (int)sizeof(T);
    uint32_t v[kV];                    /* the row's samples, packed            */
#pragma unroll
    for (int c = 0; c < kV; c++) v[c] = (uint32_t)mid * McRow<T>::kOne;
#pragma unroll 1
    for (int q = 0; q < (COMPOUND ? 2 : 1); q++) {
        const int rf = on ? (q ? b.ref1 : b.ref0) : 0;
        if (q && !__any_sync(0xffffffffu, on && rf != 0)) break;
        const cvp9_ref_t &R = job.ref[job.ref_slot_of[clampi(rf - 1, 0, 2)] & 7];
        on = on && R.plane;
        const bool go = on && (q == 0 || rf != 0);
        McRef m;
        if (go) {
            m = mc_ref<T>(R, p, gx, gy, q ? b.mv1x : b.mvx, q ? b.mv1y : b.mvy);
            const uint32_t ta = P[m.fx][0], tb = P[m.fx][1];
            const int ym = m.ph > 0 ? m.ph - 1 : 0;
            for (int j = k; j < h + 7; j += 8) {
                uint32_t x[McRow<T>::kWords];
                mc_load<T>((const T *)m.plane + (size_t)clampi(m.Y + j, 0, ym) * m.pw, m.X, m.pw, x);
                McRow<T>::filter(x, m.fx, ta, tb, rows + j * 8);
            }
        }
        __syncwarp();
        if (go && k < h) {
            uint32_t u[kV];
            McRow<T>::down(rows + k * 8, m.fy, P[m.fy][0], P[m.fy][1], u);
            /* (a + b + 1) >> 1 of each sample: a | b less half of a ^ b, no bit crossing into the next */
            constexpr uint32_t half = ~(McRow<T>::kOne << (8 * sizeof(T) - 1));
#pragma unroll
            for (int c = 0; c < kV; c++) v[c] = q ? (v[c] | u[c]) - (((v[c] ^ u[c]) >> 1) & half) : u[c];
        }
        __syncwarp();
    }
    if (k < h) {
        if (w == 8 && !((uintptr_t)dst & 3)) {
            uint32_t *d = reinterpret_cast<uint32_t *>(dst);
#pragma unroll
            for (int c = 0; c < kV; c++) d[c] = v[c];
        } else {
#pragma unroll
            for (int c = 0; c < 8; c++)
                if (c < w) dst[c] = (T)(v[c / kPer] >> (8 * (int)sizeof(T) * (c & (kPer - 1))));
        }
    }
}

/* A block's chunks: luma, then U, then V, raster of 8x8 each. */
__device__ __forceinline__ int mc_chunks(int cw, int ch, int ccw, int cch)
{
    return ((cw + 7) >> 3) * ((ch + 7) >> 3) + 2 * ((ccw + 7) >> 3) * ((cch + 7) >> 3);
}

/* Chunk i of them: plane, position in the block, size. */
__device__ __forceinline__ void mc_chunk_at(int i, int cw, int ch, int ccw, int cch, int &p, int &x, int &y, int &w, int &h)
{
    const int nl = ((cw + 7) >> 3) * ((ch + 7) >> 3), nc = ((ccw + 7) >> 3) * ((cch + 7) >> 3);
    p = i < nl ? 0 : (i < nl + nc ? 1 : 2);
    i -= p == 0 ? 0 : nl + (p - 1) * nc;
    const int bw = p ? ccw : cw, bh = p ? cch : ch, nx = (bw + 7) >> 3;
    const int r = div_small(i, nx);
    x = (i - r * nx) * 8;
    y = r * 8;
    w = min(8, bw - x);
    h = min(8, bh - y);
}

/* Geometry of one chunk's REFCPU bilinear prediction: integer positions and
 * fractions of the luma and chroma windows (vp9_reconstruct.c:94-131,
 * :313-327) and whether each window can be staged with aligned 16-byte
 * copies (inside its plane, rows 16-byte aligned). */
struct McGeo {
    const uint8_t *rp, *ru, *rv;
    int rw, rh, rcs;
    int ix, iy, fx, fy, cix, ciy, cfx, cfy, la, ca;
    bool lfast, cfast;
};

__device__ __forceinline__ bool refcpu_geo(const ReconSmem &s, const BlkS &b, int sbx, int sby,
                                           int lx0, int ly0, int lw, int lh, int cx0, int cy0,
                                           int clw, int clh, McGeo &g)
{
    const int slot = (int)b.ref0 - 1;
    if (slot < 0 || slot >= 8 || !s.jc.ref[slot].plane) return false;
    const cvp9_ref_t &R = s.jc.ref[slot];
    g.rp = R.plane;
    g.rw = R.w;
    g.rh = R.h;
    g.rcs = (g.rw + 1) >> 1;
    g.ru = g.rp + (size_t)g.rw * g.rh;
    g.rv = g.ru + (size_t)g.rcs * ((g.rh + 1) >> 1);
    const int px8 = (sbx + lx0) * 8 + b.mvx, py8 = (sby + ly0) * 8 + b.mvy;
    g.ix = px8 >> 3; g.iy = py8 >> 3; g.fx = px8 & 7; g.fy = py8 & 7;
    const int cmx = b.mvx / 2, cmy = b.mvy / 2;            /* halves toward zero */
    const int cpx8 = ((sbx >> 1) + cx0) * 8 + cmx, cpy8 = ((sby >> 1) + cy0) * 8 + cmy;
    g.cix = cpx8 >> 3; g.ciy = cpy8 >> 3; g.cfx = cpx8 & 7; g.cfy = cpy8 & 7;
    const int crw = g.rw >> 1, crh = g.rh >> 1;            /* floor half of the ref size */
    const bool aligned = !(g.rw & 15) && !(g.rcs & 15) && !((uintptr_t)g.rp & 15) &&
                         !((uintptr_t)g.ru & 15) && !((uintptr_t)g.rv & 15);
    g.lfast = aligned && g.ix >= 0 && g.iy >= 0 && g.ix + lw < g.rw && g.iy + lh < g.rh;
    g.cfast = aligned && g.cix >= 0 && g.ciy >= 0 && g.cix + clw < crw && g.ciy + clh < crh;
    g.la = g.ix & ~15;
    g.ca = g.cix & ~15;
    return true;
}

/* Stage layout of one chunk (608 bytes): luma rows at 32-byte pitch, then U
 * and V rows. Rows needing bytes past the first 16 take a second copy. */
constexpr int kChunkStage = 608;

/* Lane-group variants: 8 lanes per chunk (k = lane & 7). Issue: the group's
 * lanes share the chunk's window copies. Compute: lane k produces luma row k
 * (up to 8 samples) and, for k < 4 / k >= 4, row k&3 of U / V. */
__device__ __forceinline__ void refcpu_issue8(uint8_t *st, const McGeo &g, int lw, int lh,
                                              int clw, int clh, int k)
{
    if (g.lfast) {
        const int two = (g.ix - g.la) + lw >= 16;
        for (int j = k; j < 2 * (lh + 1); j += 8) {
            const int row = j >> 1, half = j & 1;
            if (half == 0 || two)
                cp_async16(st + row * 32 + half * 16, g.rp + (size_t)(g.iy + row) * g.rw + g.la + half * 16);
        }
    }
    if (g.cfast) {
        const int two = (g.cix - g.ca) + clw >= 16;
        const int per = 2 * (clh + 1);
        for (int j = k; j < 2 * per; j += 8) {
            const int pl = j >= per, jj = j - pl * per, row = jj >> 1, half = jj & 1;
            if (half == 0 || two)
                cp_async16(st + 288 + pl * 160 + row * 32 + half * 16,
                           (pl ? g.rv : g.ru) + (size_t)(g.ciy + row) * g.rcs + g.ca + half * 16);
        }
    }
}

/* nine consecutive bytes of a staged row starting at byte `off`, from three
 * aligned 32-bit shared-memory words */
__device__ __forceinline__ void row9(const uint8_t *row, int off, unsigned v[9])
{
    const uint32_t *w = reinterpret_cast<const uint32_t *>(row) + (off >> 2);
    const unsigned sh = 8u * (unsigned)(off & 3);
    const unsigned w0 = w[0], w1 = w[1], w2 = w[2];
    const unsigned lo = __funnelshift_r(w0, w1, sh), mid = __funnelshift_r(w1, w2, sh), hi = w2 >> sh;
#pragma unroll
    for (int i = 0; i < 4; i++) { v[i] = (lo >> (8 * i)) & 0xffu; v[4 + i] = (mid >> (8 * i)) & 0xffu; }
    v[8] = hi & 0xffu;
}

__device__ __forceinline__ void refcpu_compute8(ReconSmem &s, const uint8_t *st, const McGeo &g,
                                                int lx0, int ly0, int lw, int lh,
                                                int cx0, int cy0, int clw, int clh, int k)
{
    if (k < lh) {
        unsigned a[9], b[9];
        if (g.lfast) {
            row9(st + k * 32, g.ix - g.la, a);
            row9(st + (k + 1) * 32, g.ix - g.la, b);
        } else {
            const int y0 = clampi(g.iy + k, 0, g.rh - 1), y1 = clampi(g.iy + k + 1, 0, g.rh - 1);
            const uint8_t *r0 = g.rp + (size_t)y0 * g.rw, *r1 = g.rp + (size_t)y1 * g.rw;
#pragma unroll
            for (int c = 0; c < 9; c++) {
                const int x = clampi(g.ix + c, 0, g.rw - 1);
                a[c] = __ldg(r0 + x);
                b[c] = __ldg(r1 + x);
            }
        }
        const unsigned wx = 8 - g.fx, wy = 8 - g.fy;
        unsigned out[8];
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const unsigned t = (a[c] * wx + a[c + 1] * g.fx + 4) >> 3;
            const unsigned u = (b[c] * wx + b[c + 1] * g.fx + 4) >> 3;
            out[c] = (t * wy + u * g.fy + 4) >> 3;
        }
        uint8_t *d = &TY(s, lx0, ly0 + k);
        if (lw == 8) {
            uint32_t *d4 = reinterpret_cast<uint32_t *>(d);
            d4[0] = out[0] | out[1] << 8 | out[2] << 16 | out[3] << 24;
            d4[1] = out[4] | out[5] << 8 | out[6] << 16 | out[7] << 24;
        } else {
#pragma unroll
            for (int c = 0; c < 8; c++) if (c < lw) d[c] = (uint8_t)out[c];
        }
    }
    {
        const int p = 1 + (k >> 2), r = k & 3;
        if (r < clh) {
            unsigned a[5], b[5];
            if (g.cfast) {
                const uint8_t *s0 = st + 288 + (p - 1) * 160 + r * 32 + (g.cix - g.ca), *s1 = s0 + 32;
#pragma unroll
                for (int c = 0; c < 5; c++) { a[c] = s0[c]; b[c] = s1[c]; }
            } else {
                const int crw = g.rw >> 1, crh = g.rh >> 1;
                const int xm = crw > 0 ? crw - 1 : 0, ym = crh > 0 ? crh - 1 : 0;
                const uint8_t *pl = p == 1 ? g.ru : g.rv;
                const uint8_t *r0 = pl + (size_t)clampi(g.ciy + r, 0, ym) * g.rcs;
                const uint8_t *r1 = pl + (size_t)clampi(g.ciy + r + 1, 0, ym) * g.rcs;
#pragma unroll
                for (int c = 0; c < 5; c++) {
                    const int x = clampi(g.cix + c, 0, xm);
                    a[c] = __ldg(r0 + x);
                    b[c] = __ldg(r1 + x);
                }
            }
            uint8_t *d = &TC(s, p, cx0, cy0 + r);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (c >= clw) break;
                const unsigned t = (a[c] * (8 - g.cfx) + a[c + 1] * g.cfx + 4) >> 3;
                const unsigned u = (b[c] * (8 - g.cfx) + b[c + 1] * g.cfx + 4) >> 3;
                d[c] = (uint8_t)((t * (8 - g.cfy) + u * g.cfy + 4) >> 3);
            }
        }
    }
}

/* Lane-group flat fill (missing reference): lane k fills luma row k and one
 * chroma row, like refcpu_compute8. */
__device__ __forceinline__ void refcpu_fill8(ReconSmem &s, int v, int lx0, int ly0, int lw, int lh,
                                             int cx0, int cy0, int clw, int clh, int k)
{
    if (k < lh)
        for (int c = 0; c < lw; c++) TY(s, lx0 + c, ly0 + k) = (uint8_t)v;
    const int p = 1 + (k >> 2), r = k & 3;
    if (r < clh)
        for (int c = 0; c < clw; c++) TC(s, p, cx0 + c, cy0 + r) = (uint8_t)v;
}

/* ── Residual ──────────────────────────────────────────────────────────── */

template <class T>
__device__ __forceinline__ void idct_n(T *x, int n)
{
    if (n == 4) idct4(x);
    else if (n == 8) idct8(x);
    else if (n == 16) idct16(x);
    else idct32(x);
}

/* ── FULL profile: ADST and WHT, rows-then-columns residual, per-TX intra ── */

/* sin(k*pi/9) * 2/3 * sqrt(2) in Q14, the 4-point ADST multipliers */
enum : int { KS1 = 5283, KS2 = 9929, KS3 = 13377, KS4 = 15212 };

/* 1-D inverse ADSTs in place, 32-bit wrap and Q14 rounding as the DCTs. */
template <class T>
__device__ __forceinline__ void iadst4(T *x)
{
    using P = typename T::P;
    P a = x[0] * KS1 + x[2] * KS4 + x[3] * KS2;
    P b = x[0] * KS2 - x[2] * KS1 - x[3] * KS4;
    P c = (x[0] - x[2] + x[3]) * KS3;
    P d = x[1] * KS3;
    x[0] = RS(a + d); x[1] = RS(b + d); x[2] = RS(c); x[3] = RS(a + b - d);
}

template <class T>
__device__ __forceinline__ void rot(T x, T y, int ca, int cb, typename T::P &o0, typename T::P &o1)
{
    o0 = x * ca + y * cb;
    o1 = x * cb - y * ca;
}

template <class T>
__device__ __forceinline__ void iadst8(T *in)
{
    T x0 = in[7], x1 = in[0], x2 = in[5], x3 = in[2], x4 = in[3], x5 = in[4], x6 = in[1], x7 = in[6];
    typename T::P s0, s1, s2, s3, s4, s5, s6, s7;
    rot(x0, x1, K2, K30, s0, s1);
    rot(x2, x3, K10, K22, s2, s3);
    rot(x4, x5, K18, K14, s4, s5);
    rot(x6, x7, K26, K6, s6, s7);
    x0 = RS(s0 + s4); x1 = RS(s1 + s5); x2 = RS(s2 + s6); x3 = RS(s3 + s7);
    x4 = RS(s0 - s4); x5 = RS(s1 - s5); x6 = RS(s2 - s6); x7 = RS(s3 - s7);
    s4 = x4 * K8 + x5 * K24;
    s5 = x4 * K24 - x5 * K8;
    s6 = x7 * K8 - x6 * K24;
    s7 = x6 * K8 + x7 * K24;
    T u0 = x0 + x2, u1 = x1 + x3, u2 = x0 - x2, u3 = x1 - x3;
    x4 = RS(s4 + s6); x5 = RS(s5 + s7); x6 = RS(s4 - s6); x7 = RS(s5 - s7);
    x2 = RS((u2 + u3) * K16);
    x3 = RS((u2 - u3) * K16);
    T y6 = RS((x6 + x7) * K16), y7 = RS((x6 - x7) * K16);
    in[0] = u0; in[1] = -x4; in[2] = y6; in[3] = -x2;
    in[4] = x3; in[5] = -y7; in[6] = x5; in[7] = -u1;
}

template <class T>
__device__ __forceinline__ void iadst16(T *in)
{
    T x[16], u[16];
    typename T::P s[16];
    x[0] = in[15]; x[1] = in[0]; x[2] = in[13]; x[3] = in[2]; x[4] = in[11]; x[5] = in[4];
    x[6] = in[9]; x[7] = in[6]; x[8] = in[7]; x[9] = in[8]; x[10] = in[5]; x[11] = in[10];
    x[12] = in[3]; x[13] = in[12]; x[14] = in[1]; x[15] = in[14];
    rot(x[0], x[1], K1, K31, s[0], s[1]);
    rot(x[2], x[3], K5, K27, s[2], s[3]);
    rot(x[4], x[5], K9, K23, s[4], s[5]);
    rot(x[6], x[7], K13, K19, s[6], s[7]);
    rot(x[8], x[9], K17, K15, s[8], s[9]);
    rot(x[10], x[11], K21, K11, s[10], s[11]);
    rot(x[12], x[13], K25, K7, s[12], s[13]);
    rot(x[14], x[15], K29, K3, s[14], s[15]);
#pragma unroll
    for (int k = 0; k < 8; k++) { x[k] = RS(s[k] + s[k + 8]); x[k + 8] = RS(s[k] - s[k + 8]); }
#pragma unroll
    for (int k = 0; k < 8; k++) u[k] = x[k];
    s[8] = x[8] * K4 + x[9] * K28;
    s[9] = x[8] * K28 - x[9] * K4;
    s[10] = x[10] * K20 + x[11] * K12;
    s[11] = x[10] * K12 - x[11] * K20;
    s[12] = x[13] * K4 - x[12] * K28;
    s[13] = x[12] * K4 + x[13] * K28;
    s[14] = x[15] * K20 - x[14] * K12;
    s[15] = x[14] * K20 + x[15] * K12;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        x[k] = u[k] + u[k + 4];
        x[k + 4] = u[k] - u[k + 4];
        x[k + 8] = RS(s[k + 8] + s[k + 12]);
        x[k + 12] = RS(s[k + 8] - s[k + 12]);
    }
#pragma unroll
    for (int g = 0; g < 16; g += 8) {
        u[g + 0] = x[g + 0]; u[g + 1] = x[g + 1]; u[g + 2] = x[g + 2]; u[g + 3] = x[g + 3];
        s[g + 4] = x[g + 4] * K8 + x[g + 5] * K24;
        s[g + 5] = x[g + 4] * K24 - x[g + 5] * K8;
        s[g + 6] = x[g + 7] * K8 - x[g + 6] * K24;
        s[g + 7] = x[g + 6] * K8 + x[g + 7] * K24;
        x[g + 0] = u[g + 0] + u[g + 2];
        x[g + 1] = u[g + 1] + u[g + 3];
        x[g + 2] = u[g + 0] - u[g + 2];
        x[g + 3] = u[g + 1] - u[g + 3];
        x[g + 4] = RS(s[g + 4] + s[g + 6]);
        x[g + 5] = RS(s[g + 5] + s[g + 7]);
        x[g + 6] = RS(s[g + 4] - s[g + 6]);
        x[g + 7] = RS(s[g + 5] - s[g + 7]);
    }
    T t2 = RS(-((x[2] + x[3]) * K16)), t3 = RS((x[2] - x[3]) * K16);
    T t6 = RS((x[6] + x[7]) * K16), t7 = RS((x[7] - x[6]) * K16);
    T t10 = RS((x[10] + x[11]) * K16), t11 = RS((x[11] - x[10]) * K16);
    T t14 = RS(-((x[14] + x[15]) * K16)), t15 = RS((x[14] - x[15]) * K16);
    in[0] = x[0];  in[1] = -x[8];  in[2] = x[12];  in[3] = -x[4];
    in[4] = t6;    in[5] = t14;    in[6] = t10;    in[7] = t2;
    in[8] = t3;    in[9] = t11;    in[10] = t15;   in[11] = t7;
    in[12] = x[5]; in[13] = -x[13]; in[14] = x[9]; in[15] = -x[1];
}

/* 4-point inverse Walsh-Hadamard (lossless frames); the row pass first
 * undoes the quantiser step 4 with a shift. */
template <class T>
__device__ __forceinline__ void iwht4(T *x, bool rows)
{
    T a = x[0], c = x[1], d = x[2], b = x[3];
    if (rows) { a = shr(a, 2); c = shr(c, 2); d = shr(d, 2); b = shr(b, 2); }
    a = a + c; d = d - b;
    T e = shr(a - d, 1);
    b = e - b; c = e - c;
    a = a - b; d = d + c;
    x[0] = a; x[1] = b; x[2] = c; x[3] = d;
}

template <int N, class T>
__device__ __forceinline__ void itx1(T *v, bool adst)
{
    if (N == 4 && adst) iadst4(v);
    else if (N == 8 && adst) iadst8(v);
    else if (N == 16 && adst) iadst16(v);
    else idct_n(v, N);
}

/* First MI column of the tile column holding mi_col (VP9 tile offsets). */
__device__ __forceinline__ int full_tile_start(int mi_col, int mi_cols, int log2_tile_cols)
{
    const int sb_cols = (mi_cols + 7) >> 3;
    int start = 0;
    for (int t = 1; t < (1 << log2_tile_cols); t++) {
        int o = ((t * sb_cols) >> log2_tile_cols) << 3;
        if (o > mi_cols) o = mi_cols;
        if (o <= mi_col) start = o;
    }
    return start;
}

/* Residual grid (and SPEC temp) index of a plane's sample. */
__device__ __forceinline__ int plane_at(int p, int x, int y)
{
    return p == 0 ? y * 64 + x : 4096 + (p - 1) * 1024 + y * 32 + x;
}

/* Sum of e[min(i, last)] over i < n (n <= 64). An aligned edge without
 * repeats goes as independent word loads, as many as its size needs. */
template <class T>
__device__ __forceinline__ unsigned edge_sum(const T *e, int n, int last)
{
    constexpr int kPer = 4 / (int)sizeof(T);
    unsigned s = 0;
    if (last >= n - 1 && !((uintptr_t)e & 3) && !(n & (kPer - 1))) {
        const uint32_t *w = reinterpret_cast<const uint32_t *>(e);
        auto add = [&](uint32_t v) { s = sizeof(T) == 1 ? __dp4a(v, 0x01010101u, s) : s + (v & 0xffffu) + (v >> 16); };
        const int m = n / kPer;
        int k = 0;
        for (; k + 4 <= m; k += 4) {
            const uint32_t a = w[k], b = w[k + 1], c = w[k + 2], d = w[k + 3];
            add(a); add(b); add(c); add(d);
        }
        if (m & 2) {
            const uint32_t a = w[k], b = w[k + 1];
            add(a); add(b);
            k += 2;
        }
        if (m & 1) add(w[k]);
    } else {
        for (int i = 0; i < n; i++) s += e[min(i, last)];
    }
    return s;
}

/* The samples that a task's DC counts, as the reciprocal of its division:
 * (sum * inv) >> 32 is sum / n for sum < 2^32 / n. */
__device__ __forceinline__ uint32_t dc_inverse(int n)
{
    return n > 1 ? (uint32_t)((0x100000000ull + (unsigned)n - 1u) / (unsigned)n) : 0u;
}

/* Four samples of a task, in two parts: what does not wait for other samples
 * (where they are, their residuals), then the prediction. */
template <class T>
struct IntraQuad {
    const T *up, *lf;                /* the task's row above, left column    */
    T *dst, *col;                    /* the samples; column copies of their row */
    uint32_t r0, r1;                 /* their residuals                      */
    ITask t;
    int r, c0, nc;
    __device__ __forceinline__ void load(const IntraView<T> &V, const ITask &task, int row, int q)
    {
        t = task;
        r = row;
        c0 = 4 * q;
        const int p = t.plane(), pitch = p ? kCPitch : kYPitch, x = t.x(), y = t.y();
        T *const tile = V.tile(p);
        nc = min(4, t.w() - c0);
        up = tile + (y - 1) * pitch + x;
        lf = V.col(p) + (p ? (x >> 1) * 32 : (x >> 2) * 64) + y;
        dst = tile + (y + r) * pitch + x + c0;
        col = V.col(p) + y + r;
        /* x is even: two words of residuals */
        const uint32_t *rs = reinterpret_cast<const uint32_t *>(V.res + plane_at(p, x + c0, y + r));
        r0 = rs[0];
        r1 = nc > 2 ? rs[1] : 0u;
    }
    /* A: the profile; directional modes are FULL's. Every directional sample
     * is a copy, a two-tap or a three-tap average at one place of the edge E:
     * E(i) = above[i] for i >= -1 (-1 the corner), left[-i - 2] below (the same
     * places as in IntraLane::prepare, which has a sample a lane). LIST:
     * the superblock runs in list order; only there FULL misses an edge that
     * is not the tile's (a block off the 8x8 grid whose first MI is the
     * picture's or tile column's first), so that the halo does not hold it. */
    template <int A, int MAXV, bool LIST>
    __device__ __forceinline__ void run() const
    {
        const int mode = t.mode();
        const bool no_up = LIST && A == CVP9_ARITH_FULL && !(t.avail() & 1u), no_lf = LIST && A == CVP9_ARITH_FULL && !(t.avail() & 2u);
        auto above = [&](int i) -> int { return no_up ? MAXV / 2 : no_lf && i < 0 ? MAXV / 2 + 2 : up[min(i, t.acl())]; };
        auto left = [&](int i) -> int { return no_lf ? MAXV / 2 + 2 : lf[min(i, t.lcl())]; };
        int v[4];
        if (mode == 0) {
            const unsigned av = t.avail(), n = (av & 1u ? t.pw() : 0) + (av & 2u ? t.ph() : 0);
            const unsigned sum = (av & 1u ? edge_sum(up, t.pw(), t.acl()) : 0u) +
                                 (av & 2u ? edge_sum(lf, t.ph(), t.lcl()) : 0u) + (n >> 1);
            const unsigned dc = n == 0 ? (unsigned)(MAXV + 1) / 2 : t.inv ? __umulhi(sum, t.inv) : sum;
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = (int)dc;
        } else if (A != CVP9_ARITH_FULL || mode == 9 || mode <= 2) {
            const int l = left(r), tl = above(-1);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int a = above(c0 + i);
                v[i] = mode == 1 ? a : mode == 2 ? l : clampi(a + l - tl, 0, MAXV);
            }
        } else {
            const int n = t.pw();
            auto E = [&](int i) -> int {
                if (LIST) return i >= -1 ? above(i) : left(-i - 2);
                return *(i >= -1 ? up + min(i, t.acl()) : lf + min(-i - 2, t.lcl()));
            };
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int c = c0 + k;
                int i, taps = 3;             /* E(i), E(i) E(i+1), or E(i) E(i+1) E(i+2) */
                if (mode == 3) {
                    i = r + c;
                    if (i + 2 >= 2 * n) { i = 2 * n - 1; taps = 1; }
                } else if (mode == 8) {
                    i = (r >> 1) + c;
                    if (!(r & 1)) taps = 2;
                } else if (mode == 4) {
                    i = c - r - 2;
                } else if (mode == 5) {
                    const int d = r - 2 * c, j = c - (r >> 1);
                    i = d >= 2 ? -d - 1 : j - 2 + !(r & 1);
                    if (d < 2 && !(r & 1)) taps = 2;
                } else if (mode == 6) {
                    const int d = c - 2 * r, rr = r - (c >> 1);
                    i = d >= 2 ? d - 3 : -rr - 2;
                    if (d < 2 && !(c & 1)) taps = 2;
                } else {
                    const int j = r + (c >> 1);
                    i = -j - 4 + !(c & 1);
                    if (!(c & 1)) taps = 2;
                }
                const int e0 = E(i), e1 = E(i + 1), e2 = E(i + 2);
                v[k] = taps == 1 ? e0 : taps == 2 ? (e0 + e1 + 1) >> 1 : (e0 + 2 * e1 + e2 + 2) >> 2;
            }
        }
        if (A == CVP9_ARITH_SPEC && (r >= t.ph() || c0 + 4 > t.pw())) {
#pragma unroll
            for (int i = 0; i < 4; i++) if (r >= t.ph() || c0 + i >= t.pw()) v[i] = i < nc ? dst[i] : 0;
        }
        v[0] = clampi(v[0] + (int16_t)(r0 & 0xffffu), 0, MAXV);
        v[1] = clampi(v[1] + ((int)r0 >> 16), 0, MAXV);
        v[2] = clampi(v[2] + (int16_t)(r1 & 0xffffu), 0, MAXV);
        v[3] = clampi(v[3] + ((int)r1 >> 16), 0, MAXV);
        const int x = t.x(), cx = x + c0;
        if (nc == 4 && !(x & 3)) {
            if (sizeof(T) == 1) {
                *reinterpret_cast<uint32_t *>(dst) = (uint32_t)v[0] | (uint32_t)v[1] << 8 | (uint32_t)v[2] << 16 |
                                                     (uint32_t)v[3] << 24;
            } else {
                *reinterpret_cast<uint2 *>(dst) = make_uint2((uint32_t)v[0] | (uint32_t)v[1] << 16,
                                                             (uint32_t)v[2] | (uint32_t)v[3] << 16);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) if (i < nc) dst[i] = (T)v[i];
        }
        if (t.plane() == 0) {
            if (nc == 4 && cx < 60) col[((cx + 4) >> 2) * 64] = (T)v[3];
        } else {
            if (nc >= 2 && cx < 30) col[((cx + 2) >> 1) * 32] = (T)v[1];
            if (nc == 4 && cx < 28) col[((cx + 4) >> 1) * 32] = (T)v[3];
        }
    }
};

/* FULL: TXs of a block. */
template <class B>
__device__ __forceinline__ int intra_tx_count(const B &b, const cvp9_job_t &job, int sbx, int sby)
{
    int n = 0;
#pragma unroll
    for (int p = 0; p < 3; p++) {
        int txl, nx, ny, pbw;
        plane_layout(b, job, sbx + b.x, sby + b.y, p, txl, nx, ny, pbw);
        n += nx * ny;
    }
    return n;
}

/* FULL: TX k (coding order: planes, then raster) of an intra block as task
 * `id`, a thread each; own: mark the cells it writes. */
template <class B>
__device__ __forceinline__ void intra_tx_task(IntraWork &W, const B &b, const cvp9_job_t &job, int sbx, int sby, int k,
                                              int id, bool own)
{
    const int gx = sbx + b.x, gy = sby + b.y;
    int p = 0, txl, nx, ny, pbw;
    for (;; p++) {
        plane_layout(b, job, gx, gy, p, txl, nx, ny, pbw);
        if (k < nx * ny || p == 2) break;
        k -= nx * ny;
    }
    const bool left_ok = (gx >> 3) > full_tile_start(gx >> 3, job.mi_cols, job.log2_tile_cols);
    const int n = 4 << txl, mode = p ? (b.uvmode > 9 ? 0 : b.uvmode) : (b.ymode > 9 ? 0 : b.ymode);
    const int pw = p ? job.CW : job.W, ph = p ? job.CH : job.H, tile = p ? 32 : 64;
    const int ty = div_small(k, nx), tx = k - ty * nx;
    const int lx = (p ? (b.x >> 1) : b.x) + tx * n, ly = (p ? (b.y >> 1) : b.y) + ty * n;
    const int X0 = (p ? (gx >> 1) : gx) + tx * n, Y0 = (p ? (gy >> 1) : gy) + ty * n;
    /* above-right: not past the block's last whole 4x4 (6 samples of chroma have one) */
    const bool top = ty > 0 || gy >= 8, right = n == 4 && (tx + 1) * n < (pbw & ~3);
    const int avail = (top ? 1 : 0) | (tx > 0 || left_ok ? 2 : 0);
    st_task(&W.task[id], lx, ly, max(0, min(n, min(pw - X0, tile - lx))), max(0, min(n, min(ph - Y0, tile - ly))), p, mode,
            top ? max(1, min(n + (right ? 4 : 0), pw - X0)) - 1 : n - 1, max(0, min(n - 1, ph - 1 - Y0)), avail, n, n,
            1u << (32 - (2 + txl + (avail == 3))));
    if (own) {
        uint16_t *o = W.own + (p == 0 ? 0 : 192 + 64 * p);
        const int wpt = p ? 8 : 16;
        for (int cy = ly >> 2; cy < (ly + n) >> 2; cy++)
            for (int cx = lx >> 2; cx < (lx + n) >> 2; cx++) o[cy * wpt + cx] = (uint16_t)(id + 1);
    }
}

/* Largest k in [0, n) with base[k] <= v (base ascending, base[0] = 0). */
__device__ __forceinline__ int find_base(const uint16_t *base, int n, int v)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (base[mid] <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

/* Levels, whole CTA. A thread's tasks are rectangles of 4x4 cells; each reads
 * the cells above it (up to column `up`), to its left and at its corner, of
 * which only bottom rows and right columns of tasks matter. Those of unplaced
 * tasks are bits of two maps, so a task sees with two words whether all it
 * reads is placed; every pass places the tasks that see nothing open, the
 * pass's number their level. (Relaxing levels cell by cell took 33 k cycles a
 * superblock of 64 8x8 blocks, this 8 k.) */
struct LvlTask {
    uint32_t *ur, *lc, *br, *rc;     /* row above, column left; own bottom row, right column */
    uint32_t um, lm, cm, rm;         /* cells read there; own columns and rows */
    int      level;                  /* -1: not placed yet                   */
    __device__ __forceinline__ void set(uint32_t *prow, uint32_t *pcol, int x0, int x1, int y0, int y1, int up)
    {
        cm = ((2u << x1) - 1u) & ~((1u << x0) - 1u);
        rm = ((2u << y1) - 1u) & ~((1u << y0) - 1u);
        um = y0 > 0 ? ((2u << up) - 1u) & ~((1u << max(0, x0 - 1)) - 1u) : 0u;
        lm = x0 > 0 ? rm : 0u;
        ur = prow + max(0, y0 - 1);
        lc = pcol + max(0, x0 - 1);
        br = prow + y1;
        rc = pcol + x1;
        level = -1;
        atomicOr(br, cm);
        atomicOr(rc, rm);
    }
};

/* W.prow and W.pcol zero, then every task set, then a barrier, before this. */
template <int N>
__device__ __forceinline__ void intra_levels(LvlTask (&k)[N], const bool (&have)[N])
{
    for (int L = 0; L < kMaxTasks; L++) {
        bool go[N], open = false;
#pragma unroll
        for (int i = 0; i < N; i++)
            go[i] = have[i] && k[i].level < 0 &&
                    !((*(volatile uint32_t *)k[i].ur & k[i].um) | (*(volatile uint32_t *)k[i].lc & k[i].lm));
        __syncthreads();
#pragma unroll
        for (int i = 0; i < N; i++) {
            if (go[i]) {
                atomicAnd(k[i].br, ~k[i].cm);
                atomicAnd(k[i].rc, ~k[i].rm);
                k[i].level = L;
            }
            open |= have[i] && k[i].level < 0;
        }
        if (!__syncthreads_or(open)) break;
    }
}

/* FULL: the levels of the TX tasks (two a thread: at most kMaxTasks of them
 * on at least kMaxTasks / 2 threads). */
__device__ __forceinline__ void intra_tx_levels(IntraWork &W, int ntask, int tid, int nthreads)
{
    LvlTask lt[2];
    bool have[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int t = tid + i * nthreads;
        have[i] = t < ntask;
        if (!have[i]) continue;
        const ITask k = ld_task(&W.task[t]);
        const int p = k.plane(), n = k.pw(), x1 = (k.x() + n - 1) >> 2;
        lt[i].set(W.prow[p], W.pcol[p], k.x() >> 2, x1, k.y() >> 2, (k.y() + n - 1) >> 2,
                  min(p ? 7 : 15, x1 + (k.acl() >= n)));
    }
    __syncthreads();
    intra_levels<2>(lt, have);
#pragma unroll
    for (int i = 0; i < 2; i++) if (have[i]) W.lvl[tid + i * nthreads] = (uint16_t)max(0, lt[i].level);
}

/* How intra_run predicts a task's quads: 0 DC, 1 from the row above and the
 * left column (V, H, TM), 2 FULL's directional modes, 3 what does not consist
 * of aligned words (a clipped area, chroma two samples wide, a repeated edge,
 * no edge at all): as IntraQuad has it. */
template <int A>
__device__ __forceinline__ int intra_kind(const ITask &k)
{
    const int mode = k.mode();
    if (A == CVP9_ARITH_FULL && mode >= 3 && mode <= 8) return 2;
    const bool words = !((k.x() | k.w()) & 3) &&
                       (A != CVP9_ARITH_SPEC || (k.w() == k.pw() && k.h() == k.ph()));
    if (!words) return 3;
    if (mode) return k.acl() >= k.w() - 1 ? 1 : 3;
    return !((k.y() | k.h() | k.pw() | k.ph()) & 3) && k.acl() >= k.pw() - 1 && k.lcl() >= k.ph() - 1 && k.avail() ? 0 : 3;
}

/* A quad: x: its place in the tile (13 bits, from luma's (0, 0)), row (6),
 * column / 4 (4), task (9); y: its row in the left column (11 bits, from
 * column 0), residual / 4 (11), chroma (1), mode (4). */
template <class T>
__device__ __forceinline__ uint2 quad_word(const ITask &k, int t, int r, int q)
{
    using V = IntraView<T>;
    const int p = k.plane(), pitch = p ? kCPitch : kYPitch, y = k.y() + r, x = k.x() + 4 * q;
    const int at = (p ? V::kU + (p - 1) * V::kUV : 0) + y * pitch + x;
    const int lf = p ? 1024 + (p - 1) * 512 + (k.x() >> 1) * 32 + y : (k.x() >> 2) * 64 + y;
    return make_uint2((uint32_t)at | (uint32_t)r << 13 | (uint32_t)q << 19 | (uint32_t)t << 23,
                      (uint32_t)lf | (uint32_t)(plane_at(p, x, y) >> 2) << 11 | (p ? 1u << 22 : 0u) |
                      (uint32_t)(k.mode() & 15) << 23);
}

/* Sort the quads of all tasks by level and kind, whole CTA, and deal each
 * level's to warps: W.job[W.lvlj[L]] .. W.job[W.lvlj[L + 1]] are level L's,
 * each of one kind, so that a warp runs one path: a level waits for the
 * instructions of its longest warp, about 8 cycles each, and not for data.
 * With all kinds in one warp and places and residuals worked out by the
 * thread that predicts: three 1080p SPEC pictures, one of them key, 0.84 ms,
 * eight 10-bit 1080p key pictures 3.05 ms; by kind and prepared a level
 * ahead: 0.70 and 2.66 ms. A thread per four-sample group of the SB finds its
 * task from the owner map of the cells: W.own of each plane's (FULL), or the
 * block map `cell` of the luma ones, whose chroma groups start at even
 * samples. */
template <int A, class T, class C>
__device__ __forceinline__ void intra_sort(IntraWork &W, const C *cell, int ntask, int tid, int nthreads)
{
    const int lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kMaxTasks * 2; i += nthreads) (&W.lvlq[0][0])[i] = 0;
    for (int i = tid; i < kMaxQuads; i += nthreads) W.qtab[i] = make_uint2(kNoQuad, 0u);
    if (tid == 0) W.nlev = 0;
    __syncthreads();
    int top = 0;
    for (int t = tid; t < ntask; t += nthreads) {
        const ITask k = ld_task(&W.task[t]);
        const int kind = intra_kind<A>(k), sh = 16 * (kind & 1);
        W.qat[t] = (uint16_t)(atomicAdd(&W.lvlq[W.lvl[t]][kind >> 1], (unsigned)(((k.w() + 3) >> 2) * k.h()) << sh) >> sh);
        top = max(top, (int)W.lvl[t] + 1);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0 && top) atomicMax(&W.nlev, top);
    __syncthreads();
    if (warp == 0) {
        const int nlev = W.nlev, per = (nlev + 31) >> 5, b0 = lane * per, b1 = min(b0 + per, nlev);
        auto jobs = [](unsigned a, unsigned b) {
            return ((a & 0xffffu) + 31) / 32 + ((a >> 16) + 31) / 32 + ((b & 0xffffu) + 7) / 8 + ((b >> 16) + 31) / 32;
        };
        unsigned sum = 0, js = 0;
        for (int l = b0; l < b1; l++) {
            const unsigned a = W.lvlq[l][0], b = W.lvlq[l][1];
            sum += (a & 0xffffu) + (a >> 16) + (b & 0xffffu) + (b >> 16);
            js += jobs(a, b);
        }
        unsigned x = sum | js << 16;         /* at most kMaxQuads, kMaxJobs  */
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned z = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += z;
        }
        if (lane == 31) W.lvlj[nlev] = (uint16_t)min(x >> 16, (unsigned)kMaxJobs);
        x -= sum | js << 16;
        unsigned at = x & 0xffffu, j = x >> 16;
        for (int l = b0; l < b1; l++) {
            const unsigned a = W.lvlq[l][0], b = W.lvlq[l][1];
            unsigned first[4];
            W.lvlj[l] = (uint16_t)min(j, (unsigned)kMaxJobs);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const unsigned n = ((k < 2 ? a : b) >> (16 * (k & 1))) & 0xffffu, step = k == 2 ? 8u : 32u;
                first[k] = at;
                for (unsigned i = 0; i < n; i += step, j++)
                    if (j < (unsigned)kMaxJobs && at + i < (unsigned)kMaxQuads)
                        W.job[j] = (at + i) | (min(step, n - i) - 1u) << 11 | (unsigned)k << 16;
                at += n;
            }
            W.lvlq[l][0] = first[0] | first[1] << 16;
            W.lvlq[l][1] = first[2] | first[3] << 16;
        }
    }
    __syncthreads();
    constexpr int kGroups = A == CVP9_ARITH_FULL ? 1024 + 2 * 256 : 1024 + 2 * 512;
    for (int i = tid; i < kGroups; i += nthreads) {
        int t, x, y;
        if (i < 1024) {
            y = i >> 4;
            x = (i & 15) * 4;
            const int c = (y >> 2) * 16 + (x >> 2);
            t = A == CVP9_ARITH_FULL ? (int)W.own[c] - 1 : cell[c] ? (int)W.own[cell[c] - 1] : -1;
        } else if (A == CVP9_ARITH_FULL) {
            const int p = (i - 1024) >> 8, j = i & 255;
            y = j >> 3;
            x = (j & 7) * 4;
            t = (int)W.own[256 + 64 * p + (y >> 2) * 8 + (x >> 2)] - 1;
        } else {
            const int p = (i - 1024) >> 9, j = i & 511;
            y = j >> 4;
            x = (j & 15) * 2;
            const int o = cell[(y >> 1) * 16 + (x >> 1)];
            t = o ? (int)W.own[o - 1] : -1;
            if (t >= 0 && t != 0xFFFF) t += 1 + p;
        }
        if (t < 0 || t >= ntask) continue;
        const ITask k = ld_task(&W.task[t]);
        const int r = y - k.y(), c = x - k.x();
        if (r >= k.h() || c >= k.w() || (c & 3)) continue;
        const int kind = intra_kind<A>(k);
        const unsigned at = ((W.lvlq[W.lvl[t]][kind >> 1] >> (16 * (kind & 1))) & 0xffffu) + W.qat[t] +
                            (unsigned)(r * ((k.w() + 3) >> 2) + (c >> 2));
        if (at < (unsigned)kMaxQuads) W.qtab[at] = quad_word<T>(k, t, r, c >> 2);
    }
    __syncthreads();
}

/* What a lane of intra_run does for a level, before (prepare) and after (run)
 * the samples it reads are there: four samples of a quad, or one of a
 * directional mode's, four lanes a quad. A level waits for the instructions
 * of run, so all that can be is done in prepare; places are bytes from luma's
 * (0, 0), which shared memory loads take without pointer arithmetic. */
template <int A, int MAXV, class T>
struct IntraLane {
    static constexpr int kPer = 4 / (int)sizeof(T);      /* samples a word   */
    static constexpr uint32_t kHi = (uint32_t)MAXV << 16 | MAXV;
    int a0, a1, a2;                  /* edge samples: DC up, left less the words above; V, H, TM: up, left,
                                      * corner; else E(i) .. E(i + 2)        */
    int dst, cl;                     /* its sample(s); their column copy (cl[-32]: of the second, chroma) */
    uint32_t r0, r1;                 /* residuals                            */
    uint32_t m;                      /* DC: reciprocal; V, H, TM: 0 leaves out the row and the corner; 2: weights */
    int nu, n;                       /* DC: words of the edge above, of both */
    int kind;
    unsigned put;                    /* 1: dst, 2: cl, 4: cl[-32]            */
    uint32_t word;                   /* quad_word's x                        */

    template <class E>
    static __device__ __forceinline__ const E &at(const IntraView<T> &V, int off)
    {
        return *reinterpret_cast<const E *>(reinterpret_cast<const char *>(V.tile0) + off);
    }
    template <class E>
    static __device__ __forceinline__ void put_at(const IntraView<T> &V, int off, E v)
    {
        *reinterpret_cast<E *>(reinterpret_cast<char *>(V.tile0) + off) = v;
    }

    __device__ __forceinline__ void prepare(const IntraWork &W, const IntraView<T> &V, uint32_t job, int lane)
    {
        constexpr int S = (int)sizeof(T);
        kind = (int)(job >> 16);
        const int cnt = (int)((job >> 11) & 31u), i0 = kind == 2 ? lane >> 2 : lane;
        const uint2 d = W.qtab[(job & 2047u) + min(i0, cnt)];
        const bool have = i0 <= cnt && d.x != kNoQuad;
        word = d.x;
        const bool chroma = (d.y >> 22) & 1u;
        const int pitch = chroma ? kCPitch : kYPitch, r = (int)(d.x >> 13) & 63, q = (int)(d.x >> 19) & 15;
        const int lf = (int)(d.y & 2047u), left = (int)(reinterpret_cast<const char *>(V.col0) -
                                                        reinterpret_cast<const char *>(V.tile0)) + lf * S;
        dst = (int)(d.x & 8191u) * S;
        const int up = dst - (r + 1) * pitch * S;
        const int16_t *const rs = V.res + ((d.y >> 11) & 2047u) * 4;
        put = have;
        if (kind <= 1) {
            const uint2 w = *reinterpret_cast<const uint2 *>(rs);
            /* the samples are clamped: so may the residuals be, and sums stay in 16 bits */
            constexpr uint32_t lo = (uint32_t)(-MAXV & 0xffff) * 0x10001u;
            r0 = min2_s16(max2_s16(w.x, lo), kHi);
            r1 = min2_s16(max2_s16(w.y, lo), kHi);
            cl = left + (q + 1) * 64 * S;
            const int c = chroma ? ((lf >> 5) & 15) + 2 * q + 1 : (lf >> 6) + q;
            if (have && c < 15) put = 3u;
            if (have && chroma && c < 16) put |= 4u;
        }
        if (kind == 0) {
            const ITask t = ld_task(&W.task[min(d.x >> 23, kMaxTasks - 1u)]);
            nu = t.avail() & 1u ? t.pw() / kPer : 0;
            n = nu + (t.avail() & 2u ? t.ph() / kPer : 0);
            a0 = up - 4 * q * S;
            a1 = left - r * S - nu * 4;
            m = t.inv;
        } else if (kind == 1) {
            const int mode = (int)(d.y >> 23) & 15;
            a0 = up;
            a2 = up - (4 * q + 1) * S;
            a1 = mode == 1 ? a2 : left;
            m = mode == 2 ? 0u : 0xFFFFFFFFu;
        } else if (A == CVP9_ARITH_FULL && kind == 2) {
            const ITask t = ld_task(&W.task[min(d.x >> 23, kMaxTasks - 1u)]);
            const int mode = t.mode(), c = 4 * q + (lane & 3), size = t.pw(), acl = t.acl(), lcl = t.lcl();
            /* the place (as in IntraQuad::run) and the weights, in quarters, of
             * the sample's taps */
            int i;
            bool two = false, one = false;
            if (mode == 3) {
                i = r + c;
                one = i + 2 >= 2 * size;
                if (one) i = 2 * size - 1;
            } else if (mode == 8) {
                i = (r >> 1) + c;
                two = !(r & 1);
            } else if (mode == 4) {
                i = c - r - 2;
            } else if (mode == 5) {
                const int d5 = r - 2 * c;
                two = d5 < 2 && !(r & 1);
                i = d5 >= 2 ? -d5 - 1 : c - (r >> 1) - 2 + !(r & 1);
            } else if (mode == 6) {
                const int d6 = c - 2 * r;
                two = d6 < 2 && !(c & 1);
                i = d6 >= 2 ? d6 - 3 : (c >> 1) - r - 2;
            } else {
                i = -r - (c >> 1) - 4 + !(c & 1);
                two = !(c & 1);
            }
            m = one ? 4u : two ? 2u | 2u << 8 : 1u | 2u << 8 | 1u << 16;
            const int u = up - 4 * q * S, l = left - r * S;
            auto E = [&](int k) { return k >= -1 ? u + min(k, acl) * S : l + min(-k - 2, lcl) * S; };
            a0 = E(i);
            a1 = E(i + 1);
            a2 = E(i + 2);
            r0 = (uint32_t)(int)rs[lane & 3];
            dst += (lane & 3) * S;
            const int e = c + 1;
            cl = left + (chroma ? (e >> 1) * 32 : (e >> 2) * 64) * S;
            const bool copy = chroma ? !(e & 1) && ((lf >> 5) & 15) + (e >> 1) < 16 : !(e & 3) && (lf >> 6) + (e >> 2) < 16;
            put = have && c < t.w() ? (copy ? 3u : 1u) : 0u;
        }
    }

    __device__ __forceinline__ void run(const IntraWork &W, const IntraView<T> &V, int lane) const
    {
        if (kind <= 1) {
            uint32_t v0, v1;
            if (kind == 0) {
                /* the four lanes are of one task: its quads come in fours */
                unsigned s = 0;
                for (int j = lane & 3; j < n; j += 4) {
                    const uint32_t w = at<uint32_t>(V, (j < nu ? a0 : a1) + 4 * j);
                    s = sizeof(T) == 1 ? __dp4a(w, 0x01010101u, s) : s + (w & 0xffffu) + (w >> 16);
                }
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                v0 = v1 = __umulhi(s + (unsigned)(n * kPer >> 1), m) * 0x10001u;
            } else {
                const uint32_t w0 = at<uint32_t>(V, a0) & m, w1 = sizeof(T) == 1 ? 0u : at<uint32_t>(V, a0 + 4) & m;
                const uint32_t d = (uint32_t)at<T>(V, a1) - ((uint32_t)at<T>(V, a2) & m), dd = __byte_perm(d, 0u, 0x1010);
                v0 = sizeof(T) == 1 ? __byte_perm(w0, 0u, 0x4140) : w0;
                v1 = sizeof(T) == 1 ? __byte_perm(w0, 0u, 0x4342) : w1;
                v0 = min2_s16(__viaddmax_s16x2(v0, dd, 0u), kHi);
                v1 = min2_s16(__viaddmax_s16x2(v1, dd, 0u), kHi);
            }
            v0 = min2_s16(__viaddmax_s16x2(v0, r0, 0u), kHi);
            v1 = min2_s16(__viaddmax_s16x2(v1, r1, 0u), kHi);
            if (put & 1u) {
                if (sizeof(T) == 1) put_at<uint32_t>(V, dst, __byte_perm(v0, v1, 0x6420));
                else put_at<uint2>(V, dst, make_uint2(v0, v1));
            }
            if (put & 2u) put_at<T>(V, cl, (T)(v1 >> 16));
            if (put & 4u) put_at<T>(V, cl - 32 * (int)sizeof(T), (T)(v0 >> 16));
        } else if (A == CVP9_ARITH_FULL && kind == 2) {
            const int e = at<T>(V, a0) * (int)(m & 255u) + at<T>(V, a1) * (int)((m >> 8) & 255u) + at<T>(V, a2) * (int)(m >> 16);
            const T v = (T)clampi(((e + 2) >> 2) + (int)r0, 0, MAXV);
            if (put & 1u) put_at<T>(V, dst, v);
            if (put & 2u) put_at<T>(V, cl, v);
        } else if (put) {
            IntraQuad<T> k;
            k.load(V, ld_task(&W.task[min(word >> 23, kMaxTasks - 1u)]), (int)(word >> 13) & 63, (int)(word >> 19) & 15);
            k.template run<A, MAXV, false>();
        }
    }
};

/* The levels, whole CTA: one barrier each. A warp has a job of a level at
 * most, in general; odd levels begin at the middle warp, so that the warps
 * which a level leaves idle prepare the next one. */
template <int A, int MAXV, class T>
__device__ __forceinline__ void intra_run(const IntraWork &W, const IntraView<T> &V, int tid, int nthreads)
{
    const int nlev = W.nlev, nw = nthreads >> 5, warp = tid >> 5, lane = tid & 31;
    IntraLane<A, MAXV, T> k;
    int j = warp, end = nlev ? W.lvlj[1] : 0;
    if (j < end) k.prepare(W, V, W.job[j], lane);
    for (int L = 0; L < nlev; L++) {
        while (j < end) {
            k.run(W, V, lane);
            j += nw;
            if (j < end) k.prepare(W, V, W.job[j], lane);
        }
        if (L + 1 < nlev) {
            j = end + ((warp + (L & 1 ? 0 : nw >> 1)) & (nw - 1));
            end = W.lvlj[L + 2];
            if (j < end) k.prepare(W, V, W.job[j], lane);
        }
        __syncthreads();
    }
}

/* One task after another in coding order, whole CTA (a superblock that runs
 * in list order). */
template <int A, int MAXV, class T>
__device__ __forceinline__ void intra_run_ordered(const IntraWork &W, const IntraView<T> &V, int ntask, int tid,
                                                  int nthreads)
{
    for (int t = 0; t < ntask; t++) {
        const ITask k = ld_task(&W.task[t]);
        const int qw = (k.w() + 3) >> 2, nq = qw * k.h();
        for (int i = tid; i < nq; i += nthreads) {
            const int r = div_small(i, qw);
            IntraQuad<T> quad;
            quad.load(V, k, r, i - r * qw);
            quad.template run<A, MAXV, true>();
        }
        __syncthreads();
    }
}

/* The left-column copies of everything in the tile, whole CTA. */
template <class T>
__device__ __forceinline__ void intra_fill_cols(const IntraView<T> &V, int tid, int nthreads)
{
    for (int i = tid; i < 15 * 64; i += nthreads) {
        const int k = 1 + (i >> 6), y = i & 63;
        V.col0[k * 64 + y] = V.tile0[y * kYPitch + 4 * k - 1];
    }
    for (int i = tid; i < 2 * 15 * 32; i += nthreads) {
        const int p = 1 + (i >= 15 * 32), j = p == 2 ? i - 15 * 32 : i, k = 1 + (j >> 5), y = j & 31;
        V.col(p)[k * 32 + y] = V.tile(p)[y * kCPitch + 2 * k - 1];
    }
}

/* The halo of a superblock, whole CTA: the row above (x = -1 .. 63) and the
 * left column of each plane, from the picture where `top` / `left` say that
 * they are available, else the profile's fill values (above, left). The
 * corner is a sample only where both are. need: the neighbours whose samples
 * are read (intra_needs) and that have been waited for; the others' may still
 * be in the middle of being written, and are left alone. */
template <class T>
__device__ __forceinline__ void intra_halo(const IntraView<T> &V, const cvp9_job_t &job, int sbx, int sby, bool top,
                                           bool left, unsigned need, int fill_a, int fill_l, int tid, int nthreads)
{
    const bool load_t = top && (need & 2u), load_l = left && (need & 1u), load_c = top && left && (need & 4u);
    const T *base = reinterpret_cast<const T *>(job.out);
    /* 128 samples above, 128 to the left: one each for 256 threads, and the
     * corner for three of them at the same time */
    for (int i = tid; i < 256; i += nthreads) {
        const int half = i >> 7, j = i & 127, p = j < 64 ? 0 : j < 96 ? 1 : 2, k = p ? j & 31 : j;
        const int w = p ? job.CW : job.W, h = p ? job.CH : job.H;
        const int X = p ? sbx >> 1 : sbx, Y = p ? sby >> 1 : sby;
        const T *g = base + (p ? (size_t)job.W * job.H + (size_t)(p - 1) * job.CW * job.CH : 0);
        T *tile = V.tile(p), *col = V.col(p);
        const int pitch = p ? kCPitch : kYPitch;
        if (!half) {
            T c = (T)(top ? fill_l : fill_a);
            if (k == 0 && load_c) c = __ldcg(g + (size_t)(Y - 1) * w + X - 1);
            const T v = load_t ? (X + k < w ? __ldcg(g + (size_t)(Y - 1) * w + X + k) : (T)0) : (T)fill_a;
            tile[-pitch + k] = v;
            if (k == 0) tile[-pitch - 1] = c;
        } else {
            const T v = load_l ? (Y + k < h ? __ldcg(g + (size_t)(Y + k) * w + X - 1) : (T)0) : (T)fill_l;
            col[k] = v;
            tile[k * pitch - 1] = v;
        }
    }
}

/* f(i, k) for k < count of each of the warp's lanes (i: the lane's own number
 * or the lane in turn): up to four by the lane itself, more by the whole warp. */
template <class F>
__device__ __forceinline__ void warp_spread(int count, int lane, F f)
{
    if (count <= 4)
        for (int k = 0; k < count; k++) f(lane, k);
    for (uint32_t m = __ballot_sync(0xffffffffu, count > 4); m; m &= m - 1) {
        const int from = __ffs(m) - 1, n = __shfl_sync(0xffffffffu, count, from);
        for (int k = lane; k < n; k += 32) f(from, k);
    }
}

/* Claim the 4x4 cells of columns [c0x, c1x] and rows [c0y, c1y] for a block:
 * a bit per cell, a word per row of the SB; true when another block has one
 * of them. (A thread a block: a 64x64 block is 16 atomics.) */
__device__ __forceinline__ bool claim_cells(uint32_t *rows, int c0x, int c1x, int c0y, int c1y)
{
    const uint32_t m = ((2u << c1x) - 1u) & ~((1u << c0x) - 1u);
    uint32_t seen = 0;
    for (int cy = c0y; cy <= c1y; cy++) seen |= atomicOr(&rows[cy], m);
    return (seen & m) != 0;
}

/* Cell k of a block's, in its owner map. */
template <class C>
__device__ __forceinline__ void own_cell(C *cell, int b, int c0x, int c1x, int c0y, int k)
{
    const int w = c1x - c0x + 1, r = div_small(k, w);
    cell[(c0y + r) * 16 + c0x + k - r * w] = (C)(b + 1);
}

/* Which neighbours (1 left, 2 above, 4 above-left) the intra blocks of a
 * superblock read: a block at its left edge reads the left one, one at its
 * top edge the one above. */
__device__ __forceinline__ unsigned intra_needs(int x, int y)
{
    return (x == 0 ? 1u : 0u) | (y == 0 ? 2u : 0u) | (x == 0 && y == 0 ? 4u : 0u);
}

/* ── Synchronisation helpers ────────────────────────────────────────────── */

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(unsigned *p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

/* Bounded wait until flag == epoch; returns false on timeout. */
__device__ __forceinline__ bool wait_flag(const unsigned *flag, unsigned epoch)
{
    for (int it = 0; it < kFlagLooks; it++) {
        if (ld_acquire(flag) == epoch) return true;
        __nanosleep(32);
    }
    return false;
}

/* Exclusive prefix sums of two per-thread counts over the CTA (thread order).
 * Returns the totals; uses s_tmp[2 * kWarps]. Must be called by all threads. */
__device__ __forceinline__ void cta_scan2(int a, int b, int *ea, int *eb, int *ta, int *tb, int *s_tmp)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int xa = a, xb = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int ya = __shfl_up_sync(0xffffffffu, xa, o), yb = __shfl_up_sync(0xffffffffu, xb, o);
        if (lane >= o) { xa += ya; xb += yb; }
    }
    if (lane == 31) { s_tmp[warp] = xa; s_tmp[kWarps + warp] = xb; }
    __syncthreads();
    int pa = 0, pb = 0, sa = 0, sb = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        int va = s_tmp[w], vb = s_tmp[kWarps + w];
        if (w < warp) { pa += va; pb += vb; }
        sa += va; sb += vb;
    }
    *ea = pa + xa - a;
    *eb = pb + xb - b;
    *ta = sa;
    *tb = sb;
}

/* Position and extent of chunk `k` of block b: an 8x8 luma region of
 * its block clipped to the frame, and the matching 4x4 chroma region. */
struct ChunkP {
    const BlkS *b;
    int lx0, ly0, lw, lh, cx0, cy0, clw, clh;
};

__device__ __forceinline__ ChunkP chunk_params(const BlkS &b, int k)
{
    ChunkP c;
    c.b = &b;
    const int nx = (b.cw + 7) >> 3;
    const int ccy = nx == 1 ? k : div_small(k, nx), ccx = k - ccy * nx;
    c.lx0 = b.x + ccx * 8;
    c.ly0 = b.y + ccy * 8;
    c.lw = min(8, b.cw - ccx * 8);
    c.lh = min(8, b.ch - ccy * 8);
    const int cbw = (b.cw + 1) >> 1, cbh = (b.ch + 1) >> 1;
    c.cx0 = (b.x >> 1) + ccx * 4;
    c.cy0 = (b.y >> 1) + ccy * 4;
    c.clw = min(4, cbw - ccx * 4);
    c.clh = min(4, cbh - ccy * 4);
    return c;
}

} /* namespace */

/* ── Kernels ─────────────────────────────────────────────────────────────── */

/* Per block: SB membership and the contiguous range of each SB. The
 * per-frame scratch (sb_range, status) is zeroed before this launch. */
__global__ void __launch_bounds__(256) k_scan_blocks(const cvp9_job_t *__restrict__ jobs)
{
    grid_dependency_wait();
    const cvp9_job_t &job = jobs[blockIdx.y];
    const vp9_macroblock_info_t *B = job.blocks;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < job.num_blocks; i += gridDim.x * blockDim.x) {
    auto sb_of = [&](uint32_t k, bool *ok) -> int {
        vp9_macroblock_info_t b = B[k];
        int x = b.x, y = b.y, w = b.width, h = b.height;
        bool good = x < job.W && y < job.H && w >= 4 && h >= 4 && w <= 64 && h <= 64 &&
                    !(x & 3) && !(y & 3) && !(w & 3) && !(h & 3) &&
                    (x & 63) + w <= 64 && (y & 63) + h <= 64 && b.tx_size <= 3;
        *ok = good;
        return (y >> 6) * job.sb_cols + (x >> 6);
    };
    bool ok;
    int sb = sb_of(i, &ok);
    if (!ok) { atomicOr(job.status, (unsigned)CVP9_JOB_BAD_BLOCK); continue; }
    bool okp = true, okn = true;
    int prev = i > 0 ? sb_of(i - 1, &okp) : -1;
    int next = i + 1 < job.num_blocks ? sb_of(i + 1, &okn) : -1;
    uint32_t *r = job.sb_range + 4 * sb;
    if (prev != sb) { r[0] = i; atomicAdd(&r[2], 1u); }
    if (next != sb) r[1] = i + 1;
    }
}

/* Inter prediction, whole CTA: of every inter block's chunks (one null), or
 * of the n chunks of block *one. REFCPU stages the
 * windows of up to kRound chunks per warp with async copies into the (idle)
 * transform buffer, waits once, then computes them. */
template <int A>
__device__ __forceinline__ void recon_inter(ReconSmem &s, const BlkS *one, int n, int sbx, int sby, int warp, int lane)
{
    if (A == CVP9_ARITH_REFCPU) {
        auto params = [&](int chk) {
            const int b = one ? 0 : s.chunk_blk[chk];
            return one ? chunk_params(*one, chk) : chunk_params(s.blk[b], chk - s.chunk_off[b]);
        };
        constexpr int kRound = 4;
        uint8_t *wst = s.temp.mc + warp * (kRound * kChunkStage);
        const int q = lane >> 3, k = lane & 7;
        for (int base = warp; base < n; base += kRound * kWarps) {
            /* lane group q works on chunk base + q * kWarps */
            const int chk = base + q * kWarps;
            const bool have = chk < n;
            ChunkP c;
            McGeo g;
            bool has_ref = false;
            if (have) {
                c = params(chk);
                has_ref = refcpu_geo(s, *c.b, sbx, sby, c.lx0, c.ly0, c.lw, c.lh, c.cx0, c.cy0, c.clw, c.clh, g);
                if (has_ref) refcpu_issue8(wst + q * kChunkStage, g, c.lw, c.lh, c.clw, c.clh, k);
            }
            cp_async_commit();
            cp_async_wait_all();
            __syncwarp();
            if (have) {
                if (has_ref)
                    refcpu_compute8(s, wst + q * kChunkStage, g, c.lx0, c.ly0, c.lw, c.lh, c.cx0, c.cy0, c.clw,
                                    c.clh, k);
                else
                    refcpu_fill8(s, 127, c.lx0, c.ly0, c.lw, c.lh, c.cx0, c.cy0, c.clw, c.clh, k);
            }
            __syncwarp();
        }
    } else {
        /* SPEC and FULL: four chunks a warp */
        const cvp9_job_t &job = s.jc;
        const uint32_t (*P)[2] = A == CVP9_ARITH_FULL ? c_subpel4_pk[job.interp_filter & 3] : c_subpel_pk;
        const int g = lane >> 3, k = lane & 7;
        uint8_t *rows = s.temp.mc + (warp * 4 + g) * 128;
        for (int base = warp * 4; base < n; base += 4 * kWarps) {
            const int chk = base + g;
            const bool on = chk < n;
            const int bi = one || !on ? 0 : s.chunk_blk[chk];
            const BlkS &b = one ? *one : s.blk[bi];
            const int ccw = (b.cw + 1) >> 1, cch = (b.ch + 1) >> 1;
            int p = 0, x = 0, y = 0, w = 0, h = 0;
            if (on) mc_chunk_at(one ? chk : chk - s.chunk_off[bi], b.cw, b.ch, ccw, cch, p, x, y, w, h);
            const int lx = (p ? b.x >> 1 : b.x) + x, ly = (p ? b.y >> 1 : b.y) + y;
            uint8_t *dst = p == 0 ? &TY(s, lx, ly + k) : &TC(s, p, lx, ly + k);
            mc_chunk<uint8_t, A == CVP9_ARITH_FULL>(job, P, b, on, p, (p ? sbx >> 1 : sbx) + lx, (p ? sby >> 1 : sby) + ly, w, h, 128, rows,
                              dst, k);
        }
    }
}

/* REFCPU and SPEC: intra block `bi` as three tasks (one a plane) at W.task[at]. */
template <int A>
__device__ __forceinline__ void intra_block_tasks(IntraWork &W, const BlkS &b, const cvp9_job_t &job, int sbx,
                                                  int sby, int at, int level)
{
#pragma unroll
    for (int p = 0; p < 3; p++) {
        const int m = p ? b.uvmode : b.ymode;
        const int mode = A == CVP9_ARITH_REFCPU ? (m <= 2 ? m : 9) : (m == 0 || m == 2 || m == 9 ? m : 1);
        const int pw = p ? (b.cw + 1) >> 1 : b.cw, ph = p ? (b.ch + 1) >> 1 : b.ch;
        int w = pw, h = ph;
        if (A == CVP9_ARITH_SPEC && (b.w < 8 || b.h < 8)) {   /* the residual's area too: the whole MI */
            const int ow = max((int)b.cw, min(8, job.W - (sbx + b.x))), oh = max((int)b.ch, min(8, job.H - (sby + b.y)));
            w = p ? (ow + 1) >> 1 : ow;
            h = p ? (oh + 1) >> 1 : oh;
        }
        /* REFCPU's DC counts the filled edges too */
        const int avail = (A == CVP9_ARITH_REFCPU || sby + b.y > 0 ? 1 : 0) | (A == CVP9_ARITH_REFCPU || sbx + b.x > 0 ? 2 : 0);
        st_task(&W.task[at + p], p ? b.x >> 1 : b.x, p ? b.y >> 1 : b.y, w, h, p, mode, 255, 255, avail, pw, ph,
                dc_inverse((avail & 1 ? pw : 0) + (avail & 2 ? ph : 0)));
        W.lvl[at + p] = (uint16_t)level;
    }
}

/* The tile of the superblock into the picture, clipped to it: as words where the
 * picture's address (a caller's own, any) and its rows are multiples of 4. */
__device__ __forceinline__ void recon_write(ReconSmem &s, int sbx, int sby, int tid)
{
    const cvp9_job_t &job = s.jc;
    const int vw = min(64, job.W - sbx), vh = min(64, job.H - sby);
    uint8_t *Y = job.out;
    const bool aligned = !((uintptr_t)Y & 3);
    if (aligned && (job.W & 3) == 0) {
        for (int i = tid; i < vh * 16; i += kThreads) {
            int r = i >> 4, c4 = (i & 15) * 4;
            if (c4 >= vw) continue;
            *reinterpret_cast<uint32_t *>(Y + (size_t)(sby + r) * job.W + sbx + c4) =
                *reinterpret_cast<const uint32_t *>(&TY(s, c4, r));
        }
    } else {
        for (int i = tid; i < vh * 64; i += kThreads) {
            int r = i >> 6, c = i & 63;
            if (c < vw) Y[(size_t)(sby + r) * job.W + sbx + c] = TY(s, c, r);
        }
    }
    const int cvw = min(32, job.CW - (sbx >> 1)), cvh = min(32, job.CH - (sby >> 1));
    uint8_t *U = job.out + (size_t)job.W * job.H;
    uint8_t *V = U + (size_t)job.CW * job.CH;
    if (aligned && (job.CW & 3) == 0 && ((size_t)job.W * job.H & 3) == 0) {
        for (int i = tid; i < 2 * cvh * 8; i += kThreads) {
            int p = i >= cvh * 8;
            int k = p ? i - cvh * 8 : i;
            int r = k >> 3, c4 = (k & 7) * 4;
            if (c4 >= cvw) continue;
            *reinterpret_cast<uint32_t *>((p ? V : U) + (size_t)((sby >> 1) + r) * job.CW + (sbx >> 1) + c4) =
                *reinterpret_cast<const uint32_t *>(&TC(s, 1 + p, c4, r));
        }
    } else
    for (int i = tid; i < 2 * cvh * 32; i += kThreads) {
        int p = i >= cvh * 32;
        int k = p ? i - cvh * 32 : i;
        int r = k >> 5, c = k & 31;
        if (c >= cvw) continue;
        (p ? V : U)[(size_t)((sby >> 1) + r) * job.CW + (sbx >> 1) + c] = TC(s, 1 + p, c, r);
    }
}

/* Exclusive prefix sum of v over the CTA (thread order), *total the sum;
 * s.scan_tmp must be idle. */
__device__ __forceinline__ int cta_scan1(ReconSmem &s, int v, int *total)
{
    int ea, eb, ta, tb;
    cta_scan2(v, 0, &ea, &eb, &ta, &tb, s.scan_tmp);
    *total = ta;
    return ea;
}

/* The phases of a superblock are functions of their own, each with the whole
 * register budget of the kernel for its loops: inlined into one body, the
 * values that live across phases were kept in local memory inside the hot
 * loops, where the small L1 that the shared memory leaves (28 KB) misses. They
 * name the shared memory themselves, since a pointer parameter would make
 * every access a generic one. */
template <class S>
__device__ __forceinline__ S &smem_as()
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    return *reinterpret_cast<S *>(smem_raw);
}

__device__ __forceinline__ IntraView<uint8_t> recon_view(ReconSmem &s)
{
    IntraView<uint8_t> V;
    V.tile0 = &TY(s, 0, 0);
    V.col0 = s.col;
    V.res = s.res;
    return V;
}

/* The 4x4 cells of a block: its prediction area; under SPEC and FULL a
 * sub-8x8 block's residual spans the whole 8x8 MI (vp9_kf_tile.c:327-330),
 * so it owns that area too (a block 4 samples wide may be taller than it). */
template <int A>
__device__ __forceinline__ void block_cells(const BlkS &b, const cvp9_job_t &job, int sbx, int sby, int &c0x, int &c1x,
                                            int &c0y, int &c1y)
{
    int ow = b.cw, oh = b.ch;
    if (A != CVP9_ARITH_REFCPU && (b.w < 8 || b.h < 8)) {
        ow = max(ow, min(8, job.W - (sbx + b.x)));
        oh = max(oh, min(8, job.H - (sby + b.y)));
    }
    c0x = b.x >> 2;
    c0y = b.y >> 2;
    c1x = (b.x + ow - 1) >> 2;
    c1y = (b.y + oh - 1) >> 2;
}

/* Inter predictions: of n chunks of the whole SB (one < 0), or of block `one`. */
template <int A>
__device__ __noinline__ void phase_inter(int one, int n, int sbx, int sby)
{
    ReconSmem &s = smem_as<ReconSmem>();
    recon_inter<A>(s, one < 0 ? nullptr : &s.blk[one], n, sbx, sby, threadIdx.x >> 5, threadIdx.x & 31);
}

/* The residual TXs of a superblock, sorted by size, largest first. What
 * bounds them is the length of a transform on one thread and how evenly
 * threads are busy, so a warp takes 32 / N TXs of N x N at a time, a lane a row
 * and then a column of one, with warp barriers only: no warp mixes sizes, no
 * CTA barrier waits for the longest. The rows pass through 4 KB a warp, laid
 * out in 16-byte chunks that are permuted within 128 bytes (tx_word), so that
 * rows and columns both go through all banks. (A thread per row and column
 * over all sizes, CTA barriers between the passes, rows 256 bytes apart: 24 k
 * cycles a superblock of FULL inter blocks, 48 k at 10 bits; this 21 k and
 * 33 k, 5 k of it the list.) */
template <int N> struct std_int { static constexpr int value = N; };

/* x: first coefficient; y: x / 4 | y / 4 << 4 | plane << 8 | TX type << 10 |
 * flags. LIST: a superblock in list order, the only one with blocks off the
 * 8x8 grid, whose chroma TXs lie between 4x4 cells: kX2, kY2 two samples on. */
struct TxRef {
    static constexpr uint32_t kIntra = 1u << 12, kNone = 1u << 13, kX2 = 1u << 14, kY2 = 1u << 15;
    template <bool LIST>
    static __device__ __forceinline__ int x(uint32_t y) { return (int)(y & 15u) * 4 + (LIST && (y & kX2) ? 2 : 0); }
    template <bool LIST>
    static __device__ __forceinline__ int y(uint32_t y) { return (int)((y >> 4) & 15u) * 4 + (LIST && (y & kY2) ? 2 : 0); }
    static __device__ __forceinline__ int plane(uint32_t y) { return (int)(y >> 8) & 3; }
    static __device__ __forceinline__ int type(uint32_t y) { return (int)(y >> 10) & 3; }
};

/* Place of word e in a permuted buffer. */
__device__ __forceinline__ int tx_word(int e)
{
    const int a = e >> 2;
    return ((a ^ ((a >> 3) & 7)) << 2) | (e & 3);
}

/* List the TXs of blocks [lo, hi), whole CTA: W.tx sorted by size, W.ntx their
 * numbers. layout(b, p, txl, nx, ny): plane p's TXs of block b (0 for a
 * skipped one); type(b, p, txl): the TX type. LIST: the SB runs in list order;
 * only there TXs reach past their block, some past the SB, where the passes
 * clip them. GRID: residuals of intra blocks go to the grid. Barriers inside
 * and at the end. */
template <bool LIST, bool GRID, class S, class L, class Y>
__device__ __forceinline__ void list_txs(S &s, int lo, int hi, int nb, uint32_t num_coeffs, int tid, int nthreads, L layout,
                                         Y type)
{
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthreads >> 5, cnt = min(hi, nb) - lo;
    if (tid < 4) s.ntx[tid] = 0;
    __syncthreads();
    /* a thread a block and plane: its TXs' place among those of their size */
    for (int t = tid; t < 3 * cnt; t += nthreads) {
        const int p = t >= 2 * cnt ? 2 : (t >= cnt ? 1 : 0), b = lo + t - p * cnt;
        int txl, nx, ny;
        layout(s.blk[b], p, txl, nx, ny);
        s.tx_at[p][b] = nx * ny ? (uint16_t)atomicAdd(&s.ntx[txl], nx * ny) : (uint16_t)0;
    }
    __syncthreads();
    const int n32 = s.ntx[3], n16 = s.ntx[2], n8 = s.ntx[1];
    for (int t0 = 0; t0 < 3 * cnt; t0 += nthreads) {
        auto of = [&](int i) { return t0 + i * nwarps + warp; };     /* dealt over the warps */
        auto pair = [&](int t, int &p, int &b) {
            p = t >= 2 * cnt ? 2 : (t >= cnt ? 1 : 0);
            b = lo + t - p * cnt;
        };
        int count = 0;
        if (of(lane) < 3 * cnt) {
            int p, b, txl, nx, ny;
            pair(of(lane), p, b);
            layout(s.blk[b], p, txl, nx, ny);
            count = nx * ny;
        }
        warp_spread(count, lane, [&](int i, int k) {
            int p, b, txl, nx, ny;
            pair(of(i), p, b);
            const auto &m = s.blk[b];
            uint64_t off = m.coeff;
            for (int q = 0; q < p; q++) {
                layout(m, q, txl, nx, ny);
                off += (uint64_t)(nx * ny) << (4 + 2 * txl);
            }
            layout(m, p, txl, nx, ny);
            const int n = 4 << txl, tile = p ? 32 : 64, ty = div_small(k, nx);
            const int x = (p ? m.x >> 1 : m.x) + (k - ty * nx) * n, y = (p ? m.y >> 1 : m.y) + ty * n;
            const int to = s.tx_at[p][b] + k + (txl < 3 ? n32 : 0) + (txl < 2 ? n16 : 0) + (txl < 1 ? n8 : 0);
            const uint64_t co = off + ((uint64_t)k << (4 + 2 * txl));
            const bool none = co + (uint64_t)(n * n) > (uint64_t)num_coeffs || (!LIST && (x + n > tile || y + n > tile));
            if (to < kMaxTasks)
                s.tx[to] = make_uint2((uint32_t)co, (uint32_t)(x >> 2) | (uint32_t)(y >> 2) << 4 | (uint32_t)p << 8 |
                                                        (uint32_t)type(m, p, txl) << 10 |
                                                        (GRID && (m.flags & 1) ? TxRef::kIntra : 0u) | (none ? TxRef::kNone : 0u) |
                                                        (LIST ? (uint32_t)(x & 2) << 13 | (uint32_t)(y & 2) << 14 : 0u));
        });
    }
    __syncthreads();
}

/* Deal the listed TXs to the warps: unit(N, first, count, part) for 32 / N TXs
 * of size N; N = 32 in `parts` parts each. */
template <class F>
__device__ __forceinline__ void deal_txs(const int *ntx, int parts, int warp, int nwarps, F unit)
{
    const int n32 = ntx[3], n16 = ntx[2], n8 = ntx[1], n4 = ntx[0];
    const int u16 = parts * n32, u8 = u16 + ((n16 + 1) >> 1), u4 = u8 + ((n8 + 3) >> 2), end = u4 + ((n4 + 7) >> 3);
    if (n32 + n16 + n8 + n4 > kMaxTasks) return;
    for (int u = warp; u < end; u += nwarps) {
        if (u < u16) {
            unit(std_int<32>(), u / parts, 1, u % parts);
        } else if (u < u8) {
            const int f = (u - u16) * 2;
            unit(std_int<16>(), n32 + f, min(2, n16 - f), 0);
        } else if (u < u4) {
            const int f = (u - u8) * 4;
            unit(std_int<8>(), n32 + n16 + f, min(4, n8 - f), 0);
        } else {
            const int f = (u - u4) * 8;
            unit(std_int<4>(), n32 + n16 + n8 + f, min(8, n4 - f), 0);
        }
    }
}

/* N coefficients of a row, as ints: 16-byte loads where they are aligned. */
template <int N>
__device__ __forceinline__ void row_coeffs(int (&c)[N], const int16_t *row)
{
    if (!((uintptr_t)row & (N == 4 ? 7 : 15))) {
#pragma unroll
        for (int k = 0; k < N; k += (N == 4 ? 4 : 8)) {
            uint32_t w[4] = { 0, 0, 0, 0 };
            if (N == 4) {
                const uint2 v = *reinterpret_cast<const uint2 *>(row);
                w[0] = v.x;
                w[1] = v.y;
            } else {
                const uint4 v = *reinterpret_cast<const uint4 *>(row + k);
                w[0] = v.x;
                w[1] = v.y;
                w[2] = v.z;
                w[3] = v.w;
            }
#pragma unroll
            for (int q = 0; q < (N == 4 ? 2 : 4); q++) {
                c[k + 2 * q] = (int16_t)(w[q] & 0xffffu);
                c[k + 2 * q + 1] = (int)w[q] >> 16;
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) c[k] = row[k];
    }
}

/* Four residuals, each within int16, of a row of an intra block into the
 * grid, of an inter block onto its samples (x a multiple of 4). LIST: onto the
 * samples in either case, clipped to the SB (x even). */
template <bool LIST>
__device__ __forceinline__ void put_residual4(ReconSmem &s, int p, int x, int y, const int (&r)[4], bool intra)
{
    if (LIST) {
        const int tile = p ? 32 : 64;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (x + k >= tile || y >= tile) continue;
            uint8_t &d = p == 0 ? TY(s, x + k, y) : TC(s, p, x + k, y);
            d = (uint8_t)clampi((int)d + r[k], 0, 255);
        }
        return;
    }
    if (intra) {
        *reinterpret_cast<uint2 *>(&s.res[plane_at(p, x, y)]) =
            make_uint2(pack2_s16(r[0], r[1]), pack2_s16(r[2], r[3]));
    } else {
        uint32_t *d = reinterpret_cast<uint32_t *>(p == 0 ? &TY(s, x, y) : &TC(s, p, x, y));
        const uint32_t o = *d;
        *d = pack4_u8((int)(o & 255u) + r[0], (int)((o >> 8) & 255u) + r[1], (int)((o >> 16) & 255u) + r[2], (int)(o >> 24) + r[3]);
    }
}

/* SPEC and FULL: 32 / N TXs by a warp. SPEC (vp9_idct.comp.glsl:666-789):
 * dequantise (DC step at [0][0] only), columns, then rows; FULL: dequantise
 * with the plane's steps (32x32 halved toward zero), rows, then columns, ADST
 * by the TX type, WHT when lossless. Then the rounding shift 4/5/6/6 (none
 * after the WHT); added to an inter block's samples, left in the grid, saturated
 * to int16 (which no sum with a sample notices), for an intra one. */
template <int A, int N, bool LIST>
__device__ __forceinline__ void tx_unit(ReconSmem &s, int32_t *buf, int first, int count, bool staged, unsigned c_base, int lane)
{
    const cvp9_job_t &job = s.jc;
    const int sub = lane / N, i = lane & (N - 1);
    const bool on = sub < count;
    const uint2 tx = s.tx[first + (on ? sub : 0)];
    const int p = TxRef::plane(tx.y), type = TxRef::type(tx.y);
    const bool go = on && !(tx.y & TxRef::kNone);
    const int16_t *X = staged ? s.coef + (tx.x - c_base) : job.coeffs + tx.x;
    wi v[N];
    bool any = false;
    if (go) {
        if (A == CVP9_ARITH_FULL) {
            const int qdc = p ? job.q_dc_uv : job.q_dc, qac = p ? job.q_ac_uv : job.q_ac;
            int c[N];
            row_coeffs<N>(c, X + i * N);
#pragma unroll
            for (int k = 0; k < N; k++) {
                any |= c[k] != 0;
                const int d = c[k] * (i == 0 && k == 0 ? qdc : qac);
                v[k] = wi(N == 32 ? d / 2 : d);
            }
        } else {
#pragma unroll
            for (int k = 0; k < N; k++) {
                const int c = X[k * N + i];
                any |= c != 0;
                v[k] = wi(c) * (k == 0 && i == 0 ? job.q_dc : job.q_ac);
            }
        }
    }
    const uint32_t live = __ballot_sync(0xffffffffu, any);
    if (!live) return;
    const bool mine = N == 32 || ((live >> (sub * N)) & ((1u << (N & 31)) - 1u));
    const bool wht = A == CVP9_ARITH_FULL && N == 4 && job.lossless;
    if (mine) {
        if (any) {
            if (wht) iwht4(v, true);
            else if (A == CVP9_ARITH_FULL) itx1<N>(v, type >= 2);
            else idct_n(v, N);
        }
        if (A == CVP9_ARITH_FULL) {
#pragma unroll
            for (int k = 0; k < N; k += 4)
                *reinterpret_cast<int4 *>(&buf[tx_word(lane * N + k)]) =
                    any ? make_int4(v[k].v, v[k + 1].v, v[k + 2].v, v[k + 3].v) : make_int4(0, 0, 0, 0);
        } else {
#pragma unroll
            for (int k = 0; k < N; k++) buf[tx_word(sub * N * N + k * N + i)] = any ? v[k].v : 0;
        }
    }
    __syncwarp();
    if (mine) {
        const int x = TxRef::x<LIST>(tx.y), y = TxRef::y<LIST>(tx.y);
        const bool intra = tx.y & TxRef::kIntra;
        const int sh = N == 4 ? 4 : (N == 8 ? 5 : 6);
        const int tile = p ? 32 : 64;
        if (A == CVP9_ARITH_FULL) {
#pragma unroll
            for (int k = 0; k < N; k++) v[k] = wi(buf[tx_word(sub * N * N + k * N + i)]);
            if (wht) iwht4(v, false);
            else itx1<N>(v, type & 1);
            uint8_t *d = p == 0 ? &TY(s, x + i, y) : &TC(s, p, x + i, y);
            int16_t *r = s.res + plane_at(p, x + i, y);
            const int dp = p ? kCPitch : kYPitch, rp = p ? 32 : 64;
#pragma unroll
            for (int k = 0; k < N; k++) {
                const int q = wht ? v[k].v : ((int)((unsigned)v[k].v + (1u << (sh - 1)))) >> sh;
                if (LIST && (x + i >= tile || y + k >= tile)) continue;
                if (intra) r[k * rp] = (int16_t)clampi(q, -32768, 32767);
                else d[k * dp] = (uint8_t)clampi((int)d[k * dp] + q, 0, 255);
            }
        } else {
#pragma unroll
            for (int k = 0; k < N; k += 4) {
                const int4 w = *reinterpret_cast<const int4 *>(&buf[tx_word(lane * N + k)]);
                v[k] = wi(w.x);
                v[k + 1] = wi(w.y);
                v[k + 2] = wi(w.z);
                v[k + 3] = wi(w.w);
            }
            idct_n(v, N);
#pragma unroll
            for (int k = 0; k < N; k += 4) {
                int q[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    q[j] = ((int)((unsigned)v[k + j].v + (1u << (sh - 1)))) >> sh;
                put_residual4<LIST>(s, p, x + k, y + i, q, intra);
            }
        }
    }
    __syncwarp();
}

/* SPEC and FULL: every residual of blocks [lo, hi) of the SB. LIST: it runs in
 * list order, the only one for blocks off the 8x8 grid or smaller than their
 * transforms. There SPEC adds an intra block's residual after its prediction,
 * since it may reach past what is predicted. Barriers at both ends. */
template <int A, bool LIST>
__device__ __noinline__ void phase_residual(int lo, int hi, bool staged, unsigned c_base, int sbx, int sby)
{
    ReconSmem &s = smem_as<ReconSmem>();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < kResidGrid / 8; k += kThreads) reinterpret_cast<uint4 *>(s.res)[k] = make_uint4(0u, 0u, 0u, 0u);
    const cvp9_job_t &job = s.jc;
    list_txs<LIST, !(LIST && A == CVP9_ARITH_SPEC)>(s, lo, hi, hi, job.num_coeffs, tid, kThreads,
             [&](const BlkS &b, int p, int &txl, int &nx, int &ny) {
                 txl = b.ptxl[p];
                 nx = b.pnx[p];
                 ny = b.pny[p];
             },
             [&](const BlkS &b, int p, int txl) {
                 return A == CVP9_ARITH_FULL && (b.flags & 1) && p == 0 && !job.lossless && txl < 3 && b.ymode < 10
                            ? (int)c_tx_type[b.ymode] : 0;
             });
    deal_txs(s.ntx, 1, warp, kWarps, [&](auto n, int first, int count, int) {
        tx_unit<A, decltype(n)::value, LIST>(s, s.temp.tx[warp], first, count, staged, c_base, lane);
    });
    __syncthreads();
}

/* REFCPU: the residual of a TX, both passes at once, a warp for 32 / N TXs
 * (N = 32: half the columns of one). Lane i of a TX owns its row i:
 * for each column k with a nonzero coefficient it forms T[i][k] = sum over l
 * of M[l][i] X[l][k] over the nonzero X[l][k], l ascending
 * (vp9_reconstruct.c:31-40), and adds T[i][k] M[k][j] to its O[i][j], k
 * ascending (:42-50) — the reference's operands, order and separate
 * roundings; skipped zero terms add +-0 to a sum that is never -0. Then round
 * half away from zero, saturate to int16, add and clamp (:51-59, :351-360),
 * or leave it in the grid (an intra block's). What bounds it is the FP64 pipe
 * and its latency; a thread per column and then per row, with the basis read
 * from constant memory at addresses that differ from lane to lane, took 56 k
 * cycles a superblock of mixed sizes, this 27 k. */
template <int N>
__device__ __forceinline__ void ref_tx_unit(ReconSmem &s, int first, int count, int half, bool staged, unsigned c_base, int lane)
{
    constexpr int kCols = N == 32 ? 16 : N;
    const int sub = lane / N, i = lane & (N - 1), j0 = half * kCols;
    const bool on = sub < count;
    const uint2 tx = s.tx[first + (on ? sub : 0)];
    const int16_t *X = staged ? s.coef + (tx.x - c_base) : s.jc.coeffs + tx.x;
    const double *M = g_dct + (N == 4 ? 0 : N == 8 ? 16 : N == 16 ? 80 : 336);
    uint32_t nz = 0;                 /* this row's nonzero columns */
    if (on && !(tx.y & TxRef::kNone)) {
        const int16_t *row = X + i * N;
        if (!((uintptr_t)row & (N == 4 ? 7 : 15))) {
            uint32_t w[N / 2];
            if (N == 4) {
                const uint2 v = *reinterpret_cast<const uint2 *>(row);
                w[0] = v.x;
                w[1] = v.y;
            } else {
#pragma unroll
                for (int k = 0; k < N / 8; k++) {
                    const uint4 v = reinterpret_cast<const uint4 *>(row)[k];
                    w[4 * k] = v.x;
                    w[(4 * k + 1) % (N / 2)] = v.y;
                    w[(4 * k + 2) % (N / 2)] = v.z;
                    w[(4 * k + 3) % (N / 2)] = v.w;
                }
            }
#pragma unroll
            for (int k = 0; k < N / 2; k++)
                nz |= ((w[k] & 0xffffu ? 1u : 0u) | (w[k] >> 16 ? 2u : 0u)) << (2 * k);
        } else {
#pragma unroll
            for (int k = 0; k < N; k++) nz |= (row[k] != 0 ? 1u : 0u) << k;
        }
    }
    uint32_t cols = nz;              /* the TX's */
#pragma unroll
    for (int o = 1; o < N; o <<= 1) cols |= __shfl_xor_sync(0xffffffffu, cols, o);
    const bool any = cols != 0;
    double acc[kCols];
#pragma unroll
    for (int j = 0; j < kCols; j++) acc[j] = 0.0;
    while (__any_sync(0xffffffffu, cols != 0)) {
        const int k = cols ? __ffs(cols) - 1 : 0;
        uint32_t rows = __ballot_sync(0xffffffffu, cols && ((nz >> k) & 1u));
        if (N < 32) rows = (rows >> (sub * N)) & ((1u << (N & 31)) - 1u);
        if (cols) {
            double t = 0.0;
            while (rows) {
                const int l = __ffs(rows) - 1;
                rows &= rows - 1;
                t = __dadd_rn(t, __dmul_rn(__ldg(M + l * N + i), (double)X[l * N + k]));
            }
            const double2 *b = reinterpret_cast<const double2 *>(M + k * N + j0);
#pragma unroll
            for (int j = 0; j < kCols / 2; j++) {
                const double2 m = __ldg(b + j);
                acc[2 * j] = __dadd_rn(acc[2 * j], __dmul_rn(t, m.x));
                acc[2 * j + 1] = __dadd_rn(acc[2 * j + 1], __dmul_rn(t, m.y));
            }
            cols &= cols - 1;
        }
    }
    if (!any) return;
    const int px = TxRef::x<false>(tx.y) + j0, py = TxRef::y<false>(tx.y) + i;
    const bool intra = tx.y & TxRef::kIntra;
#pragma unroll
    for (int j = 0; j < kCols; j += 4) {
        int r[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double v = acc[j + q];
            r[q] = clampi(__double2int_rz(__dadd_rn(v, v >= 0.0 ? 0.5 : -0.5)), -32768, 32767);
        }
        put_residual4<false>(s, 0, px + j, py, r, intra);
    }
}

/* REFCPU: every residual of blocks [lo, hi) of the SB. Barriers at both ends. */
__device__ __noinline__ void phase_residual_ref(int lo, int hi, bool staged, unsigned c_base)
{
    ReconSmem &s = smem_as<ReconSmem>();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < kResidGrid / 8; k += kThreads) reinterpret_cast<uint4 *>(s.res)[k] = make_uint4(0u, 0u, 0u, 0u);
    list_txs<false, true>(s, lo, hi, hi, s.jc.num_coeffs, tid, kThreads,
             [&](const BlkS &b, int p, int &txl, int &nx, int &ny) {
                 txl = b.ptxl[p];
                 nx = b.pnx[p];
                 ny = b.pny[p];
             },
             [](const BlkS &, int, int) { return 0; });
    deal_txs(s.ntx, 2, warp, kWarps, [&](auto n, int first, int count, int part) {
        ref_tx_unit<decltype(n)::value>(s, first, count, part, staged, c_base, lane);
    });
    __syncthreads();
}

/* The intra tasks of the SB's nb blocks, their levels, the sorted quads. */
template <int A>
__device__ __noinline__ void phase_plan(int nb, int sbx, int sby)
{
    ReconSmem &s = smem_as<ReconSmem>();
    const cvp9_job_t &job = s.jc;
    IntraWork &W = s.temp.w;
    const int tid = threadIdx.x;
    const bool mine = tid < nb && (s.blk[tid].flags & 1);
    intra_fill_cols(recon_view(s), tid, kThreads);
    int ntask;
    if (A == CVP9_ARITH_FULL) {
        const int at = cta_scan1(s, mine ? intra_tx_count(s.blk[tid], job, sbx, sby) : 0, &ntask);
        ntask = min(ntask, kMaxTasks);
        if (tid < nb) s.first[tid] = (uint16_t)at;
        for (int i = tid; i < kMaxTasks; i += kThreads) W.own[i] = 0;
        if (tid < 96) (&W.prow[0][0])[tid] = 0u;
        __syncthreads();
        for (int t = tid; t < ntask; t += kThreads) {
            const int b = find_base(s.first, nb, t);
            intra_tx_task(W, s.blk[b], job, sbx, sby, t - s.first[b], t, true);
        }
        __syncthreads();
        intra_tx_levels(W, ntask, tid, kThreads);
    } else {
        /* a block's three planes share its level */
        const int at = cta_scan1(s, mine ? 3 : 0, &ntask);
        if (tid < 96) (&W.prow[0][0])[tid] = 0u;
        if (tid < nb) W.own[tid] = mine ? (uint16_t)at : (uint16_t)0xFFFF;
        __syncthreads();
        LvlTask lt[1];
        const bool have[1] = { mine };
        if (mine) {
            const BlkS &b = s.blk[tid];
            int c0x, c1x, c0y, c1y;
            block_cells<A>(b, job, sbx, sby, c0x, c1x, c0y, c1y);
            lt[0].set(W.prow[0], W.pcol[0], c0x, c1x, c0y, c1y, (b.x + b.cw - 1) >> 2);
        }
        __syncthreads();
        intra_levels<1>(lt, have);
        if (mine) intra_block_tasks<A>(W, s.blk[tid], job, sbx, sby, at, max(0, lt[0].level));
    }
    __syncthreads();
    intra_sort<A, uint8_t>(W, s.cell, ntask, tid, kThreads);
}

/* Intra block b on its own, its residual in the grid. */
template <int A>
__device__ __noinline__ void phase_ordered(int b, int sbx, int sby)
{
    ReconSmem &s = smem_as<ReconSmem>();
    const cvp9_job_t &job = s.jc;
    IntraWork &W = s.temp.w;
    const int tid = threadIdx.x;
    const IntraView<uint8_t> V = recon_view(s);
    intra_fill_cols(V, tid, kThreads);
    if (A == CVP9_ARITH_FULL) {
        const int n = min(intra_tx_count(s.blk[b], job, sbx, sby), kMaxTasks);
        for (int k = tid; k < n; k += kThreads) intra_tx_task(W, s.blk[b], job, sbx, sby, k, k, false);
        if (tid == 0) W.ntask = n;
    } else if (tid == 0) {
        intra_block_tasks<A>(W, s.blk[b], job, sbx, sby, 0, 0);
        W.ntask = 3;
    }
    __syncthreads();
    intra_run_ordered<A, 255, uint8_t>(W, V, W.ntask, tid, kThreads);
    __syncthreads();
}

/* Wait (bounded) for the neighbour SBs whose samples are read (intra_needs
 * bits), a lane a neighbour, then load the halo. */
template <class S, class T>
__device__ __forceinline__ void wait_halo(S &s, const IntraView<T> &V, unsigned need, int sb, bool full, int fill_a,
                                          int fill_l, int tid, int nthreads)
{
    const cvp9_job_t &job = s.jc;
    const int sbr = sb / job.sb_cols, sbc = sb - sbr * job.sb_cols;
    const bool have_l = full ? sbc * 8 > full_tile_start(sbc * 8, job.mi_cols, job.log2_tile_cols) : sbc > 0;
    if (tid < 3 && ((need >> tid) & 1u)) {
        const int dc = tid == 1 ? 0 : 1, dr = tid == 0 ? 0 : 1;
        if (sbc >= dc && sbr >= dr && (have_l || tid == 1) &&
            !wait_flag(job.sb_done + sb - dr * job.sb_cols - dc, job.epoch))
            atomicOr(job.status, (unsigned)CVP9_JOB_TIMEOUT);
    }
    __syncthreads();
    intra_halo<T>(V, job, sbc * 64, sbr * 64, sbr > 0, have_l, need, fill_a, fill_l, tid, nthreads);
    __syncthreads();
}

template <int A>
__device__ __noinline__ void phase_neighbours(unsigned need, int sb)
{
    ReconSmem &s = smem_as<ReconSmem>();
    constexpr int fill_a = A == CVP9_ARITH_SPEC ? 128 : 127, fill_l = A == CVP9_ARITH_FULL ? 129 : fill_a;
    wait_halo<ReconSmem, uint8_t>(s, recon_view(s), need, sb, A == CVP9_ARITH_FULL, fill_a, fill_l, threadIdx.x, kThreads);
}

/* The samples that the neighbours read (right column, bottom row; 256
 * threads, one each), then the superblock's flag: its release takes in what
 * the other threads wrote before the barrier. */
template <class T, class F>
__device__ __forceinline__ void publish(const cvp9_job_t &job, int sb, int sbx, int sby, int tid, F sample)
{
    const int vw = min(64, job.W - sbx), vh = min(64, job.H - sby);
    const int p = tid < 128 ? 0 : 1 + ((tid >> 5) & 1), n = p ? 32 : 64;
    const bool row = tid < 128 ? tid >= 64 : tid >= 192;
    const int k = p ? tid & 31 : tid & 63;
    const int pw = p ? job.CW : job.W, ph = p ? job.CH : job.H;
    const int X = (p ? sbx >> 1 : sbx) + (row ? k : n - 1), Y = (p ? sby >> 1 : sby) + (row ? n - 1 : k);
    if (X < pw && Y < ph && (row ? vh == 64 : vw == 64))
        reinterpret_cast<T *>(job.out)[(p ? (size_t)job.W * job.H + (size_t)(p - 1) * job.CW * job.CH : 0) +
                                       (size_t)Y * pw + X] = sample(p, row ? k : n - 1, row ? n - 1 : k);
    __syncthreads();
    if (tid == 0) st_release(job.sb_done + sb, job.epoch);
}

__device__ __forceinline__ void recon_publish(ReconSmem &s, int sb, int sbx, int sby, int tid)
{
    publish<uint8_t>(s.jc, sb, sbx, sby, tid, [&](int p, int x, int y) { return p == 0 ? TY(s, x, y) : TC(s, p, x, y); });
}

/* The neighbours' samples, level by level, the superblock's own: what the
 * chain of superblocks waits for, in one function (apart, they saved and
 * restored the caller's registers in between; with that, a halo read in two
 * rounds and sleeps of 256 ns between looks at a flag, three 1080p SPEC
 * pictures took 0.70 ms, with this 0.65). */
template <int A>
__device__ __noinline__ void phase_intra(unsigned need, int sb, int sbx, int sby)
{
    ReconSmem &s = smem_as<ReconSmem>();
    constexpr int fill_a = A == CVP9_ARITH_SPEC ? 128 : 127, fill_l = A == CVP9_ARITH_FULL ? 129 : fill_a;
    wait_halo<ReconSmem, uint8_t>(s, recon_view(s), need, sb, A == CVP9_ARITH_FULL, fill_a, fill_l, threadIdx.x, kThreads);
    intra_run<A, 255, uint8_t>(s.temp.w, recon_view(s), threadIdx.x, kThreads);
    recon_publish(s, sb, sbx, sby, threadIdx.x);
}

template <int A>
__global__ void __launch_bounds__(kThreads, 3) k_recon(const cvp9_job_t *__restrict__ jobs,
                                                   const uint32_t *__restrict__ tickets,
                                                   uint32_t n_tickets, uint32_t *ticket_counter,
                                                   const uint32_t *__restrict__ n_dev)
{
    grid_dependency_wait();
    /* with the inter fast path the general ticket count is known on the device */
    if (n_dev) n_tickets = *n_dev;
    ReconSmem &s = smem_as<ReconSmem>();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const cvp9_job_t &job = s.jc;     /* valid after the reset barrier */

    for (;;) {
        __syncthreads();
        if (tid == 0) s.ticket = (int)atomicAdd(ticket_counter, 1u);
        __syncthreads();
        const int ticket = s.ticket;
        if (ticket >= (int)n_tickets) return;
        const uint32_t code = tickets[ticket];
        const cvp9_job_t *gj = jobs + (code >> 20);
        {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(gj);
            uint32_t *dst = reinterpret_cast<uint32_t *>(&s.jc);
            for (int i = tid; i < (int)(sizeof(cvp9_job_t) / 4); i += kThreads) dst[i] = src[i];
        }
        const int sb = (int)(code & 0xFFFFFu);
        const int g_sb_cols = gj->sb_cols;
        const int sbr = sb / g_sb_cols, sbc = sb - sbr * g_sb_cols;
        const int sbx = sbc * 64, sby = sbr * 64;
        const uint32_t *rg = gj->sb_range + 4 * sb;
        const uint32_t start = rg[0], end = rg[1], groups = rg[2];
        const uint32_t g_nblocks = gj->num_blocks;
        const bool layout_bad = (*(volatile uint32_t *)gj->status & CVP9_JOB_BAD_BLOCK) != 0;
        bool bad = groups > 1 || end < start || end > g_nblocks ||
                   (groups && end - start > (uint32_t)kMaxBlocks);
        int nb = (groups && !bad && !layout_bad) ? (int)(end - start) : 0;

        /* reset per-SB state, tile = 128 */
        {
            uint4 *t4 = reinterpret_cast<uint4 *>(s.ty);
            const uint4 fill = make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);
            for (int i = tid; i < (kTyBytes + 2 * kTcBytes) / 16; i += kThreads) t4[i] = fill;
        }
        for (int i = tid; i < 256; i += kThreads) s.cell[i] = 0;
        if (tid < 16) s.rows[tid] = 0;
        if (tid == 0) { s.c_lo = 0xFFFFFFFFu; s.c_hi = 0u; s.needs = 0u; }
        __syncthreads();

        /* 1. load and re-check blocks (a block must sit inside this SB,
         * 4-aligned, 4..64 px, tx_size <= 3; sub-8x8 blocks on the 8x8 MI
         * grid), then mark the 4x4 cells each one covers */
        bool my_intra = false, my_seq = false, my_bad = false;
        BlkS mb;
        int nch = 0;
        if (tid < nb) {
            vp9_macroblock_info_t g = job.blocks[start + tid];
            int lx = (int)g.x - sbx, ly = (int)g.y - sby;
            my_bad = lx < 0 || ly < 0 || (lx & 3) || (ly & 3) || (g.width & 3) || (g.height & 3) ||
                     g.width < 4 || g.height < 4 || lx + g.width > 64 || ly + g.height > 64 ||
                     g.x >= job.W || g.y >= job.H || g.tx_size > 3 ||
                     ((g.width < 8 || g.height < 8) && ((lx & 7) || (ly & 7)));
            if (my_bad) { lx = 0; ly = 0; g.width = 4; g.height = 4; g.tx_size = 0; }
            mb.x = (uint8_t)lx;
            mb.y = (uint8_t)ly;
            mb.w = g.width;
            mb.h = g.height;
            int cw = g.width, ch = g.height;
            if (g.x + cw > job.W) cw = job.W - g.x;
            if (g.y + ch > job.H) ch = job.H - g.y;
            mb.cw = (uint8_t)cw;
            mb.ch = (uint8_t)ch;
            mb.txl = g.tx_size;
            mb.flags = (uint8_t)((g.is_intra ? 1 : 0) | (g.skip ? 2 : 0));
            mb.ymode = g.y_mode;
            mb.uvmode = g.uv_mode;
            mb.ref0 = g.ref_frame[0];
            mb.mvx = g.mv[0][0];
            mb.mvy = g.mv[0][1];
            mb.ref1 = 0;
            mb.mv1x = g.mv[1][0];
            mb.mv1y = g.mv[1][1];
            mb.coeff = g.coeff_offset;
            if (A == CVP9_ARITH_FULL) {
                /* the block's whole MI for a sub-8x8 block (one MV, one
                 * mode); a second reference */
                if (g.width < 8 || g.height < 8) {
                    mb.cw = (uint8_t)min(8, job.W - (int)g.x);
                    mb.ch = (uint8_t)min(8, job.H - (int)g.y);
                }
                if (!g.is_intra) mb.ref1 = g.ref_frame[1];
            }
            if (A != CVP9_ARITH_REFCPU) {
                /* TXs that do not tile their block, or whose chroma TXs
                 * straddle 4x4 cells, share samples or cells with others':
                 * such a superblock runs in list order */
                const bool sub8 = g.width < 8 || g.height < 8;
                const int ew = sub8 ? 8 : g.width, eh = sub8 ? 8 : g.height, n = 4 << g.tx_size;
                const int m = min(n, 4 << max_tx_for(max(4, ew / 2), max(4, eh / 2)));
                my_seq = ((ew | eh) & (n - 1)) || (!sub8 && (((ew | eh) >> 1) & (m - 1))) || ((lx | ly) & 7);
            }
            residual_layout<A>(mb, job, g.x, g.y);
            s.blk[tid] = mb;
            my_intra = g.is_intra != 0;
            nch = my_intra ? 0 : block_chunks<A>(mb);

        }
        if (__syncthreads_or(my_bad)) {
            /* leave the tile at 128 and flag the frame */
            if (tid == 0) atomicOr(job.status, (unsigned)CVP9_JOB_BAD_BLOCK);
            nb = 0;
            my_intra = my_seq = false;
        }
        {
            /* span of coefficients the residual pass reads */
            unsigned lo = 0xFFFFFFFFu, hi = 0u;
            if (tid < nb) {
                uint64_t n = 0;
#pragma unroll
                for (int q = 0; q < 3; q++) n += (uint64_t)(mb.pnx[q] * mb.pny[q]) * (uint64_t)(16 << (2 * mb.ptxl[q]));
                uint64_t e = (uint64_t)mb.coeff + n;
                if (n) { lo = mb.coeff; hi = e > 0xFFFFFFFFull ? 0xFFFFFFFFu : (unsigned)e; }
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (lane == 0) { atomicMin(&s.c_lo, lo); atomicMax(&s.c_hi, hi); }
        }
        int c0x = 0, c1x = 0, c0y = 0, c1y = 0;
        if (tid < nb) {
            block_cells<A>(mb, job, sbx, sby, c0x, c1x, c0y, c1y);
            my_seq |= claim_cells(s.rows, c0x, c1x, c0y, c1y);
        }
        {
            const unsigned need = __reduce_or_sync(0xffffffffu, tid < nb && my_intra ? intra_needs(mb.x, mb.y) : 0u);
            if (lane == 0 && need) atomicOr(&s.needs, need);
        }
        const int any_intra = __syncthreads_or(my_intra);
        bool seq = __syncthreads_or(my_seq) != 0;

        /* stage the SB's coefficient span in shared memory with 16-byte async
         * copies */
        const unsigned c_lo = s.c_lo, c_hi = s.c_hi;
        const unsigned c_base = c_lo & ~7u;
        const bool staged = c_hi > c_lo && c_hi <= job.num_coeffs && c_hi - c_base <= (unsigned)kCoefStage;
        const bool c_vec = !((uintptr_t)job.coeffs & 15);
        constexpr int kStageIt = kCoefStage / 8 / kThreads;
#pragma unroll
        for (int k = 0; k < kStageIt; k++) {
            unsigned e = c_base + 8u * (unsigned)(tid + k * kThreads);
            if (!staged || e >= c_hi) continue;
            if (c_vec && e + 8 <= job.num_coeffs) cp_async16(&s.coef[e - c_base], job.coeffs + e);
            else for (unsigned q = e; q < e + 8 && q < c_hi; q++) s.coef[q - c_base] = job.coeffs[q];
        }
        cp_async_commit();

        /* 2. an intra block reads the blocks above it, to its left and at its
         * corner: where one of them comes later in the list, the superblock
         * runs in list order (as it does when blocks overlap) */
        if (any_intra) {
            int n = 0;
            if (lane * kWarps + warp < nb) {      /* the blocks dealt over the warps */
                int x0, x1, y0, y1;
                block_cells<A>(s.blk[lane * kWarps + warp], job, sbx, sby, x0, x1, y0, y1);
                n = (x1 - x0 + 1) * (y1 - y0 + 1);
            }
            warp_spread(n, lane, [&](int i, int k) {
                const int b = i * kWarps + warp;
                int x0, x1, y0, y1;
                block_cells<A>(s.blk[b], job, sbx, sby, x0, x1, y0, y1);
                own_cell(s.cell, b, x0, x1, y0, k);
            });
            __syncthreads();
            bool late = false;
            if (tid < nb && my_intra) {
                const int x1 = (mb.x + mb.cw - 1) >> 2, y1 = (mb.y + mb.ch - 1) >> 2;
                if (c0y > 0) for (int cx = max(0, c0x - 1); cx <= x1; cx++) late |= s.cell[(c0y - 1) * 16 + cx] > tid;
                if (c0x > 0) for (int cy = c0y; cy <= y1; cy++) late |= s.cell[cy * 16 + c0x - 1] > tid;
            }
            seq |= __syncthreads_or(late) != 0;
        }
        /* inter chunks in list order: offsets, and chunk -> block */
        {
            int n;
            const int at = cta_scan1(s, tid < nb ? nch : 0, &n);
            if (tid < nb) s.chunk_off[tid] = (uint16_t)at;
            if (tid == 0) s.chunk_off[nb] = (uint16_t)n;
        }
        __syncthreads();
        {
            const int mine = lane * kWarps + warp;
            warp_spread(mine < nb ? s.chunk_off[mine + 1] - s.chunk_off[mine] : 0, lane, [&](int i, int k) {
                const int b = i * kWarps + warp, c = s.chunk_off[b] + k;
                if (c < 256) s.chunk_blk[c] = (uint8_t)b;
            });
        }
        __syncthreads();

        if (!seq) {
            /* 3. everything that reads no neighbour: inter predictions, then
             * the residual of every TX, added to the inter blocks and left in
             * the grid for the intra ones */
            const int n_chunks = min((int)s.chunk_off[nb], 256);
            if (n_chunks) phase_inter<A>(-1, n_chunks, sbx, sby);
            cp_async_wait_all();
            if (A == CVP9_ARITH_REFCPU) phase_residual_ref(0, nb, staged, c_base);
            else phase_residual<A, false>(0, nb, staged, c_base, sbx, sby);
            if (any_intra) {
                /* 4. the intra tasks and their levels; 5. the neighbours'
                 * samples, then level by level */
                phase_plan<A>(nb, sbx, sby);
                phase_intra<A>(s.needs, sb, sbx, sby);
            }
        } else {
            /* list order, block by block */
            cp_async_wait_all();
            if (A == CVP9_ARITH_SPEC)        /* what phase_ordered adds there */
                for (int k = tid; k < kResidGrid / 8; k += kThreads) reinterpret_cast<uint4 *>(s.res)[k] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            if (any_intra) phase_neighbours<A>(7u, sb);
            for (int b = 0; b < nb; b++) {
                const bool intra = s.blk[b].flags & 1;
                if (!intra) phase_inter<A>(b, block_chunks<A>(s.blk[b]), sbx, sby);
                if (A == CVP9_ARITH_SPEC && intra) phase_ordered<A>(b, sbx, sby);
                if (A == CVP9_ARITH_REFCPU) phase_residual_ref(b, b + 1, staged, c_base);
                else phase_residual<A, true>(b, b + 1, staged, c_base, sbx, sby);
                if (A != CVP9_ARITH_SPEC && intra) phase_ordered<A>(b, sbx, sby);
            }
        }

        /* 6. the samples the neighbours read first, with the SB's flag, then
         * the whole tile (the same values again there) */
        {
            if (seq || !any_intra) recon_publish(s, sb, sbx, sby, tid);
            if (tid == 0 && bad)
                atomicOr(job.status, (unsigned)CVP9_JOB_BAD_ORDER |
                                     ((groups && end >= start && end - start > (uint32_t)kMaxBlocks) ? (unsigned)CVP9_JOB_TOO_MANY : 0u));
            recon_write(s, sbx, sby, tid);
        }
    }
}

/* ── Inter-only superblocks: one warp per SB ─────────────────────────────
 *
 * Most superblocks of an inter frame hold inter blocks only; nothing in them
 * depends on another superblock of the same frame. k_inter gives each such
 * SB to one warp, which predicts and adds the residual in a per-warp tile
 * and writes the tile once, with no CTA barriers and no dependency analysis.
 * An SB the warp cannot take (an intra block, a block outside the supported
 * domain, overlapping blocks, uncovered 4x4 cells, more than 64 blocks) is
 * marked general and left to k_recon, which k_compact feeds with the general
 * tickets in their original SB-diagonal order. k_inter releases the done
 * flag of every SB it finishes, so general SBs that wait on a neighbour see
 * it done. The arithmetic is the REFCPU profile of k_recon, term for term. */

namespace {

constexpr int kFastWarps = 4;                     /* SBs per CTA */

/* One block, 16 bytes. geo: x/4 | y/4 << 4 | clamped cw << 8 | ch << 15 |
 * reference slot << 22 (REFCPU: pool slot, 15 none; SPEC: LAST/GOLDEN/ALTREF
 * 0..2) | tx_size << 26 | skip << 28. ext (SPEC): luma TXs per row | per
 * column << 5 | chroma TXs per row << 10 | per column << 14 | chroma
 * tx_size << 18. */
struct FastBlk {
    uint32_t geo;
    uint32_t mv;      /* mv[0]: col in the low half, row in the high half (1/8 pel) */
    uint32_t coeff;   /* first coefficient of the block */
    uint32_t ext;
};

__device__ __forceinline__ int fb_x(const FastBlk &b) { return (int)(b.geo & 0xfu) << 2; }
__device__ __forceinline__ int fb_y(const FastBlk &b) { return (int)((b.geo >> 4) & 0xfu) << 2; }
__device__ __forceinline__ int fb_cw(const FastBlk &b) { return (int)((b.geo >> 8) & 0x7fu); }
__device__ __forceinline__ int fb_ch(const FastBlk &b) { return (int)((b.geo >> 15) & 0x7fu); }
__device__ __forceinline__ int fb_slot(const FastBlk &b) { return (int)((b.geo >> 22) & 0xfu); }
__device__ __forceinline__ int fb_txl(const FastBlk &b) { return (int)((b.geo >> 26) & 3u); }
__device__ __forceinline__ bool fb_skip(const FastBlk &b) { return (b.geo >> 28) & 1u; }

/* Tile pitches: 72 and 40 bytes put eight consecutive rows in eight
 * different bank groups (a 64-byte pitch maps rows r and r+2 together). */
constexpr int kFY = 72, kFC = 40;

struct __align__(16) FastSmem {                   /* one per warp; 16-byte vector access */
    uint8_t  ty[64 * kFY];                        /* luma tile */
    uint8_t  tu[32 * kFC];
    uint8_t  tv[32 * kFC];
    union {
        int16_t  coef[1056];                      /* residual: the TXs in flight, (N*N + 2) apart */
        uint32_t cells[8];                        /* set-up: 4x4-cell occupancy, 2 cell rows per word */
    };
    FastBlk  blk[64];
    union {
        struct {                                  /* prediction */
            uint16_t choff[65];                   /* first chunk of each block */
            uint8_t  chblk[128];                  /* chunk -> block */
        };
        struct {                                  /* residual, per TX size */
            uint16_t txoff[65];                   /* first TX of each block */
            uint8_t  txblk[256];                  /* TX -> block */
        };
    };
};

static_assert(sizeof(FastSmem) % 16 == 0, "per-warp tiles must stay 16-byte aligned");
static_assert(sizeof(FastSmem) * kFastWarps + 1024 <= 233472 / 5, "five CTAs of k_inter per SM");
static_assert(offsetof(FastSmem, coef) % 16 == 0 && offsetof(FastSmem, tu) % 16 == 0 &&
              offsetof(FastSmem, tv) % 16 == 0, "vector-accessed members must be 16-byte aligned");

/* 16 bytes from an 8-byte-aligned shared-memory address */
__device__ __forceinline__ uint4 ld_smem16(const uint8_t *p)
{
    const uint2 a = reinterpret_cast<const uint2 *>(p)[0], b = reinterpret_cast<const uint2 *>(p)[1];
    return make_uint4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ int warp_incl_scan(int x, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

/* The same nine bytes from two 8-byte reads of the aligned 16 bytes around
 * them (p & 7 <= 7, so r[0..8] always lie inside; callers keep the span
 * inside the buffer): fewer L1 requests than three word reads. */
__device__ __forceinline__ void ld9d(const uint8_t *p, uint32_t &lo, uint32_t &mid, uint32_t &hi)
{
    const uintptr_t a = (uintptr_t)p;
    const uint2 *q = reinterpret_cast<const uint2 *>(a & ~(uintptr_t)7);
    const uint2 v0 = __ldg(q), v1 = __ldg(q + 1);
    const unsigned o = (unsigned)(a & 7), sh = 8u * (o & 3u);
    /* words w[o/4 .. o/4 + 2] of the four, by whether o >= 4 */
    const bool up = o >= 4;
    const uint32_t w0 = up ? v0.y : v0.x, w1 = up ? v1.x : v0.y, w2 = up ? v1.y : v1.x;
    lo = __funnelshift_r(w0, w1, sh);
    mid = __funnelshift_r(w1, w2, sh);
    hi = w2 >> sh;
}

/* The same nine bytes with every sample clamped into [0, pw-1] x [0, ph-1]. */
__device__ __forceinline__ void ld9c(const uint8_t *plane, int pw, int ph, int x0, int y,
                                     uint32_t &lo, uint32_t &mid, uint32_t &hi)
{
    const uint8_t *row = plane + (size_t)clampi(y, 0, ph - 1) * pw;
    uint32_t v[3] = { 0, 0, 0 };
#pragma unroll
    for (int x = 0; x < 9; x++) v[x >> 2] |= (uint32_t)__ldg(row + clampi(x0 + x, 0, pw - 1)) << (8 * (x & 3));
    lo = v[0]; mid = v[1]; hi = v[2];
}

__device__ __forceinline__ void ld5w(const uint8_t *p, uint32_t &lo, uint32_t &hi)
{
    const uintptr_t a = (uintptr_t)p;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    const unsigned sh = 8u * (unsigned)(a & 3);
    const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1);
    lo = __funnelshift_r(w0, w1, sh);
    hi = w1 >> sh;
}

/* five chroma bytes, clamped into [0, cw-1] x [0, ch-1] (cw, ch may be 0) */
__device__ __forceinline__ void ld5c(const uint8_t *plane, int stride, int cw, int ch, int x0, int y,
                                     uint32_t &lo, uint32_t &hi)
{
    const int xm = cw > 0 ? cw - 1 : 0, ym = ch > 0 ? ch - 1 : 0;
    const uint8_t *row = plane + (size_t)clampi(y, 0, ym) * stride;
    uint32_t v[2] = { 0, 0 };
#pragma unroll
    for (int x = 0; x < 5; x++) v[x >> 2] |= (uint32_t)__ldg(row + clampi(x0 + x, 0, xm)) << (8 * (x & 3));
    lo = v[0]; hi = v[1];
}

/* Two-stage bilinear of vp9_reconstruct.c:105-128 on two samples at once:
 * (a (8-f) + b f + 4) >> 3 per 16-bit field; every intermediate is below
 * 2^11, so fields never carry into each other. */
__device__ __forceinline__ uint32_t bil2(uint32_t a, uint32_t b, uint32_t wa, uint32_t wb)
{
    return ((a * wa + b * wb + 0x00040004u) >> 3) & 0x00ff00ffu;
}

/* Eight luma samples of one row from rows r (lo0 mid0 hi0) and r+1. */
__device__ __forceinline__ void bilinear8(uint32_t lo0, uint32_t mid0, uint32_t hi0,
                                          uint32_t lo1, uint32_t mid1, uint32_t hi1,
                                          int fx, int fy, uint32_t &o0, uint32_t &o1)
{
    const uint32_t wx = 8u - (uint32_t)fx, ux = (uint32_t)fx, wy = 8u - (uint32_t)fy, uy = (uint32_t)fy;
    /* fields (r[2k], r[2k+1]) and (r[2k+1], r[2k+2]) */
    const uint32_t s0 = __funnelshift_r(lo0, mid0, 8), t0 = __funnelshift_r(mid0, hi0, 8);
    const uint32_t s1 = __funnelshift_r(lo1, mid1, 8), t1 = __funnelshift_r(mid1, hi1, 8);
    const uint32_t h00 = bil2(__byte_perm(lo0, 0, 0x4140), __byte_perm(s0, 0, 0x4140), wx, ux);
    const uint32_t h01 = bil2(__byte_perm(lo0, 0, 0x4342), __byte_perm(s0, 0, 0x4342), wx, ux);
    const uint32_t h02 = bil2(__byte_perm(mid0, 0, 0x4140), __byte_perm(t0, 0, 0x4140), wx, ux);
    const uint32_t h03 = bil2(__byte_perm(mid0, 0, 0x4342), __byte_perm(t0, 0, 0x4342), wx, ux);
    const uint32_t h10 = bil2(__byte_perm(lo1, 0, 0x4140), __byte_perm(s1, 0, 0x4140), wx, ux);
    const uint32_t h11 = bil2(__byte_perm(lo1, 0, 0x4342), __byte_perm(s1, 0, 0x4342), wx, ux);
    const uint32_t h12 = bil2(__byte_perm(mid1, 0, 0x4140), __byte_perm(t1, 0, 0x4140), wx, ux);
    const uint32_t h13 = bil2(__byte_perm(mid1, 0, 0x4342), __byte_perm(t1, 0, 0x4342), wx, ux);
    const uint32_t v0 = bil2(h00, h10, wy, uy), v1 = bil2(h01, h11, wy, uy);
    const uint32_t v2 = bil2(h02, h12, wy, uy), v3 = bil2(h03, h13, wy, uy);
    o0 = __byte_perm(v0, v1, 0x6420);
    o1 = __byte_perm(v2, v3, 0x6420);
}

/* Four chroma samples from rows r (lo0 hi0: bytes 0..4) and r+1. */
__device__ __forceinline__ uint32_t bilinear4(uint32_t lo0, uint32_t hi0, uint32_t lo1, uint32_t hi1,
                                              int fx, int fy)
{
    const uint32_t wx = 8u - (uint32_t)fx, ux = (uint32_t)fx, wy = 8u - (uint32_t)fy, uy = (uint32_t)fy;
    const uint32_t s0 = __funnelshift_r(lo0, hi0, 8), s1 = __funnelshift_r(lo1, hi1, 8);
    const uint32_t h00 = bil2(__byte_perm(lo0, 0, 0x4140), __byte_perm(s0, 0, 0x4140), wx, ux);
    const uint32_t h01 = bil2(__byte_perm(lo0, 0, 0x4342), __byte_perm(s0, 0, 0x4342), wx, ux);
    const uint32_t h10 = bil2(__byte_perm(lo1, 0, 0x4140), __byte_perm(s1, 0, 0x4140), wx, ux);
    const uint32_t h11 = bil2(__byte_perm(lo1, 0, 0x4342), __byte_perm(s1, 0, 0x4342), wx, ux);
    return __byte_perm(bil2(h00, h10, wy, uy), bil2(h01, h11, wy, uy), 0x6420);
}

/* One lane's share of a prediction pass, split so that a warp can issue the
 * reads of two passes before computing either. */
struct FastLuma {
    uint8_t *d;
    int lw, fx, fy;
    bool act, ref;
    uint32_t lo0, mid0, hi0, lo1, mid1, hi1;
};

struct FastChroma {
    uint8_t *d;
    int clw, fx, fy;
    bool act, ref;
    uint32_t lo0, hi0, lo1, hi1;
};

/* Chunk k of block b: its 8x8 luma and 4x4 chroma regions (clipped). */
template <class S>
__device__ __forceinline__ void fast_chunk(const S &w, int c, FastBlk &fb, int &lx0, int &ly0, int &lw,
                                           int &lh, int &cx0, int &cy0, int &clw, int &clh)
{
    const int b = w.chblk[c];
    fb = w.blk[b];
    const int bx = fb_x(fb), by = fb_y(fb), cw = fb_cw(fb), ch = fb_ch(fb);
    const int k = c - w.choff[b];
    const int nx = (cw + 7) >> 3;
    const int ccy = nx == 1 ? k : div_small(k, nx), ccx = k - ccy * nx;
    lx0 = bx + ccx * 8;
    ly0 = by + ccy * 8;
    lw = min(8, cw - ccx * 8);
    lh = min(8, ch - ccy * 8);
    cx0 = (bx >> 1) + ccx * 4;
    cy0 = (by >> 1) + ccy * 4;
    clw = min(4, ((cw + 1) >> 1) - ccx * 4);
    clh = min(4, ((ch + 1) >> 1) - ccy * 4);
}

/* Where a superblock's prediction lands: its luma and chroma origins and
 * pitches (the warp's shared tiles, or the frame itself), and the extent
 * inside the frame from those origins (luma vw x vh, chroma cvw x cvh):
 * SPEC TXs follow the MI grid and can reach past the frame edge, where
 * nothing is written. */
struct PredDst {
    uint8_t *y, *u, *v;
    int      py, pc;
    int      vw, vh, cvw, cvh;
};

/* One lane's luma row (chunk c, row lane%8) and chroma row (plane
 * (lane/4)%2, row lane%4) of chunk c: geometry, reference and MV decoded
 * once for both, reads issued, nothing computed yet. */
template <class S>
__device__ __forceinline__ void fast_pred_issue(const S &w, const PredDst &D, const cvp9_job_t &job, int c, int lane,
                                                int nchunks, int sbx, int sby, FastLuma &J, FastChroma &K)
{
    /* Each lane reads one reference row of its chunk (luma row kk, chroma
     * row r of its plane) and takes the row below from the next lane; the
     * last lane of a chunk (plane) reads its second row itself. Lanes below
     * the chunk's clipped height still read, for their upper neighbours.
     * A row is read as aligned words when its needed bytes are inside the
     * reference and the words past its end stay inside the frame, else byte
     * by byte with every sample clamped — the same bytes wherever used. */
    J.act = J.ref = false;
    K.act = K.ref = false;
    const int kk = lane & 7, p = (lane >> 2) & 1, r = lane & 3;
    uint32_t l0 = 0, m0 = 0, h0 = 0, cl0 = 0, ch0 = 0;
    if (c < nchunks) {
        FastBlk fb;
        int lx0, ly0, lw, lh, cx0, cy0, clw, clh;
        fast_chunk(w, c, fb, lx0, ly0, lw, lh, cx0, cy0, clw, clh);
        const int slot = fb_slot(fb);
        const uint8_t *rp = nullptr;
        int rw = 0, rh = 0;
        if (slot < 8) {
            const cvp9_ref_t &R = job.ref[slot];
            rp = R.plane;
            rw = R.w;
            rh = R.h;
        }
        const int mvx = (int16_t)(fb.mv & 0xffffu), mvy = (int16_t)(fb.mv >> 16);
        J.act = kk < lh;
        J.d = D.y + (ly0 + kk) * D.py + lx0;
        J.lw = lw;
        K.act = r < clh && clw > 0;
        K.d = (p ? D.v : D.u) + (cy0 + r) * D.pc + cx0;
        K.clw = clw;
        if (rp) {
            J.ref = true;
            const int px8 = (sbx + lx0) * 8 + mvx, py8 = (sby + ly0) * 8 + mvy;
            const int ix = px8 >> 3, y0 = (py8 >> 3) + kk;
            J.fx = px8 & 7;
            J.fy = py8 & 7;
            /* luma rows are followed by the chroma planes: reads past a row
             * end stay inside the frame; the plane starts 8-byte aligned, so
             * with ix >= 0 they never start before it */
            const bool hin = ix >= 0 && ix + lw < rw && rw >= 16;   /* 16-byte reads stay in the frame */
            if (hin && y0 >= 0 && y0 < rh) ld9d(rp + (size_t)y0 * rw + ix, l0, m0, h0);
            else ld9c(rp, rw, rh, ix, y0, l0, m0, h0);
            if (kk == 7) {
                if (hin && y0 + 1 >= 0 && y0 + 1 < rh) ld9d(rp + (size_t)(y0 + 1) * rw + ix, J.lo1, J.mid1, J.hi1);
                else ld9c(rp, rw, rh, ix, y0 + 1, J.lo1, J.mid1, J.hi1);
            }
            if (clw > 0) {
                K.ref = true;
                const int rcs = (rw + 1) >> 1, crw = rw >> 1, crh = rh >> 1;
                const uint8_t *pl = rp + (size_t)rw * rh + (p ? (size_t)rcs * ((rh + 1) >> 1) : 0);
                const int cpx8 = ((sbx >> 1) + cx0) * 8 + mvx / 2, cpy8 = ((sby >> 1) + cy0) * 8 + mvy / 2;
                const int cix = cpx8 >> 3, y1 = (cpy8 >> 3) + r;
                K.fx = cpx8 & 7;
                K.fy = cpy8 & 7;
                /* a further chroma row below the one read: word reads stay inside */
                const bool chin = cix >= 0 && cix + clw < crw && rcs >= 8;   /* 8-byte reads stay in the plane */
                if (chin && y1 >= 0 && y1 + 1 < crh) ld5w(pl + (size_t)y1 * rcs + cix, cl0, ch0);
                else ld5c(pl, rcs, crw, crh, cix, y1, cl0, ch0);
                if (r == 3) {
                    if (chin && y1 + 1 >= 0 && y1 + 2 < crh) ld5w(pl + (size_t)(y1 + 1) * rcs + cix, K.lo1, K.hi1);
                    else ld5c(pl, rcs, crw, crh, cix, y1 + 1, K.lo1, K.hi1);
                }
            }
        }
    }
    const uint32_t nl = __shfl_down_sync(0xffffffffu, l0, 1), nm = __shfl_down_sync(0xffffffffu, m0, 1);
    const uint32_t nh = __shfl_down_sync(0xffffffffu, h0, 1);
    const uint32_t ncl = __shfl_down_sync(0xffffffffu, cl0, 1), nch = __shfl_down_sync(0xffffffffu, ch0, 1);
    J.lo0 = l0;
    J.mid0 = m0;
    J.hi0 = h0;
    if (kk != 7) {
        J.lo1 = nl;
        J.mid1 = nm;
        J.hi1 = nh;
    }
    K.lo0 = cl0;
    K.hi0 = ch0;
    if (r != 3) {
        K.lo1 = ncl;
        K.hi1 = nch;
    }
}

__device__ __forceinline__ void fast_luma_finish(const FastLuma &J)
{
    if (!J.act) return;
    uint32_t o0 = 0x7f7f7f7fu, o1 = 0x7f7f7f7fu;     /* missing reference: 127 */
    if (J.ref) bilinear8(J.lo0, J.mid0, J.hi0, J.lo1, J.mid1, J.hi1, J.fx, J.fy, o0, o1);
    if (J.lw == 8 && !((uintptr_t)J.d & 3)) {
        reinterpret_cast<uint32_t *>(J.d)[0] = o0;
        reinterpret_cast<uint32_t *>(J.d)[1] = o1;
    } else {
#pragma unroll
        for (int x = 0; x < 8; x++) if (x < J.lw) J.d[x] = (uint8_t)((x < 4 ? o0 : o1) >> (8 * (x & 3)));
    }
}

__device__ __forceinline__ void fast_chroma_finish(const FastChroma &J)
{
    if (!J.act) return;
    const uint32_t o = J.ref ? bilinear4(J.lo0, J.hi0, J.lo1, J.hi1, J.fx, J.fy) : 0x7f7f7f7fu;
    if (J.clw == 4 && !((uintptr_t)J.d & 3)) {
        *reinterpret_cast<uint32_t *>(J.d) = o;
    } else {
#pragma unroll
        for (int x = 0; x < 4; x++) if (x < J.clw) J.d[x] = (uint8_t)(o >> (8 * x));
    }
}

/* Where the q-th TX of size N in the SB sits; `ok` is false past the last
 * TX or when the TX's coefficients run past the array. */
template <int N, class S>
__device__ __forceinline__ const int16_t *fast_tx_locate(const S &w, const cvp9_job_t &job, int q, int ntx,
                                                        int i, int &px0, int &py0, bool &ok)
{
    ok = false;
    px0 = py0 = 0;
    if (q >= ntx) return nullptr;
    const int b = w.txblk[q];
    const FastBlk fb = w.blk[b];
    const int bx = fb_x(fb), by = fb_y(fb), cw = fb_cw(fb);
    const int nx = cw / N;
    const int tq = q - w.txoff[b];
    const int tyy = nx == 1 ? tq : tq / nx, txx = tq - tyy * nx;
    px0 = bx + txx * N;
    py0 = by + tyy * N;
    const uint64_t c0 = (uint64_t)fb.coeff + (uint64_t)tq * (N * N);
    if (c0 + N * N > (uint64_t)job.num_coeffs) return nullptr;
    ok = true;
    return job.coeffs + c0 + (uint64_t)i * N;
}

/* one TX row (N int16) into registers, widest loads the alignment allows */
template <int N>
__device__ __forceinline__ void fast_row_load(uint32_t (&v)[N / 2], const int16_t *src)
{
    const uintptr_t a = (uintptr_t)src;
    if (N >= 8 && !(a & 15)) {
#pragma unroll
        for (int k = 0; k < N / 8; k++) {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(src) + k);
            v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
        }
    } else if (!(a & 3)) {
#pragma unroll
        for (int k = 0; k < N / 2; k++) v[k] = __ldg(reinterpret_cast<const uint32_t *>(src) + k);
    } else {
#pragma unroll
        for (int k = 0; k < N / 2; k++)
            v[k] = (uint32_t)(uint16_t)__ldg(src + 2 * k) | (uint32_t)(uint16_t)__ldg(src + 2 * k + 1) << 16;
    }
}

/* REFCPU residual of every luma TX of size N in the SB. 32/N TXs at a time,
 * lane = (TX, row i). A lane forms T[i][k] = sum_l M[l][i] X[l][k] (l
 * ascending) for each nonzero column k and accumulates O[i][j] += T[i][k]
 * M[k][j] (k ascending) — the two passes of vp9_reconstruct.c:31-50 fused
 * per row. The loops run over the union of the group's nonzero rows and
 * columns so they stay warp-uniform; a term whose coefficient is zero in a
 * lane's own TX adds +-0 to a sum that is never -0, leaving it unchanged.
 * The next group's coefficients are loaded while the current one computes.
 * The predicted rows are read from, and the results written to, dst (the
 * warp's luma tile or the frame: row r of the superblock at dst + r *
 * pitch); frame rows (GLOBAL) are read before the transform, so that they
 * arrive while it computes. */
template <int N, bool GLOBAL, class S>
__device__ void fast_residual(S &w, uint8_t *dst, int pitch, const cvp9_job_t &job, int ntx, int lane)
{
    constexpr int G = 32 / N, NN = N * N;
    constexpr int NH = N == 32 ? 2 : 1, NJ = N / NH;
    constexpr unsigned kSeg = N == 32 ? 0xffffffffu : ((1u << N) - 1u);
    const int g = lane / N, i = lane % N;
    const int boff = N == 4 ? 0 : N == 8 ? 16 : N == 16 ? 80 : 336;
    const double *Mg = g_dct + boff;     /* lane-varying reads */
    const double *Mc = c_dct + boff;     /* warp-uniform reads */
    int16_t *X = w.coef + g * (NN + 2);      /* padded: the groups' rows fall in different banks */
    uint32_t rv[N / 2];
    int px0, py0;
    bool have;
    {
        const int16_t *src = fast_tx_locate<N>(w, job, g, ntx, i, px0, py0, have);
        if (have) fast_row_load<N>(rv, src);
    }
    for (int q0 = 0; q0 < ntx; q0 += G) {
        if (have) {
            uint32_t *dst = reinterpret_cast<uint32_t *>(X + i * N);
#pragma unroll
            for (int k = 0; k < N / 2; k++) dst[k] = rv[k];
        }
        __syncwarp();
        int npx0, npy0;
        bool nhave;
        {
            const int16_t *src = fast_tx_locate<N>(w, job, q0 + G + g, ntx, i, npx0, npy0, nhave);
            if (nhave) fast_row_load<N>(rv, src);
        }
        uint32_t cm = 0;                     /* nonzero rows of column i of this lane's TX */
        if (have) {
#pragma unroll
            for (int l = 0; l < N; l++) cm |= (X[l * N + i] != 0 ? 1u : 0u) << l;
        }
        const unsigned nzl = __ballot_sync(0xffffffffu, cm != 0);
        unsigned U = 0;
#pragma unroll
        for (int s = 0; s < G; s++) U |= nzl >> (s * N);
        U &= kSeg;
        if (U) {
#pragma unroll
            for (int h = 0; h < NH; h++) {
                uint8_t *rowp = dst + (py0 + i) * pitch + px0 + h * NJ;
                const bool words = !GLOBAL || !((uintptr_t)rowp & 3);
                uint32_t pix[NJ / 4];
#pragma unroll
                for (int j4 = 0; j4 < NJ / 4; j4++) pix[j4] = 0u;
                if (GLOBAL && have) {
                    if (words) {
#pragma unroll
                        for (int j4 = 0; j4 < NJ / 4; j4++) pix[j4] = reinterpret_cast<const uint32_t *>(rowp)[j4];
                    } else {
#pragma unroll
                        for (int j = 0; j < NJ; j++) pix[j >> 2] |= (uint32_t)rowp[j] << (8 * (j & 3));
                    }
                }
                double acc[NJ];
#pragma unroll
                for (int j = 0; j < NJ; j++) acc[j] = 0.0;
                for (unsigned u = U; u; u &= u - 1) {
                    const int k = __ffs(u) - 1;
                    const uint32_t cmk = __shfl_sync(0xffffffffu, cm, g * N + k);
                    const uint32_t cmu = __reduce_or_sync(0xffffffffu, cmk);
                    double t = 0.0;
                    for (uint32_t v = cmu; v; v &= v - 1) {
                        const int l = __ffs(v) - 1;
                        t = __dadd_rn(t, __dmul_rn(__ldg(Mg + l * N + i), (double)X[l * N + k]));
                    }
#pragma unroll
                    for (int j = 0; j < NJ; j++) acc[j] = __dadd_rn(acc[j], __dmul_rn(t, Mc[k * N + h * NJ + j]));
                }
                if (have) {
#pragma unroll
                    for (int j4 = 0; j4 < NJ / 4; j4++) {
                        const uint32_t word = GLOBAL ? pix[j4] : reinterpret_cast<const uint32_t *>(rowp)[j4];
                        int o[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            /* round half away from zero; the int16 saturation of
                             * vp9_reconstruct.c:52-59 cannot change the result of
                             * the 0..255 clamp that follows, so it is folded in */
                            const int r = __double2int_rz(__dadd_rn(acc[j4 * 4 + e], copysign(0.5, acc[j4 * 4 + e])));
                            const int px = (int)((word >> (8 * e)) & 0xffu);
                            o[e] = px + r;
                        }
                        const uint32_t outw = pack4_u8(o[0], o[1], o[2], o[3]);
                        if (words) {
                            reinterpret_cast<uint32_t *>(rowp)[j4] = outw;
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; e++) rowp[4 * j4 + e] = (uint8_t)(outw >> (8 * e));
                        }
                    }
                }
            }
        }
        __syncwarp();
        have = nhave;
        px0 = npx0;
        py0 = npy0;
    }
}

/* fast_residual with each group walking its own TX's nonzero columns
 * (ascending) instead of the union over the warp's groups: the warp loops
 * as long as its busiest group. Column k differs between groups, so the
 * basis row M[k][.] is read from the global copy (four 16-byte loads, L1
 * hits). Same operations and order per TX as fast_residual — the terms the
 * union adds are exact zeros. */
template <int N, bool GLOBAL, class S>
__device__ void fast_residual_d(S &w, uint8_t *dst, int pitch, const cvp9_job_t &job, int ntx, int lane)
{
    static_assert(N == 8, "the 8x8 transform");
    constexpr int G = 32 / N, NN = N * N;
    constexpr int boff = 16;
    const int g = lane / N, i = lane % N;
    const double *Mg = g_dct + boff;
    int16_t *X = w.coef + g * (NN + 2);
    uint32_t rv[N / 2];
    int px0, py0;
    bool have;
    {
        const int16_t *src = fast_tx_locate<N>(w, job, g, ntx, i, px0, py0, have);
        if (have) fast_row_load<N>(rv, src);
    }
    for (int q0 = 0; q0 < ntx; q0 += G) {
        uint32_t rm = 0;                     /* nonzero columns of this lane's row */
        if (have) {
            uint32_t *xs = reinterpret_cast<uint32_t *>(X + i * N);
#pragma unroll
            for (int k = 0; k < N / 2; k++) {
                xs[k] = rv[k];
                const uint32_t m = __vcmpne2(rv[k], 0u);
                rm |= ((m & 1u) | ((m >> 15) & 2u)) << (2 * k);
            }
        }
        /* nonzero columns of this lane's TX: OR over its group's lanes */
        uint32_t cols = rm;
#pragma unroll
        for (int o = 1; o < N; o <<= 1) cols |= __shfl_xor_sync(0xffffffffu, cols, o);
        __syncwarp();
        uint8_t *rowp = dst + (py0 + i) * pitch + px0;
        const bool words = !GLOBAL || !((uintptr_t)rowp & 3);
        uint32_t pix[N / 4];
#pragma unroll
        for (int j4 = 0; j4 < N / 4; j4++) pix[j4] = 0u;
        if (GLOBAL && have && cols) {
            if (words) {
#pragma unroll
                for (int j4 = 0; j4 < N / 4; j4++) pix[j4] = reinterpret_cast<const uint32_t *>(rowp)[j4];
            } else {
#pragma unroll
                for (int j = 0; j < N; j++) pix[j >> 2] |= (uint32_t)rowp[j] << (8 * (j & 3));
            }
        }
        int npx0, npy0;
        bool nhave;
        {
            const int16_t *src = fast_tx_locate<N>(w, job, q0 + G + g, ntx, i, npx0, npy0, nhave);
            if (nhave) fast_row_load<N>(rv, src);
        }
        double acc[N];
#pragma unroll
        for (int j = 0; j < N; j++) acc[j] = 0.0;
        const bool any = cols != 0;
        uint32_t left = cols;
        while (__any_sync(0xffffffffu, left != 0)) {
            const bool act = left != 0;
            const int k = act ? __ffs(left) - 1 : 0;
            left &= left - 1;
            /* rows of column k of this lane's TX: bit (group, row) of the ballot */
            const unsigned B = __ballot_sync(0xffffffffu, act && ((rm >> k) & 1u));
            if (act) {
                const unsigned rows = (B >> (g * N)) & ((1u << N) - 1u);
                double t = 0.0;
                for (unsigned v = rows; v; v &= v - 1) {
                    const int l = __ffs(v) - 1;
                    t = __dadd_rn(t, __dmul_rn(__ldg(Mg + l * N + i), (double)X[l * N + k]));
                }
                const double2 *Mr = reinterpret_cast<const double2 *>(Mg + k * N);
#pragma unroll
                for (int j2 = 0; j2 < N / 2; j2++) {
                    const double2 m = __ldg(Mr + j2);
                    acc[2 * j2] = __dadd_rn(acc[2 * j2], __dmul_rn(t, m.x));
                    acc[2 * j2 + 1] = __dadd_rn(acc[2 * j2 + 1], __dmul_rn(t, m.y));
                }
            }
        }
        if (any && have) {
#pragma unroll
            for (int j4 = 0; j4 < N / 4; j4++) {
                const uint32_t word = GLOBAL ? pix[j4] : reinterpret_cast<const uint32_t *>(rowp)[j4];
                int o[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    /* round half away from zero; the int16 saturation of
                     * vp9_reconstruct.c:52-59 cannot change the result of
                     * the 0..255 clamp that follows, so it is folded in */
                    const int r = __double2int_rz(__dadd_rn(acc[j4 * 4 + e], copysign(0.5, acc[j4 * 4 + e])));
                    const int px = (int)((word >> (8 * e)) & 0xffu);
                    o[e] = px + r;
                }
                const uint32_t outw = pack4_u8(o[0], o[1], o[2], o[3]);
                if (words) {
                    reinterpret_cast<uint32_t *>(rowp)[j4] = outw;
                } else {
#pragma unroll
                    for (int e = 0; e < 4; e++) rowp[4 * j4 + e] = (uint8_t)(outw >> (8 * e));
                }
            }
        }
        __syncwarp();
        have = nhave;
        px0 = npx0;
        py0 = npy0;
    }
}

/* ── SPEC arithmetic in k_inter ─────────────────────────────────────────── */

/* 16 consecutive bytes of a row at p as four words (aligned word reads;
 * callers keep the aligned span inside the buffer) */
__device__ __forceinline__ void ld16w(const uint8_t *p, uint32_t o[4])
{
    const uintptr_t a = (uintptr_t)p;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    const unsigned sh = 8u * (unsigned)(a & 3);
    const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3), w4 = __ldg(w + 4);
    o[0] = __funnelshift_r(w0, w1, sh);
    o[1] = __funnelshift_r(w1, w2, sh);
    o[2] = __funnelshift_r(w2, w3, sh);
    o[3] = __funnelshift_r(w3, w4, sh);
}

/* the same 16 bytes, every sample clamped into [0, pw-1] x [0, ph-1] */
__device__ __forceinline__ void ld16c(const uint8_t *plane, int stride, int pw, int ph, int x0, int y, uint32_t o[4])
{
    const int xm = pw > 0 ? pw - 1 : 0, ym = ph > 0 ? ph - 1 : 0;
    const uint8_t *row = plane + (size_t)clampi(y, 0, ym) * stride;
    o[0] = o[1] = o[2] = o[3] = 0u;
#pragma unroll
    for (int x = 0; x < 16; x++) o[x >> 2] |= (uint32_t)__ldg(row + clampi(x0 + x, 0, xm)) << (8 * (x & 3));
}


/* shader rounding of one 8-tap sum: (acc + 64) >> 7 clipped to 8 bits */

/* bytes k..k+3 of o[] as one word (k a compile-time index) */
__device__ __forceinline__ uint32_t win4(const uint32_t o[4], int k)
{
    return (k & 3) ? __funnelshift_r(o[k >> 2], o[(k >> 2) + 1], 8 * (k & 3)) : o[k >> 2];
}


/* Luma prediction of four chunks (vp9_mc.comp.glsl:61-110): lane = (chunk
 * c0 + lane/8, k = lane%8). Horizontal 8-tap rows k and k+8 of each chunk's
 * 15-row window go to shared rows (rounded, clipped to 8 bits), then lane k
 * filters output row k vertically. Fetches clamp into the reference. */
template <class S>
__device__ void spec_luma_pass(S &w, const PredDst &D, const cvp9_job_t &job, int c0, int nchunks, int sbx, int sby,
                               int lane)
{
    uint8_t *hb = reinterpret_cast<uint8_t *>(w.coef);        /* 4 chunks x 15 rows x 8 */
    const int q = lane >> 3, k = lane & 7, c = c0 + q;
    FastBlk fb;
    int lx0 = 0, ly0 = 0, lw = 0, lh = 0, cx0, cy0, clw, clh;
    const uint8_t *rp = nullptr;
    int rw = 0, rh = 0, fx = 0, fy = 0, bx = 0, by = 0;
    if (c < nchunks) {
        fast_chunk(w, c, fb, lx0, ly0, lw, lh, cx0, cy0, clw, clh);
        const cvp9_ref_t &R = job.ref[job.ref_slot_of[fb_slot(fb) & 3] & 7];
        rp = R.plane; rw = R.w; rh = R.h;
        const int mvx = (int16_t)(fb.mv & 0xffffu), mvy = (int16_t)(fb.mv >> 16);
        bx = sbx + lx0 + (mvx >> 3);
        by = sby + ly0 + (mvy >> 3);
        fx = (mvx & 7) << 1;
        fy = (mvy & 7) << 1;
        if (rp) {
            const uint32_t ta = c_subpel_pk[fx][0], tb = c_subpel_pk[fx][1];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int hr = k + 8 * h;
                if (hr >= lh + 7) continue;
                const int y = by - 3 + hr, x0 = bx - 3;
                uint32_t o[4];
                if (x0 >= 0 && x0 + lw + 6 < rw && y >= 0 && y < rh) ld16w(rp + (size_t)y * rw + x0, o);
                else ld16c(rp, rw, rw, rh, x0, y, o);
                int v[8];
#pragma unroll
                for (int cc = 0; cc < 8; cc++) v[cc] = tap8(ta, tb, fx, win4(o, cc), win4(o, cc + 4));
                uint32_t *hrow = reinterpret_cast<uint32_t *>(hb + (q * 15 + hr) * 8);
                hrow[0] = pack4_u8(v[0], v[1], v[2], v[3]);
                hrow[1] = pack4_u8(v[4], v[5], v[6], v[7]);
            }
        }
    }
    __syncwarp();
    if (c < nchunks && k < lh) {
        uint32_t o0 = 0x80808080u, o1 = 0x80808080u;           /* missing reference: 128 */
        if (rp) {
            o0 = o1 = 0;
            /* rows k..k+7 of the filtered window, transposed four by four
             * so that a column's taps meet as one word */
            const uint2 *hrows = reinterpret_cast<const uint2 *>(hb + (q * 15 + k) * 8);
            uint32_t lo[8], hi[8];
#pragma unroll
            for (int tt = 0; tt < 8; tt++) {
                const uint2 v = hrows[tt];
                lo[tt] = v.x;
                hi[tt] = v.y;
            }
            const uint32_t va = c_subpel_pk[fy][0], vb = c_subpel_pk[fy][1];
#pragma unroll
            for (int half = 0; half < 2; half++) {
                const uint32_t *rw8 = half ? hi : lo;
                uint32_t ca[4], cb[4];
                tr4(rw8[0], rw8[1], rw8[2], rw8[3], ca);
                tr4(rw8[4], rw8[5], rw8[6], rw8[7], cb);
                int v[4];
#pragma unroll
                for (int j = 0; j < 4; j++) v[j] = tap8(va, vb, fy, ca[j], cb[j]);
                const uint32_t word = pack4_u8(v[0], v[1], v[2], v[3]);
                if (half) o1 = word; else o0 = word;
            }
        }
        uint8_t *d = D.y + (ly0 + k) * D.py + lx0;
        if (lw == 8 && !((uintptr_t)d & 3)) {
            reinterpret_cast<uint32_t *>(d)[0] = o0;
            reinterpret_cast<uint32_t *>(d)[1] = o1;
        } else {
#pragma unroll
            for (int x = 0; x < 8; x++) if (x < lw) d[x] = (uint8_t)((x < 4 ? o0 : o1) >> (8 * (x & 3)));
        }
    }
    __syncwarp();
}

/* Chroma prediction of four chunks, both planes: lane = (chunk c0 + lane/8,
 * plane, r = lane%4); the chroma MV is read as 1/16 chroma pel (16 phases),
 * fetches clamp into the ceil-half planes. */
template <class S>
__device__ void spec_chroma_pass(S &w, const PredDst &D, const cvp9_job_t &job, int c0, int nchunks, int sbx, int sby,
                                 int lane)
{
    uint8_t *hb = reinterpret_cast<uint8_t *>(w.coef) + 480;  /* 4 chunks x 2 planes x 11 rows x 4 */
    const int q = lane >> 3, p = (lane >> 2) & 1, r = lane & 3, c = c0 + q;
    FastBlk fb;
    int lx0, ly0, lw, lh, cx0 = 0, cy0 = 0, clw = 0, clh = 0;
    const uint8_t *pl = nullptr;
    int cw2 = 0, ch2 = 0, rcs = 0, fx = 0, fy = 0, bx = 0, by = 0;
    if (c < nchunks) {
        fast_chunk(w, c, fb, lx0, ly0, lw, lh, cx0, cy0, clw, clh);
        const cvp9_ref_t &R = job.ref[job.ref_slot_of[fb_slot(fb) & 3] & 7];
        if (R.plane && clw > 0) {
            const int rw = R.w, rh = R.h;
            rcs = (rw + 1) >> 1;
            cw2 = rcs;
            ch2 = (rh + 1) >> 1;
            pl = R.plane + (size_t)rw * rh + (p ? (size_t)rcs * ch2 : 0);
            const int mvx = (int16_t)(fb.mv & 0xffffu), mvy = (int16_t)(fb.mv >> 16);
            bx = (sbx >> 1) + cx0 + (mvx >> 4);
            by = (sby >> 1) + cy0 + (mvy >> 4);
            fx = mvx & 15;
            fy = mvy & 15;
            const uint32_t ta = c_subpel_pk[fx][0], tb = c_subpel_pk[fx][1];
#pragma unroll
            for (int h = 0; h < 3; h++) {
                const int hr = r + 4 * h;
                if (hr >= clh + 7) continue;
                const int y = by - 3 + hr, x0 = bx - 3;
                uint32_t o[4];
                /* a further chroma row exists below: word reads stay inside */
                if (x0 >= 0 && x0 + clw + 6 < cw2 && y >= 0 && y + 1 < ch2) ld16w(pl + (size_t)y * rcs + x0, o);
                else ld16c(pl, rcs, cw2, ch2, x0, y, o);
                int v[4];
#pragma unroll
                for (int cc = 0; cc < 4; cc++) v[cc] = tap8(ta, tb, fx, win4(o, cc), win4(o, cc + 4));
                *reinterpret_cast<uint32_t *>(hb + ((q * 2 + p) * 11 + hr) * 4) = pack4_u8(v[0], v[1], v[2], v[3]);
            }
        }
    }
    __syncwarp();
    if (c < nchunks && clw > 0 && r < clh) {
        uint32_t o = 0x80808080u;                             /* missing reference: 128 */
        if (pl) {
            const uint32_t *hrows = reinterpret_cast<const uint32_t *>(hb + ((q * 2 + p) * 11 + r) * 4);
            uint32_t ca[4], cb[4];
            tr4(hrows[0], hrows[1], hrows[2], hrows[3], ca);
            tr4(hrows[4], hrows[5], hrows[6], hrows[7], cb);
            const uint32_t va = c_subpel_pk[fy][0], vb = c_subpel_pk[fy][1];
            int v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = tap8(va, vb, fy, ca[j], cb[j]);
            o = pack4_u8(v[0], v[1], v[2], v[3]);
        }
        uint8_t *d = (p ? D.v : D.u) + (cy0 + r) * D.pc + cx0;
        if (clw == 4 && !((uintptr_t)d & 3)) {
            *reinterpret_cast<uint32_t *>(d) = o;
        } else {
#pragma unroll
            for (int x = 0; x < 4; x++) if (x < clw) d[x] = (uint8_t)(o >> (8 * x));
        }
    }
    __syncwarp();
}

/* SPEC TX layout of a block in plane p (vp9_kf_tile.c:320-396 for blocks of
 * 8x8 and up): TX log2 size, TXs per row and column (MI-clipped), plane
 * origin in the SB tile, coefficients before this plane. */
struct SpecTx {
    int txl, nx, ny, ox, oy;
    uint64_t base;
};

__device__ __forceinline__ SpecTx spec_tx_layout(const FastBlk &b, int p)
{
    SpecTx s;
    const int l_nx = (int)(b.ext & 0x1fu), l_ny = (int)((b.ext >> 5) & 0x1fu);
    const int c_nx = (int)((b.ext >> 10) & 0xfu), c_ny = (int)((b.ext >> 14) & 0xfu);
    const int ltx = fb_txl(b), ctx = (int)((b.ext >> 18) & 3u);
    const int lc = l_nx * l_ny * (16 << (2 * ltx)), cc = c_nx * c_ny * (16 << (2 * ctx));
    if (p == 0) { s.txl = ltx; s.nx = l_nx; s.ny = l_ny; s.ox = fb_x(b); s.oy = fb_y(b); s.base = 0; }
    else { s.txl = ctx; s.nx = c_nx; s.ny = c_ny; s.ox = fb_x(b) >> 1; s.oy = fb_y(b) >> 1;
           s.base = (uint64_t)lc + (p == 2 ? (uint64_t)cc : 0); }
    return s;
}

/* SPEC residual of every TX of size N in plane P: 32/N TXs at a time.
 * Column pass, lane = (TX, column j): dequantise (DC step at [0][0] only),
 * 1-D butterfly down the column (vp9_idct.comp.glsl:666-679); the group's
 * int32 column results replace its staged coefficients in shared memory;
 * row pass, lane = (TX, row i): butterfly along the row, final shift 4/5/6,
 * add and clamp into the tile (:680-789). A group with no nonzero
 * coefficient adds nothing and is skipped. */
template <int N, bool GLOBAL, class S>
__device__ void spec_fast_residual(S &w, const PredDst &D, const cvp9_job_t &job, int P, int ntx, int lane)
{
    constexpr int G = 32 / N, NN = N * N;
    const int g = lane / N, i = lane % N;
    int16_t *X = w.coef + g * NN;
    int32_t *T = reinterpret_cast<int32_t *>(w.coef) + g * NN;
    uint8_t *tile = P == 0 ? D.y : (P == 1 ? D.u : D.v);
    const int pitch = P == 0 ? D.py : D.pc;
    const int sh = N == 4 ? 4 : (N == 8 ? 5 : 6);
    for (int q0 = 0; q0 < ntx; q0 += G) {
        const int q = q0 + g;
        bool have = q < ntx;
        int px0 = 0, py0 = 0;
        if (have) {
            const int b = w.txblk[q];
            const FastBlk fb = w.blk[b];
            const SpecTx L = spec_tx_layout(fb, P);
            const int tq = q - w.txoff[b];
            const int tyy = L.nx == 1 ? tq : tq / L.nx, txx = tq - tyy * L.nx;
            px0 = L.ox + txx * N;
            py0 = L.oy + tyy * N;
            const uint64_t c0 = (uint64_t)fb.coeff + L.base + (uint64_t)tq * NN;
            if (c0 + NN > (uint64_t)job.num_coeffs) have = false;
            else {
                uint32_t rv[N / 2];
                fast_row_load<N>(rv, job.coeffs + c0 + (uint64_t)i * N);
                uint32_t *dst = reinterpret_cast<uint32_t *>(X + i * N);
#pragma unroll
                for (int k = 0; k < N / 2; k++) dst[k] = rv[k];
            }
        }
        __syncwarp();
        wi v[N];
        bool any = false;
        if (have) {
#pragma unroll
            for (int k = 0; k < N; k++) {
                const int cf = X[k * N + i];
                any |= cf != 0;
                v[k] = wi(cf) * ((k == 0 && i == 0) ? job.q_dc : job.q_ac);
            }
            if (any) idct_n(v, N);
        }
        const bool grp_any = __any_sync(0xffffffffu, any);
        __syncwarp();                          /* every lane has read its column */
        if (grp_any) {
            if (have) {
#pragma unroll
                for (int k = 0; k < N; k++) T[k * N + i] = any ? v[k].v : 0;
            }
            __syncwarp();
            if (have) {
#pragma unroll
                for (int k = 0; k < N; k++) v[k] = wi(T[i * N + k]);
                idct_n(v, N);
                uint8_t *rowp = tile + (py0 + i) * pitch + px0;
                const int vw = P == 0 ? D.vw : D.cvw, vh = P == 0 ? D.vh : D.cvh;
                const int xin = vw - px0;            /* samples of the row inside the frame */
                const bool rowin = py0 + i < vh;
                const bool words = (!GLOBAL || !((uintptr_t)rowp & 3)) && xin >= N;
#pragma unroll
                for (int j4 = 0; j4 < N / 4; j4++) {
                    if (!rowin || 4 * j4 >= xin) continue;
                    uint32_t word;
                    if (words) {
                        word = reinterpret_cast<const uint32_t *>(rowp)[j4];
                    } else {
                        word = 0;
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (4 * j4 + e < xin) word |= (uint32_t)rowp[4 * j4 + e] << (8 * e);
                    }
                    int o[4];
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        o[e] = (int)((word >> (8 * e)) & 0xffu) + (((int)((unsigned)v[j4 * 4 + e].v + (1u << (sh - 1)))) >> sh);
                    const uint32_t outw = pack4_u8(o[0], o[1], o[2], o[3]);
                    if (words) {
                        reinterpret_cast<uint32_t *>(rowp)[j4] = outw;
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (4 * j4 + e < xin) rowp[4 * j4 + e] = (uint8_t)(outw >> (8 * e));
                    }
                }
            }
        }
        __syncwarp();
    }
}

} /* namespace */

/* Steps 1-2 of a superblock on the warp-per-SB paths: load, check and pack
 * its block descriptors (w.blk), check that they tile the visible SB exactly
 * (4x4-cell occupancy in w.cells), and map its 8x8 prediction chunks
 * (w.choff, w.chblk). Returns the number of chunks, or -1 when the SB
 * belongs to the general kernel (intra, malformed, odd layouts). nb_out: the
 * SB's block count. CHECK = false: only load and pack the descriptors (a
 * second kernel on an SB the first one already took; returns 0). */
template <int A, bool CHECK = true, class S>
__device__ int fast_sb_setup(S &w, const cvp9_job_t &job, int sb, int sbx, int sby, int lane, int &nb_out)
{
    const int W = job.W, H = job.H;
    const uint32_t *rg = job.sb_range + 4 * sb;
    const uint32_t start = rg[0], end = rg[1], groups = rg[2];
    bool gen = groups != 1 || end < start || end > job.num_blocks || end - start > 64u ||
               (*job.status & CVP9_JOB_BAD_BLOCK) != 0;
    const int nb = gen ? 0 : (int)(end - start);
    nb_out = nb;

    /* 1. blocks: load, check, pack; 4x4-cell occupancy */
    if (CHECK) {
        if (lane < 8) w.cells[lane] = 0u;
        __syncwarp();
    }
    bool bad = false, ovl = false;
    int nch[2] = { 0, 0 };
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int i = lane + 32 * r;
        if (i >= nb) continue;
        const uint32_t *g = reinterpret_cast<const uint32_t *>(job.blocks + start + i);
        const uint32_t g0 = __ldg(g), g1 = __ldg(g + 1), g2 = __ldg(g + 2), g3 = __ldg(g + 3);
        const uint32_t g5 = __ldg(g + 5), g6 = __ldg(g + 6);
        const int gx = (int)(g0 & 0xffffu), gy = (int)(g0 >> 16);
        const int bw = (int)(g1 & 0xffu), bh = (int)((g1 >> 8) & 0xffu);
        const int txl = (int)((g1 >> 16) & 0xffu), intra = (int)(g1 >> 24);
        const int ref0 = (int)((g2 >> 16) & 0xffu), skip = (int)(g5 & 0xffu);
        const int lx = gx - sbx, ly = gy - sby;
        const bool mb = lx < 0 || ly < 0 || (lx & 3) || (ly & 3) || (bw & 3) || (bh & 3) ||
                        bw < 4 || bh < 4 || lx + bw > 64 || ly + bh > 64 || gx >= W || gy >= H || txl > 3 ||
                        ((bw < 8 || bh < 8) && ((lx & 7) || (ly & 7)));
        bad |= mb || intra;
        if (mb) continue;
        const int cw = min(bw, W - gx), ch = min(bh, H - gy);
        FastBlk fb;
        uint32_t slot4 = (ref0 >= 1 && ref0 <= 8) ? (uint32_t)(ref0 - 1) : 15u;
        fb.ext = 0u;
        if (A == CVP9_ARITH_SPEC) {
            /* sub-8x8 residuals span their whole 8x8 MI (they overlap), and
             * 32x32 TXs need more staging than a warp has: general path */
            slot4 = (uint32_t)clampi(ref0 - 1, 0, 2);
            int uvtx = min(txl, max_tx_for(max(bw / 2, 4), max(bh / 2, 4)));
            /* the fast path keeps every TX inside its block and its rows
             * word-aligned: MI-aligned power-of-two blocks, TX <= block */
            bad |= bw < 8 || bh < 8 || txl == 3 || uvtx == 3 || (lx & 7) || (ly & 7) ||
                   (bw & (bw - 1)) || (bh & (bh - 1)) || (4 << txl) > min(bw, bh);
            if (!skip) {
                int nxy[2][2];
#pragma unroll
                for (int pp = 0; pp < 2; pp++) {
                    const int t4 = 1 << (pp ? uvtx : txl);
                    const int pw = max(pp ? bw / 2 : bw, 4), ph = max(pp ? bh / 2 : bh, 4);
                    const int o4x = ((gx >> 3) * 2) >> pp, o4y = ((gy >> 3) * 2) >> pp;
                    const int mw = min(pw / 4, ((job.mi_cols * 2) >> pp) - o4x);
                    const int mh = min(ph / 4, ((job.mi_rows * 2) >> pp) - o4y);
                    nxy[pp][0] = mw > 0 ? (mw + t4 - 1) / t4 : 0;
                    nxy[pp][1] = mh > 0 ? (mh + t4 - 1) / t4 : 0;
                }
                fb.ext = (uint32_t)nxy[0][0] | (uint32_t)nxy[0][1] << 5 | (uint32_t)nxy[1][0] << 10 |
                         (uint32_t)nxy[1][1] << 14 | (uint32_t)uvtx << 18;
            }
        }
        fb.geo = (uint32_t)(lx >> 2) | (uint32_t)(ly >> 2) << 4 | (uint32_t)cw << 8 | (uint32_t)ch << 15 |
                 slot4 << 22 | (uint32_t)txl << 26 | (skip ? 1u : 0u) << 28;
        fb.mv = g3;
        fb.coeff = g6;
        w.blk[i] = fb;
        if (!CHECK) continue;
        nch[r] = ((cw + 7) >> 3) * ((ch + 7) >> 3);
        const int c0x = lx >> 2, c1x = (lx + cw - 1) >> 2, c0y = ly >> 2, c1y = (ly + ch - 1) >> 2;
        const uint32_t m = (2u << c1x) - (1u << c0x);
        for (int cy = c0y; cy <= c1y; cy++) {
            const uint32_t mm = m << (16 * (cy & 1));
            ovl |= (atomicOr(&w.cells[cy >> 1], mm) & mm) != 0u;
        }
    }
    __syncwarp();
    if (!CHECK) return 0;
    const int vw = min(64, W - sbx), vh = min(64, H - sby);
    bool gap = false;
    if (lane < 8) {
        const int ncx = (vw + 3) >> 2, ncy = (vh + 3) >> 2;
        const uint32_t rowm = ncx >= 16 ? 0xffffu : ((1u << ncx) - 1u);
        const uint32_t expect = (2 * lane < ncy ? rowm : 0u) | (2 * lane + 1 < ncy ? rowm << 16 : 0u);
        gap = w.cells[lane] != expect;
    }
    gen = __any_sync(0xffffffffu, gen || bad || ovl || gap) != 0;
    if (gen) return -1;

    /* 2. chunk (8x8 luma + 4x4 chroma) offsets and map */
    int nchunks;
    {
        const int x0 = warp_incl_scan(nch[0], lane), x1 = warp_incl_scan(nch[1], lane);
        const int tot0 = __shfl_sync(0xffffffffu, x0, 31), tot1 = __shfl_sync(0xffffffffu, x1, 31);
        nchunks = tot0 + tot1;
        if (nchunks > 128) return -1;   /* more chunks than the map holds (odd block sizes) */
        const int e0 = x0 - nch[0], e1 = tot0 + x1 - nch[1];
        if (lane < nb) { w.choff[lane] = (uint16_t)e0; for (int c = 0; c < nch[0]; c++) w.chblk[e0 + c] = (uint8_t)lane; }
        if (lane + 32 < nb) { w.choff[lane + 32] = (uint16_t)e1; for (int c = 0; c < nch[1]; c++) w.chblk[e1 + c] = (uint8_t)(lane + 32); }
    }
    __syncwarp();
    return nchunks;
}

/* REFCPU luma residual of a set-up superblock (fast_sb_setup): one pass
 * per TX size present, TXs counted on the frame-clamped block
 * (vp9_reconstruct.c:338-340), added to the predicted rows at dst. U8: 8x8
 * TXs through fast_residual_d, each TX walking its own nonzero columns
 * (measured faster on both 8x8-only and mixed content; an unrolled
 * union-of-columns form, tried before it, cut instructions on 8x8 content
 * but its code size cost more on mixed TX sizes). */
template <bool GLOBAL, bool U8, class S, bool ONLY8 = false>
__device__ void fast_refcpu_residual(S &w, uint8_t *dst, int pitch, const cvp9_job_t &job, int nb, int lane)
{
    unsigned sizes = 0;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int i = lane + 32 * r;
        if (i < nb && !fb_skip(w.blk[i])) sizes |= 1u << fb_txl(w.blk[i]);
    }
    sizes = __reduce_or_sync(0xffffffffu, sizes);
    for (unsigned sz = sizes; sz; sz &= sz - 1) {
        const int txl = __ffs(sz) - 1, n = 4 << txl;
        int cnt[2] = { 0, 0 };
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int i = lane + 32 * r;
            if (i < nb) {
                const FastBlk fb = w.blk[i];
                if (!fb_skip(fb) && fb_txl(fb) == txl) cnt[r] = (fb_cw(fb) / n) * (fb_ch(fb) / n);
            }
        }
        const int x0 = warp_incl_scan(cnt[0], lane), x1 = warp_incl_scan(cnt[1], lane);
        const int tot0 = __shfl_sync(0xffffffffu, x0, 31), tot1 = __shfl_sync(0xffffffffu, x1, 31);
        const int e0 = x0 - cnt[0], e1 = tot0 + x1 - cnt[1];
        const int ntx = tot0 + tot1;        /* at most 256: the TXs tile the SB's luma */
        if (lane < nb) { w.txoff[lane] = (uint16_t)e0; for (int c = 0; c < cnt[0]; c++) w.txblk[e0 + c] = (uint8_t)lane; }
        if (lane + 32 < nb) { w.txoff[lane + 32] = (uint16_t)e1; for (int c = 0; c < cnt[1]; c++) w.txblk[e1 + c] = (uint8_t)(lane + 32); }
        __syncwarp();
        if (ONLY8) {
            /* the caller took superblocks whose TXs are all 8x8 */
            fast_residual_d<8, GLOBAL>(w, dst, pitch, job, ntx, lane);
        } else {
            switch (txl) {
            case 0: fast_residual<4, GLOBAL>(w, dst, pitch, job, ntx, lane); break;
            case 1:
                if (U8) fast_residual_d<8, GLOBAL>(w, dst, pitch, job, ntx, lane);
                else fast_residual<8, GLOBAL>(w, dst, pitch, job, ntx, lane);
                break;
            case 2: fast_residual<16, GLOBAL>(w, dst, pitch, job, ntx, lane); break;
            default: fast_residual<32, GLOBAL>(w, dst, pitch, job, ntx, lane); break;
            }
        }
        __syncwarp();
    }
}

/* SPEC residual of a set-up superblock: one pass per (plane, TX size)
 * present, every plane in the tile parser's MI-clipped layout, added to the
 * predicted planes at D. */
template <bool GLOBAL, class S>
__device__ void fast_spec_residual(S &w, const PredDst &D, const cvp9_job_t &job, int nb, int lane)
{
    for (int P = 0; P < 3; P++) {
        unsigned sizes = 0;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int i = lane + 32 * r;
            if (i < nb && !fb_skip(w.blk[i])) sizes |= 1u << spec_tx_layout(w.blk[i], P).txl;
        }
        sizes = __reduce_or_sync(0xffffffffu, sizes);
        for (unsigned sz = sizes; sz; sz &= sz - 1) {
            const int txl = __ffs(sz) - 1;
            int cnt[2] = { 0, 0 };
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int i = lane + 32 * r;
                if (i < nb) {
                    const FastBlk fb = w.blk[i];
                    if (fb_skip(fb)) continue;
                    const SpecTx L = spec_tx_layout(fb, P);
                    if (L.txl == txl) cnt[r] = L.nx * L.ny;
                }
            }
            const int x0 = warp_incl_scan(cnt[0], lane), x1 = warp_incl_scan(cnt[1], lane);
            const int tot0 = __shfl_sync(0xffffffffu, x0, 31), tot1 = __shfl_sync(0xffffffffu, x1, 31);
            const int e0 = x0 - cnt[0], e1 = tot0 + x1 - cnt[1];
            const int ntx = tot0 + tot1;    /* at most 256: the TXs tile the SB's plane */
            if (lane < nb) { w.txoff[lane] = (uint16_t)e0; for (int c = 0; c < cnt[0]; c++) w.txblk[e0 + c] = (uint8_t)lane; }
            if (lane + 32 < nb) { w.txoff[lane + 32] = (uint16_t)e1; for (int c = 0; c < cnt[1]; c++) w.txblk[e1 + c] = (uint8_t)(lane + 32); }
            __syncwarp();
            switch (txl) {
            case 0: spec_fast_residual<4, GLOBAL>(w, D, job, P, ntx, lane); break;
            case 1: spec_fast_residual<8, GLOBAL>(w, D, job, P, ntx, lane); break;
            default: spec_fast_residual<16, GLOBAL>(w, D, job, P, ntx, lane); break;   /* 32 went general */
            }
            __syncwarp();
        }
    }
}

/* MINB: CTAs per SM the register allocation is sized for (5: up to 96
 * registers, no spills; 6: 80 registers, a few spilled). */
template <int A, int MINB>
__global__ void __launch_bounds__(kFastWarps * 32, MINB) k_inter(const cvp9_job_t *__restrict__ jobs,
                                                            const uint32_t *__restrict__ tickets,
                                                            uint32_t n_tickets, uint32_t *__restrict__ general)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    FastSmem &w = reinterpret_cast<FastSmem *>(smem_raw)[warp];
    const uint32_t t = blockIdx.x * kFastWarps + warp;
    if (t >= n_tickets) return;
    const uint32_t code = __ldg(tickets + t);
    const cvp9_job_t &job = jobs[code >> 20];
    const int sb = (int)(code & 0xFFFFFu);
    const int sb_cols = job.sb_cols;
    const int sbr = sb / sb_cols, sbc = sb - sbr * sb_cols;
    const int sbx = sbc * 64, sby = sbr * 64;
    const int W = job.W, H = job.H;
    int nb;
    int nchunks = fast_sb_setup<A>(w, job, sb, sbx, sby, lane, nb);
    if (lane == 0) general[t] = nchunks < 0 ? 1u : 0u;
    if (nchunks < 0) {
        if (lane == 0) atomicAdd(general + 2 * n_tickets + 1, 1u);   /* k_compact skips when 0 */
        return;
    }

    /* 3. prediction (vp9_reconstruct.c:94-131). Luma passes: lane = (chunk
     * c0 + lane/8, row lane%8); chroma passes: lane = (chunk c0 + lane/8,
     * plane, row). Two luma and two chroma passes are in flight: all four
     * issue their loads before any computes. */
    if (A == CVP9_ARITH_SPEC) {
        const PredDst DS = { w.ty, w.tu, w.tv, kFY, kFC, 64, 64, 32, 32 };
        for (int c0 = 0; c0 < nchunks; c0 += 4) spec_luma_pass(w, DS, job, c0, nchunks, sbx, sby, lane);
        for (int c0 = 0; c0 < nchunks; c0 += 4) spec_chroma_pass(w, DS, job, c0, nchunks, sbx, sby, lane);
        nchunks = 0;                      /* the REFCPU passes below do nothing */
    }
    for (int c0 = 0; c0 < nchunks; c0 += 8) {
        FastLuma a, b;
        FastChroma ca, cb;
        const PredDst D = { w.ty, w.tu, w.tv, kFY, kFC, 64, 64, 32, 32 };
        fast_pred_issue(w, D, job, c0 + (lane >> 3), lane, nchunks, sbx, sby, a, ca);
        fast_pred_issue(w, D, job, c0 + 4 + (lane >> 3), lane, nchunks, sbx, sby, b, cb);
        fast_luma_finish(a);
        fast_luma_finish(b);
        fast_chroma_finish(ca);
        fast_chroma_finish(cb);
    }
    __syncwarp();

    /* 4. residual, one pass per (plane, TX size) present: REFCPU luma only
     * with TXs counted on the frame-clamped block; SPEC every plane in the
     * tile parser's MI-clipped layout */
    if (A == CVP9_ARITH_REFCPU) fast_refcpu_residual<false, false>(w, w.ty, kFY, job, nb, lane);
    if (A == CVP9_ARITH_SPEC) {
        const PredDst D = { w.ty, w.tu, w.tv, kFY, kFC, 64, 64, 32, 32 };
        fast_spec_residual<false>(w, D, job, nb, lane);
    }

    /* 5. write the tile (clipped to the frame) and release the SB */
    {
        const int vw = min(64, W - sbx), vh = min(64, H - sby);
        uint8_t *Y = job.out;
        if (!(W & 15) && !((uintptr_t)Y & 15)) {
            for (int i = lane; i < vh * 4; i += 32) {
                const int r = i >> 2, c16 = (i & 3) * 16;
                if (c16 < vw)
                    *reinterpret_cast<uint4 *>(Y + (size_t)(sby + r) * W + sbx + c16) =
                        ld_smem16(w.ty + r * kFY + c16);
            }
        } else if (!(W & 3) && !((uintptr_t)Y & 3)) {
            for (int i = lane; i < vh * 16; i += 32) {
                const int r = i >> 4, c4 = (i & 15) * 4;
                if (c4 < vw)
                    *reinterpret_cast<uint32_t *>(Y + (size_t)(sby + r) * W + sbx + c4) =
                        *reinterpret_cast<const uint32_t *>(w.ty + r * kFY + c4);
            }
        } else {
            for (int i = lane; i < vh * 64; i += 32) {
                const int r = i >> 6, c = i & 63;
                if (c < vw) Y[(size_t)(sby + r) * W + sbx + c] = w.ty[r * kFY + c];
            }
        }
        const int CW = job.CW, CH = job.CH;
        const int cvw = min(32, CW - (sbx >> 1)), cvh = min(32, CH - (sby >> 1));
        uint8_t *U = Y + (size_t)W * H;
        uint8_t *V = U + (size_t)CW * CH;
        if (!(CW & 15) && !((uintptr_t)U & 15) && !((uintptr_t)V & 15)) {
            for (int i = lane; i < 2 * cvh * 2; i += 32) {
                const int p = i >= cvh * 2, k = p ? i - cvh * 2 : i;
                const int r = k >> 1, c16 = (k & 1) * 16;
                if (c16 < cvw)
                    *reinterpret_cast<uint4 *>((p ? V : U) + (size_t)((sby >> 1) + r) * CW + (sbx >> 1) + c16) =
                        ld_smem16((p ? w.tv : w.tu) + r * kFC + c16);
            }
        } else if (!(CW & 3) && !((uintptr_t)U & 3) && !((uintptr_t)V & 3)) {
            for (int i = lane; i < 2 * cvh * 8; i += 32) {
                const int p = i >= cvh * 8, k = p ? i - cvh * 8 : i;
                const int r = k >> 3, c4 = (k & 7) * 4;
                if (c4 < cvw)
                    *reinterpret_cast<uint32_t *>((p ? V : U) + (size_t)((sby >> 1) + r) * CW + (sbx >> 1) + c4) =
                        *reinterpret_cast<const uint32_t *>((p ? w.tv : w.tu) + r * kFC + c4);
            }
        } else {
            for (int i = lane; i < 2 * cvh * 32; i += 32) {
                const int p = i >= cvh * 32, k = p ? i - cvh * 32 : i;
                const int r = k >> 5, c = k & 31;
                if (c < cvw) (p ? V : U)[(size_t)((sby >> 1) + r) * CW + (sbx >> 1) + c] = (p ? w.tv : w.tu)[r * kFC + c];
            }
        }
    }
    __syncwarp();
    if (lane == 0) {
        __threadfence();
        st_release(job.sb_done + sb, job.epoch);
    }
}

/* ── Prediction with its reads one pass ahead (k_pred) ──────────────────
 * The passes of fast_pred_issue / fast_*_finish, but each lane's reference
 * rows go to a shared-memory slot by cp.async, and the next iteration's
 * rows are requested before the current one is filtered, so a warp has two
 * iterations' reads in flight instead of waiting on each. A lane's slot:
 * its luma row (16 bytes around the 9 it needs), the row below (the chunk's
 * last lane only), its chroma row (8 bytes around 5) and the row below
 * (the plane's last lane only). The rows below of the other lanes are their
 * neighbours' rows, read from the neighbour's slot. Rows that need clamped
 * samples are read at once, byte by byte, and stored already extracted. */
constexpr int kSlot = 48, kSlotLB = 16, kSlotCA = 32, kSlotCB = 40;

struct PredGeo {                 /* one lane's pass: what the filter step needs */
    uint8_t *dl, *dc;            /* luma / chroma destination (frame) */
    uint32_t fl;                 /* lw | fx << 4 | fy << 7 | act << 10 | ref << 11 | o0 << 12 | o1 << 15 */
    uint32_t fc;                 /* clw | fx << 3 | fy << 6 | act << 9 | ref << 10 | o0 << 11 | o1 << 13 */
};

/* 9 bytes at offset o (0..7) of the 16 at q (shared memory, 16-byte aligned) */
__device__ __forceinline__ void slot9(const uint8_t *q, unsigned o, uint32_t &lo, uint32_t &mid, uint32_t &hi)
{
    const uint4 v = *reinterpret_cast<const uint4 *>(q);
    const bool up = o >= 4;
    const unsigned sh = 8u * (o & 3u);
    const uint32_t w0 = up ? v.y : v.x, w1 = up ? v.z : v.y, w2 = up ? v.w : v.z;
    lo = __funnelshift_r(w0, w1, sh);
    mid = __funnelshift_r(w1, w2, sh);
    hi = w2 >> sh;
}

/* 5 bytes at offset o (0..3) of the 8 at q (shared memory, 8-byte aligned) */
__device__ __forceinline__ void slot5(const uint8_t *q, unsigned o, uint32_t &lo, uint32_t &hi)
{
    const uint2 v = *reinterpret_cast<const uint2 *>(q);
    const unsigned sh = 8u * o;
    lo = __funnelshift_r(v.x, v.y, sh);
    hi = v.y >> sh;
}

/* Geometry of chunk c for this lane (as fast_pred_issue) and its row reads,
 * into slot (this lane's, this pass's). */
template <class S>
__device__ __forceinline__ void pred_request(const S &w, const PredDst &D, const cvp9_job_t &job, int c, int lane,
                                             int nchunks, int sbx, int sby, uint8_t *slot, PredGeo &G)
{
    G.fl = 0u;
    G.fc = 0u;
    if (c >= nchunks) return;
    const int kk = lane & 7, p = (lane >> 2) & 1, r = lane & 3;
    FastBlk fb;
    int lx0, ly0, lw, lh, cx0, cy0, clw, clh;
    fast_chunk(w, c, fb, lx0, ly0, lw, lh, cx0, cy0, clw, clh);
    const int slotr = fb_slot(fb);
    const uint8_t *rp = nullptr;
    int rw = 0, rh = 0;
    if (slotr < 8) {
        const cvp9_ref_t &R = job.ref[slotr];
        rp = R.plane;
        rw = R.w;
        rh = R.h;
    }
    const int mvx = (int16_t)(fb.mv & 0xffffu), mvy = (int16_t)(fb.mv >> 16);
    G.dl = D.y + (ly0 + kk) * D.py + lx0;
    G.dc = (p ? D.v : D.u) + (cy0 + r) * D.pc + cx0;
    uint32_t fl = (uint32_t)lw | (kk < lh ? 1u << 10 : 0u);
    uint32_t fc = (uint32_t)max(clw, 0) | (r < clh && clw > 0 ? 1u << 9 : 0u);
    if (rp) {
        const int px8 = (sbx + lx0) * 8 + mvx, py8 = (sby + ly0) * 8 + mvy;
        const int ix = px8 >> 3, y0 = (py8 >> 3) + kk;
        fl |= (uint32_t)(px8 & 7) << 4 | (uint32_t)(py8 & 7) << 7 | 1u << 11;
        /* luma rows are followed by the chroma planes: 16-byte reads past a
         * row end stay inside the frame; the plane starts 8-byte aligned */
        const bool hin = ix >= 0 && ix + lw < rw && rw >= 16;   /* 16-byte reads stay in the frame */
#pragma unroll
        for (int e = 0; e < 2; e++) {
            if (e == 1 && kk != 7) break;            /* the row below: the chunk's last lane */
            const int y = y0 + e;
            uint8_t *dst = slot + (e ? kSlotLB : 0);
            if (hin && y >= 0 && y < rh) {
                const uint8_t *a = rp + (size_t)y * rw + ix;
                const uint8_t *a8 = reinterpret_cast<const uint8_t *>((uintptr_t)a & ~(uintptr_t)7);
                cp_async8(dst, a8);
                cp_async8(dst + 8, a8 + 8);
                fl |= (uint32_t)((uintptr_t)a & 7) << (12 + 3 * e);
            } else {
                uint32_t lo, mid, hi;
                ld9c(rp, rw, rh, ix, y, lo, mid, hi);
                *reinterpret_cast<uint4 *>(dst) = make_uint4(lo, mid, hi, 0u);
            }
        }
        /* the row below of the other lanes is their neighbour's row: the
         * filter step needs its offset, from the same column and y0 + 1 */
        if (kk != 7 && hin && y0 + 1 >= 0 && y0 + 1 < rh)
            fl |= (uint32_t)(((uintptr_t)rp + (size_t)(y0 + 1) * rw + ix) & 7) << 15;
        if (clw > 0) {
            const int rcs = (rw + 1) >> 1, crw = rw >> 1, crh = rh >> 1;
            const uint8_t *pl = rp + (size_t)rw * rh + (p ? (size_t)rcs * ((rh + 1) >> 1) : 0);
            const int cpx8 = ((sbx >> 1) + cx0) * 8 + mvx / 2, cpy8 = ((sby >> 1) + cy0) * 8 + mvy / 2;
            const int cix = cpx8 >> 3, y1 = (cpy8 >> 3) + r;
            fc |= (uint32_t)(cpx8 & 7) << 3 | (uint32_t)(cpy8 & 7) << 6 | 1u << 10;
            /* a further chroma row below the one read: reads stay inside */
            const bool chin = cix >= 0 && cix + clw < crw && rcs >= 8;   /* 8-byte reads stay in the plane */
#pragma unroll
            for (int e = 0; e < 2; e++) {
                if (e == 1 && r != 3) break;         /* the row below: the plane's last lane */
                const int y = y1 + e;
                uint8_t *dst = slot + (e ? kSlotCB : kSlotCA);
                if (chin && y >= 0 && y + 1 < crh) {
                    const uint8_t *a = pl + (size_t)y * rcs + cix;
                    const uint8_t *a4 = reinterpret_cast<const uint8_t *>((uintptr_t)a & ~(uintptr_t)3);
                    cp_async4(dst, a4);
                    cp_async4(dst + 4, a4 + 4);
                    fc |= (uint32_t)((uintptr_t)a & 3) << (11 + 2 * e);
                } else {
                    uint32_t lo, hi;
                    ld5c(pl, rcs, crw, crh, cix, y, lo, hi);
                    *reinterpret_cast<uint2 *>(dst) = make_uint2(lo, hi);
                }
            }
            if (r != 3 && chin && y1 + 1 >= 0 && y1 + 2 < crh)
                fc |= (uint32_t)(((uintptr_t)pl + (size_t)(y1 + 1) * rcs + cix) & 3) << 13;
        }
    }
    G.fl = fl;
    G.fc = fc;
}

/* The filter step of a pass whose rows have landed: base is the warp's
 * slots for this pass (lane i at base + i * kSlot). */
__device__ __forceinline__ void pred_filter(const PredGeo &G, const uint8_t *base, int lane)
{
    const int kk = lane & 7, r = lane & 3;
    const uint8_t *own = base + lane * kSlot;
    if (G.fl & (1u << 10)) {
        uint32_t o0 = 0x7f7f7f7fu, o1 = 0x7f7f7f7fu;     /* missing reference: 127 */
        if (G.fl & (1u << 11)) {
            uint32_t lo0, mid0, hi0, lo1, mid1, hi1;
            slot9(own, (G.fl >> 12) & 7u, lo0, mid0, hi0);
            slot9(kk == 7 ? own + kSlotLB : own + kSlot, (G.fl >> 15) & 7u, lo1, mid1, hi1);
            bilinear8(lo0, mid0, hi0, lo1, mid1, hi1, (G.fl >> 4) & 7, (G.fl >> 7) & 7, o0, o1);
        }
        const int lw = G.fl & 15u;
        if (lw == 8 && !((uintptr_t)G.dl & 3)) {
            reinterpret_cast<uint32_t *>(G.dl)[0] = o0;
            reinterpret_cast<uint32_t *>(G.dl)[1] = o1;
        } else {
#pragma unroll
            for (int x = 0; x < 8; x++) if (x < lw) G.dl[x] = (uint8_t)((x < 4 ? o0 : o1) >> (8 * (x & 3)));
        }
    }
    if (G.fc & (1u << 9)) {
        uint32_t o = 0x7f7f7f7fu;
        if (G.fc & (1u << 10)) {
            uint32_t lo0, hi0, lo1, hi1;
            slot5(own + kSlotCA, (G.fc >> 11) & 3u, lo0, hi0);
            slot5(r == 3 ? own + kSlotCB : own + kSlot + kSlotCA, (G.fc >> 13) & 3u, lo1, hi1);
            o = bilinear4(lo0, hi0, lo1, hi1, (G.fc >> 3) & 7, (G.fc >> 6) & 7);
        }
        const int clw = G.fc & 7u;
        if (clw == 4 && !((uintptr_t)G.dc & 3)) {
            *reinterpret_cast<uint32_t *>(G.dc) = o;
        } else {
#pragma unroll
            for (int x = 0; x < 4; x++) if (x < clw) G.dc[x] = (uint8_t)(o >> (8 * x));
        }
    }
}

/* ── REFCPU superblocks in two kernels ──────────────────────────────────
 * k_inter's REFCPU work split in two leaner kernels. k_inter holds a
 * superblock's tiles, its coefficient staging and the transform's registers
 * at once, which caps it at 20 warps per SM; its time follows the warps it
 * keeps resident. k_pred predicts straight into the output frame and marks
 * the general superblocks; k_resid adds the luma residual to the frame in
 * place and releases the superblock. Same operations in the same order as
 * k_inter, so the same bytes; the frame's luma makes one more round trip
 * through L2/HBM. */
struct __align__(16) PredSmem {                   /* k_pred, one per warp */
    union {
        uint8_t stage[2 * 2 * 32 * kSlot];        /* REFCPU: 2 iterations x 2 passes x 32 lane slots */
        int16_t coef[2 * 32 * kSlot];             /* SPEC: the filtered rows of the 8-tap passes */
    };
    FastBlk  blk[64];
    uint32_t cells[8];
    uint16_t choff[65];
    uint8_t  chblk[128];
};

struct __align__(16) ResidSmem {                  /* k_resid, one per warp */
    union {
        int16_t  coef[1056];
        uint32_t cells[8];
    };
    FastBlk  blk[64];
    union {
        struct {
            uint16_t choff[65];
            uint8_t  chblk[128];
        };
        struct {
            uint16_t txoff[65];
            uint8_t  txblk[256];
        };
    };
};

static_assert(sizeof(PredSmem) % 16 == 0 && sizeof(ResidSmem) % 16 == 0, "per-warp areas stay 16-byte aligned");
static_assert(offsetof(ResidSmem, coef) % 16 == 0, "coefficient rows are written as words");

/* CTAs of 4 warps per SM the registers are sized for: prediction at 96
 * registers (20 warps), residual at 64 (32 warps, some spilled); measured
 * best of 5..8 each on 64 x 1080p steps (1.016 ms against 1.028 for 80/64
 * and 1.10 for 80/80). */
constexpr int kPredMinB = 5, kResidMinB = 8, kResid8MinB = 8;

/* MARK (REFCPU inter path 5): a taken superblock with a TX other than 8x8
 * is marked 2 instead of 0, for k_resid's PART 2. */
template <int A, int MINB, bool MARK = false>
__global__ void __launch_bounds__(kFastWarps * 32, MINB) k_pred(const cvp9_job_t *__restrict__ jobs,
                                                           const uint32_t *__restrict__ tickets,
                                                           uint32_t n_tickets, uint32_t *__restrict__ general)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    PredSmem &w = reinterpret_cast<PredSmem *>(smem_raw)[warp];
    const uint32_t t = blockIdx.x * kFastWarps + warp;
    if (t >= n_tickets) return;
    const uint32_t code = __ldg(tickets + t);
    const cvp9_job_t &job = jobs[code >> 20];
    const int sb = (int)(code & 0xFFFFFu);
    const int sbr = sb / job.sb_cols, sbc = sb - sbr * job.sb_cols;
    const int sbx = sbc * 64, sby = sbr * 64;
    int nb;
    const int nchunks = fast_sb_setup<A>(w, job, sb, sbx, sby, lane, nb);
    unsigned mark = 0u;
    if (MARK && nchunks >= 0) {
        unsigned sizes = 0u;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int i = lane + 32 * r;
            if (i < nb && !fb_skip(w.blk[i])) sizes |= 1u << fb_txl(w.blk[i]);
        }
        mark = (__reduce_or_sync(0xffffffffu, sizes) & ~2u) ? 2u : 0u;
    }
    if (lane == 0) general[t] = nchunks < 0 ? 1u : mark;
    if (nchunks < 0) {
        if (lane == 0) atomicAdd(general + 2 * n_tickets + 1, 1u);   /* k_compact skips when 0 */
        return;
    }
    const int W = job.W, H = job.H, CW = job.CW, CH = job.CH;
    uint8_t *Y = job.out;
    uint8_t *U = Y + (size_t)W * H;
    uint8_t *V = U + (size_t)CW * CH;
    const size_t coff = (size_t)(sby >> 1) * CW + (sbx >> 1);
    const PredDst D = { Y + (size_t)sby * W + sbx, U + coff, V + coff, W, CW,
                        min(64, W - sbx), min(64, H - sby), min(32, CW - (sbx >> 1)), min(32, CH - (sby >> 1)) };
    if (A == CVP9_ARITH_SPEC) {
        for (int c0 = 0; c0 < nchunks; c0 += 4) spec_luma_pass(w, D, job, c0, nchunks, sbx, sby, lane);
        for (int c0 = 0; c0 < nchunks; c0 += 4) spec_chroma_pass(w, D, job, c0, nchunks, sbx, sby, lane);
        return;
    }
    /* two passes of four chunks per iteration; the next iteration's rows
     * are requested before this one's are filtered */
    const int nit = (nchunks + 7) >> 3;
    auto slots = [&](int st, int pass) { return w.stage + (st * 2 + pass) * 32 * kSlot; };
    PredGeo a, b, na, nx;
    na.fl = na.fc = nx.fl = nx.fc = 0u;
    na.dl = na.dc = nx.dl = nx.dc = nullptr;
    pred_request(w, D, job, lane >> 3, lane, nchunks, sbx, sby, slots(0, 0) + lane * kSlot, a);
    pred_request(w, D, job, 4 + (lane >> 3), lane, nchunks, sbx, sby, slots(0, 1) + lane * kSlot, b);
    cp_async_commit();
    for (int it = 0; it < nit; it++) {
        const int cur = it & 1;
        if (it + 1 < nit) {
            const int c1 = (it + 1) * 8;
            pred_request(w, D, job, c1 + (lane >> 3), lane, nchunks, sbx, sby, slots(cur ^ 1, 0) + lane * kSlot, na);
            pred_request(w, D, job, c1 + 4 + (lane >> 3), lane, nchunks, sbx, sby, slots(cur ^ 1, 1) + lane * kSlot, nx);
            cp_async_commit();
            cp_async_wait_prev();
        } else {
            cp_async_wait_all();
        }
        __syncwarp();
        pred_filter(a, slots(cur, 0), lane);
        pred_filter(b, slots(cur, 1), lane);
        __syncwarp();                    /* the stage is refilled next iteration */
        a = na;
        b = nx;
    }
}

/* U8: the REFCPU 8x8 transform through fast_residual_d (inter path 4) */
/* PART 0: every superblock k_pred took (general[t] == 0); with k_pred
 * marking TX sizes (inter path 5, REFCPU), PART 1 takes the superblocks
 * whose TXs are all 8x8 (general[t] == 0) with only the 8x8 transform in its
 * code, PART 2 the others (general[t] == 2). */
template <int A, int MINB, bool U8, int PART = 0>
__global__ void __launch_bounds__(kFastWarps * 32, MINB) k_resid(const cvp9_job_t *__restrict__ jobs,
                                                            const uint32_t *__restrict__ tickets,
                                                            uint32_t n_tickets, const uint32_t *__restrict__ general)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ResidSmem &w = reinterpret_cast<ResidSmem *>(smem_raw)[warp];
    const uint32_t t = blockIdx.x * kFastWarps + warp;
    if (t >= n_tickets || general[t] != (PART == 2 ? 2u : 0u)) return;    /* general superblocks: k_recon */
    const uint32_t code = __ldg(tickets + t);
    const cvp9_job_t &job = jobs[code >> 20];
    const int sb = (int)(code & 0xFFFFFu);
    const int sbr = sb / job.sb_cols, sbc = sb - sbr * job.sb_cols;
    const int sbx = sbc * 64, sby = sbr * 64;
    int nb;
    /* the same descriptors k_pred checked and packed: packing alone */
    fast_sb_setup<A, false>(w, job, sb, sbx, sby, lane, nb);
    __syncwarp();
    if (A == CVP9_ARITH_SPEC) {
        const int W = job.W, H = job.H, CW = job.CW, CH = job.CH;
        uint8_t *Y = job.out;
        uint8_t *U = Y + (size_t)W * H;
        uint8_t *V = U + (size_t)CW * CH;
        const size_t coff = (size_t)(sby >> 1) * CW + (sbx >> 1);
        const PredDst D = { Y + (size_t)sby * W + sbx, U + coff, V + coff, W, CW,
                        min(64, W - sbx), min(64, H - sby), min(32, CW - (sbx >> 1)), min(32, CH - (sby >> 1)) };
        fast_spec_residual<true>(w, D, job, nb, lane);
    } else {
        fast_refcpu_residual<true, U8, ResidSmem, PART == 1>(w, job.out + (size_t)sby * job.W + sbx, job.W, job,
                                                             nb, lane);
    }
    __syncwarp();
    if (lane == 0) {
        __threadfence();
        st_release(job.sb_done + sb, job.epoch);
    }
}

/* Order-preserving compaction of the tickets k_inter marked general, one
 * CTA: each thread counts a contiguous segment, a CTA-wide scan places the
 * segments, the thread copies its general tickets. */
__global__ void __launch_bounds__(1024) k_compact(const uint32_t *__restrict__ tickets,
                                                  const uint32_t *__restrict__ general, uint32_t n,
                                                  uint32_t *__restrict__ out, uint32_t *__restrict__ count)
{
    __shared__ uint32_t wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (count[1] == 0u) {                /* k_inter took every superblock */
        if (tid == 0) *count = 0u;
        return;
    }
    const uint32_t per = (n + 1023u) / 1024u;
    const uint32_t b = min(n, (uint32_t)tid * per), e = min(n, b + per);
    uint32_t c = 0;
    for (uint32_t i = b; i < e; i++) c += general[i] == 1u;
    uint32_t x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t v = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        wsum[lane] = v;
    }
    __syncthreads();
    uint32_t pos = x - c + (wid ? wsum[wid - 1] : 0u);
    for (uint32_t i = b; i < e; i++)
        if (general[i] == 1u) out[pos++] = tickets[i];
    if (tid == 1023) *count = pos;
}

/* ── Loop filter ─────────────────────────────────────────────────────────── */

__device__ __forceinline__ void filter4(uint8_t *p1, uint8_t *p0, uint8_t *q0, uint8_t *q1, int thr)
{
    int P1 = *p1, P0 = *p0, Q0 = *q0, Q1 = *q1;
    int d0 = P0 - Q0, d1 = P1 - Q1;
    if ((d0 < 0 ? -d0 : d0) * 2 + (d1 < 0 ? -d1 : d1) / 2 > thr) return;
    int delta = clampi((3 * (Q0 - P0) + 4) >> 3, -thr, thr);
    *p0 = (uint8_t)clampi(P0 + delta, 0, 255);
    *q0 = (uint8_t)clampi(Q0 - delta, 0, 255);
    *p1 = (uint8_t)clampi(P1 + delta / 2, 0, 255);
    *q1 = (uint8_t)clampi(Q1 - delta / 2, 0, 255);
}

__device__ __forceinline__ int lf_threshold(int level, int sharp)
{
    int t = level;
    if (sharp > 0) {
        t >>= (sharp > 4) ? 2 : 1;
        if (t > 9 - sharp) t = 9 - sharp;
    }
    return t < 1 ? 1 : t;
}

/* Tile (tx, ty) covers luma [64tx-4, 64tx+60) x [TH ty-4, TH ty+TH-4): every
 * tap of every 8-px edge (rows/cols e-2..e+1) lies in one tile and every
 * row in one tile, so the horizontal pass then the vertical pass run
 * tile-locally and in place with the same result as the frame-wide passes
 * (vp9_reconstruct.c:146-190). TH is 64 or 32 (tile height, chosen per shape
 * by the engine's tuner). Requires W and H not of the form 8k+1 (lf_tiled).
 * Rows move as 32-bit words when the frame width allows. */
template <int A, int TH>
__global__ void __launch_bounds__(256) k_loopfilter(const cvp9_job_t *__restrict__ jobs)
{
    grid_dependency_wait();
    __shared__ __align__(16) uint8_t t[TH * 68];
    const cvp9_job_t &job = jobs[blockIdx.z];
    const int tx = blockIdx.x, ty = blockIdx.y;
    const int x0 = tx * 64 - 4, y0 = ty * TH - 4;
    if (job.lf_tiled != 1 || x0 >= job.W || y0 >= job.H) return;
    const bool filt = !(A == CVP9_ARITH_REFCPU && job.lf_level == 0);
    if (!filt && !job.nv12) return;
    const int tid = threadIdx.x;
    const int xa = max(x0, 0), xb = min(x0 + 64, job.W);
    const int ya = max(y0, 0), yb = min(y0 + TH, job.H);
    uint8_t *Y = job.out;
    const int W = job.W;
    const bool words = !(W & 3) && !((uintptr_t)Y & 3);
    /* tile byte (x - x0, y - y0) at t[(y - y0) * 68 + (x - x0)] */
    if (words) {
        const int w0 = (xa - x0) >> 2, nw = (xb - xa) >> 2;
        for (int i = tid; i < (yb - ya) * 16; i += 256) {
            const int r = i >> 4, c = i & 15;
            if (c < nw)
                *reinterpret_cast<uint32_t *>(&t[(ya - y0 + r) * 68 + 4 * (w0 + c)]) =
                    *reinterpret_cast<const uint32_t *>(Y + (size_t)(ya + r) * W + xa + 4 * c);
        }
    } else {
        for (int i = tid; i < (yb - ya) * 64; i += 256) {
            const int r = i >> 6, c = i & 63;
            const int gx = xa + c;
            if (gx < xb) t[(ya - y0 + r) * 68 + (gx - x0)] = Y[(size_t)(ya + r) * W + gx];
        }
    }
    __syncthreads();
    if (filt) {
        const int thr = lf_threshold(job.lf_level, job.lf_sharpness);
        /* horizontal edges e = y0 + 4 + 8k */
        for (int i = tid; i < (TH / 8) * 64; i += 256) {
            const int k = i >> 6, c = i & 63;
            const int e = y0 + 4 + 8 * k, gx = x0 + c;
            if (e < 8 || e >= job.H || gx < xa || gx >= xb) continue;
            const int r = e - y0;
            filter4(&t[(r - 2) * 68 + c], &t[(r - 1) * 68 + c], &t[r * 68 + c], &t[(r + 1) * 68 + c], thr);
        }
        __syncthreads();
        for (int i = tid; i < 8 * TH; i += 256) {
            const int k = i / TH, r = i % TH;
            const int e = x0 + 4 + 8 * k, gy = y0 + r;
            if (e < 8 || e >= job.W || gy < ya || gy >= yb) continue;
            const int c = e - x0;
            uint8_t *row = &t[r * 68];
            filter4(&row[c - 2], &row[c - 1], &row[c], &row[c + 1], thr);
        }
        __syncthreads();
        if (words) {
            const int w0 = (xa - x0) >> 2, nw = (xb - xa) >> 2;
            for (int i = tid; i < (yb - ya) * 16; i += 256) {
                const int r = i >> 4, c = i & 15;
                if (c < nw)
                    *reinterpret_cast<uint32_t *>(Y + (size_t)(ya + r) * W + xa + 4 * c) =
                        *reinterpret_cast<const uint32_t *>(&t[(ya - y0 + r) * 68 + 4 * (w0 + c)]);
            }
        } else {
            for (int i = tid; i < (yb - ya) * 64; i += 256) {
                const int r = i >> 6, c = i & 63;
                const int gx = xa + c;
                if (gx < xb) Y[(size_t)(ya + r) * W + gx] = t[(ya - y0 + r) * 68 + (gx - x0)];
            }
        }
    }
    if (job.nv12) {
        uint8_t *D = job.nv12;
        for (int i = tid; i < (yb - ya) * 64; i += 256) {
            const int r = i >> 6, c = i & 63;
            const int gx = xa + c;
            if (gx < xb) D[(size_t)(ya + r) * W + gx] = t[(ya - y0 + r) * 68 + (gx - x0)];
        }
        /* chroma [32tx-2, 32tx+30) x [TH/2 ty-2, TH/2 ty+TH/2-2) interleaved */
        const int cxa = max(tx * 32 - 2, 0), cxb = min(tx * 32 + 30, job.CW);
        const int cya = max(ty * (TH / 2) - 2, 0), cyb = min(ty * (TH / 2) + TH / 2 - 2, job.CH);
        const uint8_t *U = job.out + (size_t)W * job.H;
        const uint8_t *V = U + (size_t)job.CW * job.CH;
        uint8_t *UV = D + (size_t)W * job.H;
        for (int i = tid; i < (cyb - cya) * 32; i += 256) {
            const int r = i >> 5, c = i & 31;
            const int gx = cxa + c, gy = cya + r;
            if (gx >= cxb) continue;
            const size_t so = (size_t)gy * job.CW + gx;
            const size_t d = (size_t)gy * 2 * job.CW + 2 * gx;
            UV[d] = U[so];
            UV[d + 1] = V[so];
        }
    }
}

/* Register strips: thread (k, j) owns luma columns [8k-4, 8k+4) and rows
 * [16j-4, 16j+12) as two 32-bit words per row. Its two horizontal edges
 * (rows 16j, 16j+8) have every tap inside the strip's rows, and its one
 * vertical edge (column 8k) every tap inside its columns; every pixel lies in
 * one strip. So the horizontal pass then the vertical pass run in registers,
 * with the frame-wide result (vp9_reconstruct.c:146-190) and no shared
 * memory or barriers. Jobs with lf_tiled == 2: W a multiple of 4 (whole
 * words), W and H not of the form 8k+1, no NV12 target. */
__device__ __forceinline__ uint32_t lf_byte(uint32_t w, int i) { return (w >> (8 * i)) & 0xffu; }
__device__ __forceinline__ uint32_t lf_put(uint32_t w, int i, int v)
{
    return (w & ~(0xffu << (8 * i))) | ((uint32_t)v << (8 * i));
}

__device__ __forceinline__ void lf_filter_vals(int &P1, int &P0, int &Q0, int &Q1, int thr)
{
    const int d0 = P0 - Q0, d1 = P1 - Q1;
    if (abs(d0) * 2 + abs(d1) / 2 > thr) return;
    const int delta = clampi((3 * (Q0 - P0) + 4) >> 3, -thr, thr);
    P0 = clampi(P0 + delta, 0, 255);
    Q0 = clampi(Q0 - delta, 0, 255);
    P1 = clampi(P1 + delta / 2, 0, 255);
    Q1 = clampi(Q1 - delta / 2, 0, 255);
}

template <int A>
__global__ void __launch_bounds__(128) k_lf_strip(const cvp9_job_t *__restrict__ jobs)
{
    grid_dependency_wait();
    const cvp9_job_t &job = jobs[blockIdx.z];
    const int k = blockIdx.x * 128 + threadIdx.x;
    const int xs = 8 * k - 4, y0 = 16 * (int)blockIdx.y - 4;
    if (job.lf_tiled != 2 || xs >= job.W || y0 >= job.H) return;
    if (A == CVP9_ARITH_REFCPU && job.lf_level == 0) return;
    const int W = job.W, H = job.H;
    uint8_t *Y = job.out;
    const bool hasA = xs >= 0, hasB = xs + 4 < W;     /* word A: xs..xs+3, word B: xs+4..xs+7 */
    uint32_t a[16], b[16];
#pragma unroll
    for (int r = 0; r < 16; r++) {
        const int gy = y0 + r;
        a[r] = 0u;
        b[r] = 0u;
        if (gy >= 0 && gy < H) {
            const uint8_t *row = Y + (size_t)gy * W;
            if (hasA) a[r] = *reinterpret_cast<const uint32_t *>(row + xs);
            if (hasB) b[r] = *reinterpret_cast<const uint32_t *>(row + xs + 4);
        }
    }
    const int thr = lf_threshold(job.lf_level, job.lf_sharpness);
    /* horizontal edges at strip rows 4 and 12 */
#pragma unroll
    for (int m = 4; m <= 12; m += 8) {
        const int e = y0 + m;
        if (e < 8 || e >= H) continue;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            if (c < 4 ? !hasA : !hasB) continue;
            uint32_t *wv = c < 4 ? a : b;
            const int bi = c & 3;
            int P1 = (int)lf_byte(wv[m - 2], bi), P0 = (int)lf_byte(wv[m - 1], bi);
            int Q0 = (int)lf_byte(wv[m], bi), Q1 = (int)lf_byte(wv[m + 1], bi);
            lf_filter_vals(P1, P0, Q0, Q1, thr);
            wv[m - 2] = lf_put(wv[m - 2], bi, P1);
            wv[m - 1] = lf_put(wv[m - 1], bi, P0);
            wv[m] = lf_put(wv[m], bi, Q0);
            wv[m + 1] = lf_put(wv[m + 1], bi, Q1);
        }
    }
    /* vertical edge at column xs + 4 = 8k: bytes 2, 3 of A and 0, 1 of B */
    const int ev = xs + 4;
    if (ev >= 8 && ev < W) {
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const int gy = y0 + r;
            if (gy < 0 || gy >= H) continue;
            int P1 = (int)lf_byte(a[r], 2), P0 = (int)lf_byte(a[r], 3);
            int Q0 = (int)lf_byte(b[r], 0), Q1 = (int)lf_byte(b[r], 1);
            lf_filter_vals(P1, P0, Q0, Q1, thr);
            a[r] = (a[r] & 0x0000ffffu) | (uint32_t)P1 << 16 | (uint32_t)P0 << 24;
            b[r] = (b[r] & 0xffff0000u) | (uint32_t)Q0 | (uint32_t)Q1 << 8;
        }
    }
#pragma unroll
    for (int r = 0; r < 16; r++) {
        const int gy = y0 + r;
        if (gy < 0 || gy >= H) continue;
        uint8_t *row = Y + (size_t)gy * W;
        if (hasA) *reinterpret_cast<uint32_t *>(row + xs) = a[r];
        if (hasB) *reinterpret_cast<uint32_t *>(row + xs + 4) = b[r];
    }
}

/* Frame-wide loop filter for widths/heights of the form 8k+1, with the
 * reference's flat addressing (vertical edges at the last column read the
 * next row's first sample) and out-of-plane accesses skipped. */
__global__ void k_lf_flat_h(const cvp9_job_t *__restrict__ jobs, int refcpu)
{
    grid_dependency_wait();
    const cvp9_job_t &job = jobs[blockIdx.y];
    if (job.lf_tiled || (refcpu && job.lf_level == 0)) return;
    int thr = lf_threshold(job.lf_level, job.lf_sharpness);
    int nedge = job.H > 8 ? (job.H - 1) / 8 : 0;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nedge * job.W) return;
    int e = 8 * (int)(i / job.W + 1), x = (int)(i % job.W);
    if (e + 1 >= job.H) return;
    uint8_t *Y = job.out;
    size_t S = (size_t)job.W;
    filter4(Y + (e - 2) * S + x, Y + (e - 1) * S + x, Y + e * S + x, Y + (e + 1) * S + x, thr);
}

__global__ void k_lf_flat_v(const cvp9_job_t *__restrict__ jobs, int refcpu)
{
    grid_dependency_wait();
    const cvp9_job_t &job = jobs[blockIdx.y];
    if (job.lf_tiled || (refcpu && job.lf_level == 0)) return;
    int thr = lf_threshold(job.lf_level, job.lf_sharpness);
    int nedge = job.W > 8 ? (job.W - 1) / 8 : 0;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nedge * job.H) return;
    int e = 8 * (int)(i / job.H + 1), r = (int)(i % job.H);
    uint8_t *Y = job.out;
    size_t S = (size_t)job.W, plane = S * job.H;
    size_t base = (size_t)r * S + e;
    if (base + 1 >= plane) return;
    filter4(Y + base - 2, Y + base - 1, Y + base, Y + base + 1, thr);
}

/* ── FULL profile: the VP9 loop filter ───────────────────────────────────
 *
 * k_lf_mimap records, per 8x8 MI, what the filter needs of the block that
 * covers it: luma and chroma TX size, whether it is a skipped inter block,
 * and the MI's offset inside the block (bits 0-1, 2-3, 4, 5-7, 8-10), tagged
 * with the frame's epoch in the high half so that entries of earlier frames
 * read as "no block". k_lf_full then filters the picture in the VP9 order. */
__global__ void __launch_bounds__(256) k_lf_mimap(const cvp9_job_t *__restrict__ jobs)
{
    const cvp9_job_t &job = jobs[blockIdx.y];
    if (!job.full || !job.mi_map) return;
    const uint32_t tag = (job.epoch & 0xFFFFu) << 16;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < job.num_blocks; i += gridDim.x * blockDim.x) {
        const vp9_macroblock_info_t b = job.blocks[i];
        if (b.x >= job.W || b.y >= job.H || b.tx_size > 3 || b.width < 4 || b.height < 4) continue;
        const bool sub8 = b.width < 8 || b.height < 8;
        const int bw = sub8 ? 8 : b.width, bh = sub8 ? 8 : b.height;
        const int uvw = bw / 2 < 4 ? 4 : bw / 2, uvh = bh / 2 < 4 ? 4 : bh / 2;
        const int txuv = sub8 ? 0 : min((int)b.tx_size, max_tx_for(uvw, uvh));
        const uint32_t info = tag | (uint32_t)b.tx_size | ((uint32_t)txuv << 2) |
                              ((uint32_t)(b.skip && !b.is_intra) << 4);
        const int mc = b.x >> 3, mr = b.y >> 3;
        const int nc = min((bw + 7) >> 3, job.mi_cols - mc), nr = min((bh + 7) >> 3, job.mi_rows - mr);
        for (int r = 0; r < nr; r++)
            for (int c = 0; c < nc; c++)
                job.mi_map[(size_t)(mr + r) * job.mi_cols + mc + c] = info | ((uint32_t)c << 5) | ((uint32_t)r << 8);
    }
}

struct LfThr { int lim, mblim, hev; };

/* The 4-tap filter on p1 p0 | q0 q1; hev: high edge variance there. At 10
 * bits (SH 2) it clamps to the signed range of the bit depth around mid. */
template <int SH>
__device__ __forceinline__ void lf_four(int &p1, int &p0, int &q0, int &q1, int hev_thr)
{
    constexpr int kMid = 128 << SH;
    auto sc = [](int v) { return clampi(v, -kMid, kMid - 1); };
    const int ps1 = p1 - kMid, ps0 = p0 - kMid, qs0 = q0 - kMid, qs1 = q1 - kMid;
    const bool hev = abs(p1 - p0) > hev_thr || abs(q1 - q0) > hev_thr;
    const int f = sc((hev ? sc(ps1 - qs1) : 0) + 3 * (qs0 - ps0));
    const int f1 = sc(f + 4) >> 3, f2 = sc(f + 3) >> 3;
    q0 = sc(qs0 - f1) + kMid;
    p0 = sc(ps0 + f2) + kMid;
    if (!hev) {
        const int f3 = (f1 + 1) >> 1;
        q1 = sc(qs1 - f3) + kMid;
        p1 = sc(ps1 + f3) + kMid;
    }
}

__device__ __forceinline__ int lf_diff(int a, int b) { return (int)__sad(a, b, 0u); }

/* Whether the edge between a[K + 3] and a[K + 4] is filtered at all. */
template <int K>
__device__ __forceinline__ bool lf_mask(const int (&a)[16], LfThr th)
{
    const int m = max(max(max(lf_diff(a[K], a[K + 1]), lf_diff(a[K + 1], a[K + 2])), lf_diff(a[K + 2], a[K + 3])),
                      max(max(lf_diff(a[K + 5], a[K + 4]), lf_diff(a[K + 6], a[K + 5])), lf_diff(a[K + 7], a[K + 6])));
    return m <= th.lim && lf_diff(a[K + 3], a[K + 4]) * 2 + (lf_diff(a[K + 2], a[K + 5]) >> 1) <= th.mblim;
}

/* The edge in the middle of a[0..15] (p7..p0, q0..q7): code 1, 2, 3 = 4, 8 or
 * 16 wide at most, narrowed by the flatness tests. The wide filters' outputs
 * are sliding sums of the samples, the outermost repeated. */
template <int SH>
__device__ __forceinline__ void lf_edge(int (&a)[16], int code, LfThr th)
{
    constexpr int kFlat = 1 << SH;
    if (!lf_mask<4>(a, th)) return;
    int near = 0, far = 0;
#pragma unroll
    for (int i = 1; i < 4; i++) near = max(near, max(lf_diff(a[7 - i], a[7]), lf_diff(a[8 + i], a[8])));
    const bool flat = code >= 2 && near <= kFlat;
    if (flat && code == 3) {
#pragma unroll
        for (int i = 4; i < 8; i++) far = max(far, max(lf_diff(a[7 - i], a[7]), lf_diff(a[8 + i], a[8])));
    }
    if (flat && code == 3 && far <= kFlat) {
        /* o[k] = (a[k] + sum of a[k - 7 .. k + 7] + 8) >> 4, k = 1 .. 14 */
        int s = 8 + 7 * a[0], o[16];
#pragma unroll
        for (int i = 1; i < 9; i++) s += a[i];
#pragma unroll
        for (int k = 1; k < 15; k++) {
            o[k] = (s + a[k]) >> 4;
            s += a[k + 8 < 15 ? k + 8 : 15] - a[k - 7 > 0 ? k - 7 : 0];
        }
#pragma unroll
        for (int k = 1; k < 15; k++) a[k] = o[k];
    } else if (flat) {
        /* the same on a[4 .. 11], 3 to each side */
        int s = 4 + 3 * a[4], o[16];
#pragma unroll
        for (int i = 5; i < 9; i++) s += a[i];
#pragma unroll
        for (int k = 5; k < 11; k++) {
            o[k] = (s + a[k]) >> 3;
            s += a[k + 4 < 11 ? k + 4 : 11] - a[k - 3 > 4 ? k - 3 : 4];
        }
#pragma unroll
        for (int k = 5; k < 11; k++) a[k] = o[k];
    } else {
        lf_four<SH>(a[6], a[7], a[8], a[9], th.hev);
    }
}

/* Filter size of the edge on the left (dir 0) or top (dir 1) of 8x8 unit
 * (ux, uy) of a plane as a code (0 none, 1, 2, 3 = 4, 8, 16 wide) | 4 when the
 * 4x4 edge 4 samples in is filtered too. Chroma units take the block at their
 * top-left MI; e: its mode-info word (k_lf_mimap). */
struct LfGeom { int W, H, CW, CH, mi_cols, mi_rows; unsigned epoch; };

__device__ __forceinline__ int lf_unit_edge(const LfGeom &job, int plane, int ux, int uy, int dir, uint32_t e)
{
    const int ss = plane > 0;
    const uint32_t info = (e >> 16) == (job.epoch & 0xFFFFu) ? (e & 0xFFFFu) : 0u;
    const int tx = ss ? (int)((info >> 2) & 3u) : (int)(info & 3u);
    const bool skipi = (info >> 4) & 1u;
    const int pos = (int)(dir ? (info >> 8) & 7u : (info >> 5) & 7u) * (ss ? 4 : 8);
    const int u = dir ? uy : ux, edge = u * 8;
    const bool half = ss && ((u << 1) + 1 >= (dir ? job.mi_rows : job.mi_cols));
    const int dim = dir ? (ss ? job.CH : job.H) : (ss ? job.CW : job.W);
    const int inner = tx == 0 && !skipi && !half && edge + 4 < dim ? 4 : 0;
    if (edge == 0) return inner;
    const bool block_edge = pos == 0, tx_edge = (pos & ((4 << tx) - 1)) == 0;
    if (!block_edge && !(tx_edge && !skipi)) return inner;
    int code = tx == 0 ? 1 : (tx == 1 ? 2 : 3);
    if (code == 1 && (edge & 31) == 0) code = 2;
    if (code == 3 && half) code = 2;
    return code | inner;
}

__device__ bool wait_at_least(const unsigned *flag, unsigned v)
{
    for (int it = 0; it < kRowLooks; it++) {
        if (ld_acquire(flag) >= v) return true;
        __nanosleep(it < 64 ? 32 : 256);
    }
    return false;
}

/* 4 and 8 samples as one load or store. */
template <class T> struct Quad;
template <> struct Quad<uint8_t> { using q4 = unsigned int; using q8 = uint2; };
template <> struct Quad<uint16_t> { using q4 = uint2; using q8 = uint4; };

/* 256 threads filter, 64 bring the rows above, 64 load and write back. */
constexpr int kLfWork = 256, kLfHalo = 64, kLfCopy = 64, kLfThreads = kLfWork + kLfHalo + kLfCopy;

/* Four superblocks of a superblock row in shared memory, used in turn, with
 * the 8 rows above; a row's pitch is 16 bytes past a multiple of 128, so that
 * the row threads' loads spread over the banks. */
template <class T>
struct LfSmem {
    static constexpr int kP = 256 + 16 / (int)sizeof(T), kPC = 128 + 16 / (int)sizeof(T);
    T        y[72 * kP];
    T        c[2][40 * kPC];
    uint32_t mi[64];                  /* mode-info words of the superblock being prepared */
    uint8_t  edge[4][2][64 + 16];     /* lf_unit_edge by slot, direction, unit (luma, chroma) */
    int      ticket;
    volatile int body, halo, done;    /* superblocks loaded, with their rows above, written back */
};

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" :: "r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" :: "r"(id), "r"(n) : "memory"); }

/* Bounded wait on a shared-memory count. */
__device__ __forceinline__ bool lf_wait(const volatile int *count, int v)
{
    for (int it = 0; *count < v; it++) {
        if (it >= kShmLooks) return false;
        if (it > 64) __nanosleep(64);
    }
    __threadfence_block();
    return true;
}

__device__ __forceinline__ void lf_unpack(int *a, uint2 w)
{
#pragma unroll
    for (int i = 0; i < 4; i++) { a[i] = (int)((w.x >> (8 * i)) & 255u); a[4 + i] = (int)((w.y >> (8 * i)) & 255u); }
}
__device__ __forceinline__ void lf_unpack(int *a, uint4 w)
{
    const uint32_t x[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
    for (int i = 0; i < 4; i++) { a[2 * i] = (int)(x[i] & 0xffffu); a[2 * i + 1] = (int)(x[i] >> 16); }
}
__device__ __forceinline__ void lf_pack(const int *a, uint2 &w)
{
    w.x = (uint32_t)a[0] | (uint32_t)a[1] << 8 | (uint32_t)a[2] << 16 | (uint32_t)a[3] << 24;
    w.y = (uint32_t)a[4] | (uint32_t)a[5] << 8 | (uint32_t)a[6] << 16 | (uint32_t)a[7] << 24;
}
__device__ __forceinline__ void lf_pack(const int *a, uint4 &w)
{
    w.x = (uint32_t)a[0] | (uint32_t)a[1] << 16;
    w.y = (uint32_t)a[2] | (uint32_t)a[3] << 16;
    w.z = (uint32_t)a[4] | (uint32_t)a[5] << 16;
    w.w = (uint32_t)a[6] | (uint32_t)a[7] << 16;
}
__device__ __forceinline__ void lf_async(unsigned int *d, const unsigned int *s) { cp_async4(d, s); }
__device__ __forceinline__ void lf_async(uint2 *d, const uint2 *s) { cp_async8(d, s); }
__device__ __forceinline__ void lf_async(uint4 *d, const uint4 *s) { cp_async16(d, s); }

/* One CTA takes a superblock row (ticket) and filters it in 8x8 units by a
 * fixed schedule of steps with a barrier each. Superblock c's vertical edges
 * of unit (i, j) (column, row; with the inner 4x4 edges) run in step 10c + i +
 * j; its horizontal ones in 10c + i + j + 2 (luma's last column: 10c + j + 8),
 * which is after every vertical edge of the superblock that reaches their
 * samples; the next superblock's first vertical edges, ten steps on, come
 * after the horizontal edges of the units they reach into. So every sample
 * sees its edges in the VP9 order (a superblock's vertical edges, then its
 * horizontal ones, superblocks in raster order) while 8 + 8 units of luma and
 * as many of chroma are at work at a time. A filtering thread owns a row
 * (vertical edges) or a column (horizontal ones) and keeps the 8 samples that
 * it passes from unit to unit in registers.
 * What bounds this is the chain of steps along a row and from row to row, so
 * the filtering threads do nothing else: two warps of their own load
 * superblocks two ahead, write them back when their last sample is final
 * (after step 10c + 17), bottom rows first, and publish them; two more wait
 * (bounded) for the row above and bring the 8 rows that it shares. Six 2160p
 * 10-bit pictures 1.84 -> 0.80 ms, eight 1080p 8-bit ones 0.99 -> 0.41 ms,
 * against a superblock's vertical and then horizontal edges a thread per row
 * and column, superblock after superblock (loads, waits and write-back by the
 * filtering threads between their steps: 1.21 and 0.61 ms). */
template <class T, int SH>
__global__ void __launch_bounds__(kLfThreads, 2) k_lf_full(const cvp9_job_t *__restrict__ jobs, int njobs,
                                                           uint32_t n_tickets, uint32_t *counter)
{
    using Q4 = typename Quad<T>::q4;
    using Q8 = typename Quad<T>::q8;
    constexpr int kP = LfSmem<T>::kP, kPC = LfSmem<T>::kPC;
    enum { kBarStep = 1, kBarCycle, kBarHalo, kBarCopy };
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LfSmem<T> &s = *reinterpret_cast<LfSmem<T> *>(smem_raw);
    const int tid = threadIdx.x;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            s.ticket = (int)atomicAdd(counter, 1u);
            s.body = s.halo = s.done = 0;
        }
        __syncthreads();
        const int ticket = s.ticket;
        if (ticket >= (int)n_tickets) return;
        const cvp9_job_t &job = jobs[ticket % njobs];
        const int row = ticket / njobs;
        if (!job.full || row >= job.sb_rows || job.lf_level == 0) continue;
        const LfGeom g = { job.W, job.H, job.CW, job.CH, job.mi_cols, job.mi_rows, job.epoch };
        const int W = g.W, H = g.H, CW = g.CW, CH = g.CH, ncols = job.sb_cols;
        T *const Y = reinterpret_cast<T *>(job.out);
        T *const U = Y + (size_t)W * H, *const V = U + (size_t)CW * CH;
        unsigned *const status = job.status;
        const int Y0 = row * 64, YC = row * 32;
        if (tid < kLfWork) {
            /* this thread's line: a row of luma (tid < 64) or chroma
             * (128..191), or a column (64..127, 192..255) */
            LfThr th;
            {
                const int level = job.lf_level, sharp = job.lf_sharpness;
                int bil = level >> ((sharp > 0) + (sharp > 4));
                if (sharp > 0 && bil > 9 - sharp) bil = 9 - sharp;
                if (bil < 1) bil = 1;
                th.lim = bil << SH;
                th.mblim = (2 * (level + 2) + bil) << SH;
                th.hev = (level >> 4) << SH;
            }
            const int p = tid < 128 ? 0 : 1 + ((tid >> 5) & 1);
            const bool horiz = (tid >> 6) & 1;                /* filters horizontal edges: a column */
            const int line = p ? tid & 31 : tid & 63, lu = line >> 3;
            const int units = p ? 4 : 8, sz = p ? 32 : 64, pitch = p ? kPC : kP;
            T *const ring = p == 0 ? s.y : s.c[p - 1];
            const int first = horiz ? (p ? YC : Y0) : 0, end = horiz ? (p ? CH : H) : (p ? CW : W);
            /* lines of the superblocks that lie inside the picture */
            const int cols = horiz ? ((p ? CW : W) - line + sz - 1) / sz : ((p ? YC : Y0) + line < (p ? CH : H) ? ncols : 0);
            const uint8_t *const tab = &s.edge[0][horiz][p ? 64 : 0] + (horiz ? lu : lu * units);
            const int tstep = horiz ? units : 1;
            int a[16], k = -(!horiz ? lu : (p == 0 && lu == 7 ? 8 : lu + 2)), c = 0, ph10 = 0, cc = 0;
#pragma unroll
            for (int i = 0; i < 16; i++) a[i] = 0;
            bool ok = lf_wait(&s.body, 2);
            bar_sync(kBarStep, kLfWork);
            for (int t = 0; t < 10 * ncols + 8; t++) {
                if (k >= 0 && k < units && c < cols) {
                    const int slot = (c & 3) * sz, pos = first + (horiz ? 0 : c * sz) + 8 * k;
                    if (pos < end) {
                        const int e = tab[(c & 3) * 160 + k * tstep];
                        const bool last = k == units - 1 || pos + 8 >= end;
                        if (!horiz) {
                            T *const r = ring + (8 + line) * pitch;
                            T *const q = r + slot + 8 * k, *const o = r + ((slot + 8 * k - 8) & (4 * sz - 1));
                            if (k == 0 && c > 0) lf_unpack(a, *reinterpret_cast<const Q8 *>(o));
                            lf_unpack(a + 8, *reinterpret_cast<const Q8 *>(q));
                            if (e & 3) lf_edge<SH>(a, e & 3, th);
                            if ((e & 4) && lf_mask<8>(a, th)) lf_four<SH>(a[10], a[11], a[12], a[13], th.hev);
                            Q8 w;
                            if (k > 0 || c > 0) {
                                lf_pack(a, w);
                                *reinterpret_cast<Q8 *>(o) = w;
                            }
                            if (last) {
                                lf_pack(a + 8, w);
                                *reinterpret_cast<Q8 *>(q) = w;
                            }
                        } else {
                            T *const q = ring + (8 + 8 * k) * pitch + slot + line;
                            if (k == 0 && row > 0) {
#pragma unroll
                                for (int i = 0; i < 8; i++) a[i] = q[(i - 8) * pitch];
                            }
#pragma unroll
                            for (int i = 0; i < 8; i++) a[8 + i] = q[i * pitch];
                            if (e & 3) lf_edge<SH>(a, e & 3, th);
                            if ((e & 4) && lf_mask<8>(a, th)) lf_four<SH>(a[10], a[11], a[12], a[13], th.hev);
                            if (k > 0 || row > 0) {
#pragma unroll
                                for (int i = 0; i < 8; i++) q[(i - 8) * pitch] = (T)a[i];
                            }
                            if (last) {
#pragma unroll
                                for (int i = 0; i < 8; i++) q[i * pitch] = (T)a[8 + i];
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 8; i++) a[i] = a[8 + i];
                    }
                }
                if (++k == 10) { k = 0; c++; }
                /* the next step's first horizontal edges need the rows above */
                if (ph10 == 1 && row > 0 && cc < ncols) ok = ok && lf_wait(&s.halo, cc + 1);
                bar_sync(kBarStep, kLfWork);
                if (ph10 == 7) {
                    /* superblock cc - 1 is final; cc + 1 must be there, and the
                     * copying warps past the last of these barriers */
                    ok = ok && lf_wait(&s.body, cc + 2);
                    bar_arrive(kBarCycle, kLfWork + kLfCopy);
                }
                if (++ph10 == 10) { ph10 = 0; cc++; }
            }
            if (!ok && tid == 0) atomicOr(status, (unsigned)CVP9_JOB_TIMEOUT);
        } else if (tid < kLfWork + kLfHalo) {
            /* the 8 rows above, as the row above publishes them */
            const int ht = tid - kLfWork, r = ht >> 3, v = ht & 7;
            const unsigned *const prev = job.sb_range + 4 * (size_t)(row - 1) * ncols + 3;
            bool ok = true;                  /* a wait that gave up is not repeated */
            for (int c = 0; row > 0 && c < ncols; c++) {
                const int slot = c & 3;
                ok = ok && (c < 4 || lf_wait(&s.done, c - 3));   /* its slot is free */
                if (ht == 0) ok = ok && wait_at_least(prev, (unsigned)c + 1u);
                if (!ok) atomicOr(status, (unsigned)CVP9_JOB_TIMEOUT);
                bar_sync(kBarHalo, kLfHalo);
                const int x = c * 64 + 8 * v, xc = c * 32 + 4 * v;
                Q8 y = {};
                Q4 cu = {}, cv = {};
                if (x < W) y = __ldcg(reinterpret_cast<const Q8 *>(Y + (size_t)(Y0 - 8 + r) * W + x));
                if (xc < CW) {
                    cu = __ldcg(reinterpret_cast<const Q4 *>(U + (size_t)(YC - 8 + r) * CW + xc));
                    cv = __ldcg(reinterpret_cast<const Q4 *>(V + (size_t)(YC - 8 + r) * CW + xc));
                }
                *reinterpret_cast<Q8 *>(&s.y[r * kP + slot * 64 + 8 * v]) = y;
                *reinterpret_cast<Q4 *>(&s.c[0][r * kPC + slot * 32 + 4 * v]) = cu;
                *reinterpret_cast<Q4 *>(&s.c[1][r * kPC + slot * 32 + 4 * v]) = cv;
                __threadfence_block();
                bar_sync(kBarHalo, kLfHalo);
                if (ht == 0) s.halo = c + 1;
            }
        } else {
            const int wt = tid - kLfWork - kLfHalo, v = wt & 7, r0 = wt >> 3;
            unsigned *const prog = job.sb_range + 4 * (size_t)row * ncols + 3;
            const uint32_t *const mi_map = job.mi_map;
            auto load = [&](int c) {
                const int slot = c & 3, x = c * 64 + 8 * v, xc = c * 32 + 4 * v;
                const int mr = row * 8 + r0, mc = c * 8 + v;
                const uint32_t e = mr < g.mi_rows && mc < g.mi_cols ? __ldg(mi_map + (size_t)mr * g.mi_cols + mc) : 0u;
                if (x < W)
                    for (int r = r0; r < 64 && Y0 + r < H; r += 8)
                        lf_async(reinterpret_cast<Q8 *>(&s.y[(8 + r) * kP + slot * 64 + 8 * v]),
                                 reinterpret_cast<const Q8 *>(Y + (size_t)(Y0 + r) * W + x));
                if (xc < CW)
                    for (int r = r0; r < 32 && YC + r < CH; r += 8) {
                        lf_async(reinterpret_cast<Q4 *>(&s.c[0][(8 + r) * kPC + slot * 32 + 4 * v]),
                                 reinterpret_cast<const Q4 *>(U + (size_t)(YC + r) * CW + xc));
                        lf_async(reinterpret_cast<Q4 *>(&s.c[1][(8 + r) * kPC + slot * 32 + 4 * v]),
                                 reinterpret_cast<const Q4 *>(V + (size_t)(YC + r) * CW + xc));
                    }
                cp_async_commit();
                s.mi[wt] = e;
                bar_sync(kBarCopy, kLfCopy);
                for (int i = wt; i < 160; i += kLfCopy) {
                    const int pl = i >= 128, j = pl ? i - 128 : i, dir = pl ? j >> 4 : j >> 6;
                    const int u = pl ? j & 15 : j & 63, ux = pl ? u & 3 : u & 7, uy = pl ? u >> 2 : u >> 3;
                    s.edge[slot][dir][pl * 64 + u] = (uint8_t)lf_unit_edge(
                        g, pl, c * (pl ? 4 : 8) + ux, row * (pl ? 4 : 8) + uy, dir, s.mi[(uy << pl) * 8 + (ux << pl)]);
                }
                cp_async_wait_all();
                __threadfence_block();
                bar_sync(kBarCopy, kLfCopy);
            };
            /* rows [lo, hi) of the window (0..7: the rows above) */
            auto write_y = [&](int c, int lo, int hi) {
                const int x = c * 64 + 8 * v;
                if (x >= W) return;
                for (int r = lo + r0; r < hi; r += 8)
                    if (Y0 - 8 + r >= 0 && Y0 - 8 + r < H)
                        *reinterpret_cast<Q8 *>(Y + (size_t)(Y0 - 8 + r) * W + x) =
                            *reinterpret_cast<const Q8 *>(&s.y[r * kP + (c & 3) * 64 + 8 * v]);
            };
            auto write_c = [&](int c, int lo, int hi) {
                const int x = c * 32 + 4 * v;
                if (x >= CW) return;
                for (int r = lo + r0; r < hi; r += 8)
                    if (YC - 8 + r >= 0 && YC - 8 + r < CH) {
                        const size_t o = (size_t)(YC - 8 + r) * CW + x;
                        *reinterpret_cast<Q4 *>(U + o) = *reinterpret_cast<const Q4 *>(&s.c[0][r * kPC + (c & 3) * 32 + 4 * v]);
                        *reinterpret_cast<Q4 *>(V + o) = *reinterpret_cast<const Q4 *>(&s.c[1][r * kPC + (c & 3) * 32 + 4 * v]);
                    }
            };
            load(0);
            if (ncols > 1) load(1);
            if (wt == 0) s.body = 2;
            for (int n = 0; n <= ncols; n++) {
                bar_sync(kBarCycle, kLfWork + kLfCopy);
                const int c = n - 1;
                if (c >= 0) {
                    write_y(c, 64, 72);
                    write_c(c, 32, 40);
                    bar_sync(kBarCopy, kLfCopy);
                    if (wt == 0) {
                        __threadfence();
                        st_release(prog, (unsigned)c + 1u);
                    }
                    write_y(c, 0, 64);
                    write_c(c, 0, 32);
                    bar_sync(kBarCopy, kLfCopy);
                    if (wt == 0) s.done = c + 1;
                }
                if (n + 2 < ncols) load(n + 2);
                if (wt == 0) s.body = n + 3;
            }
        }
    }
}

/* ── Profile 2 (10-bit 4:2:0): k_hbd_recon ─────────────────────────────
 *
 * The FULL profile's reconstruction on 16-bit samples in [0, 1023]. The
 * frame brings its coefficients dequantised, as int32 (coeffs32, the dense
 * layout of coeffs; the 32x32 halving already applied): the butterflies give
 * what 64-bit integers would (wn: 32-bit values, 64-bit products; wl where a
 * coefficient is outside +-2^18), with 32-bit values between the row and the
 * column pass, both 8-tap passes of a prediction round and clip to 10 bits, intra
 * edges that are missing read 511 above and 513 on the left (512 for a DC
 * with neither), and every residual add clips to [0, 1023]. The loop filter
 * is k_lf_full<uint16_t, 2>.
 *
 * One CTA per superblock ticket (SB-diagonal order over the step's jobs,
 * persistent, as k_recon). What reads no neighbour goes first and together:
 * the inter predictions eight lanes a chunk, then every residual, a warp for
 * TXs of one size. The intra blocks follow
 * as in k_recon, TX by TX in dependency levels over the whole CTA (8x1080p
 * key step 15.6 -> 2.65 ms against a warp per block, prediction and
 * transforms in turn). A superblock whose blocks overlap, lie
 * off the 8x8 grid or are no multiple of their transforms, or whose intra
 * blocks read samples of blocks later in the list, runs block by block in list
 * order, so every sample is what the list order makes it. */
namespace {

constexpr int kHbdThreads = 256, kHbdWarps = kHbdThreads / 32;
constexpr int kHbdMaxBlocks = 256;
constexpr int kHYP = 72, kHCP = 40;      /* tile pitches in samples; column -1 at index 3 */
constexpr int kHbdMax = 1023, kHbdMid = 512;

struct HbdBlk {
    uint8_t  x, y;            /* local luma origin in the SB                 */
    uint8_t  w, h;            /* coded size                                  */
    uint8_t  cw, ch;          /* luma region (a sub-8x8 block's whole 8x8)
                               * clamped to the frame                        */
    uint8_t  ccw, cch;        /* chroma region, clamped                      */
    uint8_t  txl, flags;      /* tx_size; 1 intra, 2 skip                    */
    uint8_t  ymode, uvmode;
    uint8_t  ref0, ref1;
    int16_t  mvx, mvy, mv1x, mv1y;
    uint32_t coeff;
};

struct HbdSmem {
    uint16_t ty[65 * kHYP];                /* luma tile, row 0 = the row above */
    uint16_t tc[2][33 * kHCP];
    union {
        int32_t i[kResidGrid + 32];        /* coefficients (tx_word), then the row pass's output */
        IntraWork w;                       /* then the intra tasks             */
    } tmp;
    alignas(16) int16_t res[kResidGrid];   /* prediction rows; then residuals of intra blocks */
    uint16_t col[16 * 64 + 2 * 16 * 32];   /* left-column copies (IntraView)   */
    HbdBlk   blk[kHbdMaxBlocks];
    uint2    tx[kMaxTasks];                /* residual TXs by size (TxRef)     */
    uint16_t tx_at[3][kHbdMaxBlocks];      /* first TX of a block's plane in tx */
    int      ntx[4];                       /* TXs of each size                 */
    uint16_t it_base[kHbdMaxBlocks + 1];   /* prefix over blocks of their chunks, tasks */
    uint16_t cell[256];                    /* owner block + 1 per 4x4          */
    uint32_t rows[16];                     /* claimed cells, a bit each        */
    unsigned c_lo, c_hi, c_sum;            /* coefficient span of the SB, its blocks' number */
    int      scan[kHbdWarps];
    cvp9_job_t jc;
    unsigned needs;                        /* intra_needs of its blocks        */
    int      ticket;
};

static_assert(sizeof(HbdSmem) <= 75 * 1024, "three CTAs per SM");

__device__ __forceinline__ uint16_t &HT(HbdSmem &s, int p, int x, int y)
{
    return p == 0 ? s.ty[(y + 1) * kHYP + x + 4] : s.tc[p - 1][(y + 1) * kHCP + x + 4];
}

/* Exclusive prefix of v over the CTA's threads (thread order); *total: the
 * sum. Every thread calls it. */
__device__ __forceinline__ int hbd_scan(HbdSmem &s, int v, int *total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s.scan[warp] = x;
    __syncthreads();
    int off = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < kHbdWarps; w++) {
        const int t = s.scan[w];
        off += w < warp ? t : 0;
        tot += t;
    }
    *total = tot;
    __syncthreads();
    return off + x - v;
}

/* The inter predictions of blocks [lo, hi) of the SB, whole CTA, four chunks
 * a warp. */
__device__ __noinline__ void hbd_predict(int lo, int hi, int nb, int sbx, int sby)
{
    HbdSmem &s = smem_as<HbdSmem>();
    const cvp9_job_t &job = s.jc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 3, k = lane & 7;
    const bool inter = tid >= lo && tid < hi && tid < nb && !(s.blk[tid].flags & 1);
    int n;
    const int at = hbd_scan(s, inter ? mc_chunks(s.blk[tid].cw, s.blk[tid].ch, s.blk[tid].ccw, s.blk[tid].cch) : 0, &n);
    if (tid < kHbdMaxBlocks) s.it_base[tid] = (uint16_t)min(at, 0xFFFF);
    __syncthreads();
    const uint32_t (*P)[2] = c_subpel4_pk[job.interp_filter & 3];
    uint16_t *rows = reinterpret_cast<uint16_t *>(s.res) + (warp * 4 + g) * 128;
    for (int base = warp * 4; base < n; base += 4 * kHbdWarps) {
        const int chk = base + g;
        const bool on = chk < n;
        const int bi = on ? find_base(s.it_base, nb, chk) : 0;
        const HbdBlk &b = s.blk[bi];
        int p = 0, x = 0, y = 0, w = 0, h = 0;
        if (on) mc_chunk_at(chk - s.it_base[bi], b.cw, b.ch, b.ccw, b.cch, p, x, y, w, h);
        const int lx = (p ? b.x >> 1 : b.x) + x, ly = (p ? b.y >> 1 : b.y) + y;
        mc_chunk<uint16_t, true>(job, P, b, on, p, (p ? sbx >> 1 : sbx) + lx, (p ? sby >> 1 : sby) + ly, w, h, kHbdMid, rows,
                           &HT(s, p, lx, ly + k), k);
    }
    __syncthreads();
}

/* 32 / N TXs by a warp, T the type of the butterflies' values: the rows of the
 * frame's dequantised coefficients (DCT, ADST along the row by the TX type, WHT
 * when lossless) in place in the permuted coefficient buffer — 64-bit products
 * inside, 32 bits between the passes —, then the columns, rounding shift
 * 4/5/6/6 (none after the WHT); an inter block's residual is added and clipped
 * to 10 bits, an intra block's goes to the grid, saturated to int16, which no
 * sum with a sample notices. c: the lane's row, at: its TX's place. */
template <int N, class T, bool LIST>
__device__ __forceinline__ void hbd_tx_passes(HbdSmem &s, const int (&c)[N], int at, uint2 tx, bool any, bool mine, int i)
{
    const bool lossless = s.jc.lossless;
    const int p = TxRef::plane(tx.y), type = TxRef::type(tx.y);
    const bool wht = N == 4 && lossless;
    int32_t *buf = s.tmp.i;
    T v[N];
    if (mine && any) {               /* a row of zeros stays as it is */
#pragma unroll
        for (int k = 0; k < N; k++) v[k] = T(c[k]);
        if (wht) iwht4(v, true);
        else itx1<N>(v, type >= 2);
#pragma unroll
        for (int k = 0; k < N; k += 4)
            *reinterpret_cast<int4 *>(&buf[tx_word(at + i * N + k)]) =
                make_int4((int)v[k].v, (int)v[k + 1].v, (int)v[k + 2].v, (int)v[k + 3].v);
    }
    __syncwarp();
    if (mine) {
#pragma unroll
        for (int k = 0; k < N; k++) v[k] = T(buf[tx_word(at + k * N + i)]);
        if (wht) iwht4(v, false);
        else itx1<N>(v, type & 1);
        const int sh = wht ? 0 : N == 4 ? 4 : (N == 8 ? 5 : 6), round = wht ? 0 : 1 << (sh - 1);
        const int x = TxRef::x<LIST>(tx.y) + i, y = TxRef::y<LIST>(tx.y);
        const bool intra = tx.y & TxRef::kIntra;
        int16_t *r = s.res + plane_at(p, x, y);
        uint16_t *d = &HT(s, p, x, y);
        const int rp = p ? 32 : 64, dp = p ? kHCP : kHYP;
#pragma unroll
        for (int k = 0; k < N; k++) {
            const auto q = (v[k].v + round) >> sh;
            const int e = q < -32768 ? -32768 : (q > 32767 ? 32767 : (int)q);
            if (LIST && (x >= (p ? 32 : 64) || y + k >= (p ? 32 : 64))) continue;
            if (intra) r[k * rp] = (int16_t)e;
            else d[k * dp] = (uint16_t)clampi((int)d[k * dp] + e, 0, kHbdMax);
        }
    }
}

template <int N, bool LIST>
__device__ __noinline__ void hbd_tx_wide(int at, uint2 tx, bool any, bool mine, int i)
{
    HbdSmem &s = smem_as<HbdSmem>();
    int c[N];
    for (int k = 0; k < N; k++) c[k] = s.tmp.i[tx_word(at + i * N + k)];
    __syncwarp();
    hbd_tx_passes<N, wl, LIST>(s, c, at, tx, any, mine, i);
}

/* The butterflies run on 32-bit values (wn) unless one of the warp's
 * coefficients is outside +-2^18 (a 10-bit stream's reach +-2^17): then on
 * 64-bit ones (wl), with the same results. */
template <int N, bool LIST>
__device__ __forceinline__ void hbd_tx_unit(HbdSmem &s, int first, int count, bool staged, unsigned c_base, int slot, int lane)
{
    const int sub = lane / N, i = lane & (N - 1);
    const bool on = sub < count;
    const uint2 tx = s.tx[first + (on ? sub : 0)];
    const bool go = on && !(tx.y & TxRef::kNone);
    const int at = !go ? 0 : staged ? (int)(tx.x - c_base) : slot + sub * N * N;
    if (!staged) {                   /* bring the TXs here */
        if (go)
            for (int k = 0; k < N; k++) s.tmp.i[tx_word(at + k * N + i)] = __ldg(s.jc.coeffs32 + tx.x + k * N + i);
        __syncwarp();
    }
    int c[N], any = 0;
    unsigned wide = 0;
#pragma unroll
    for (int k = 0; k < N; k += 4) {
        const int4 w = go ? *reinterpret_cast<const int4 *>(&s.tmp.i[tx_word(at + i * N + k)]) : make_int4(0, 0, 0, 0);
        c[k] = w.x;
        c[k + 1] = w.y;
        c[k + 2] = w.z;
        c[k + 3] = w.w;
        any |= w.x | w.y | w.z | w.w;
        wide |= (((unsigned)w.x + (1u << 18)) | ((unsigned)w.y + (1u << 18)) | ((unsigned)w.z + (1u << 18)) |
                 ((unsigned)w.w + (1u << 18))) >> 19;
    }
    const uint32_t live = __ballot_sync(0xffffffffu, any != 0);
    if (live) {
        const bool mine = go && (N == 32 || ((live >> (sub * N)) & ((1u << (N & 31)) - 1u)));
        if (__any_sync(0xffffffffu, wide != 0)) hbd_tx_wide<N, LIST>(at, tx, any != 0, mine, i);
        else hbd_tx_passes<N, wn, LIST>(s, c, at, tx, any != 0, mine, i);
    }
    __syncwarp();
}

/* Every residual of blocks [lo, hi) of the SB, whole CTA; staged: their
 * coefficients are in the permuted buffer, from c_base on. */
template <bool LIST>
__device__ __noinline__ void hbd_residual(int lo, int hi, int nb, bool staged, unsigned c_base, int sbx, int sby)
{
    HbdSmem &s = smem_as<HbdSmem>();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const cvp9_job_t &job = s.jc;
    for (int i = tid; i < kResidGrid / 8; i += kHbdThreads) reinterpret_cast<uint4 *>(s.res)[i] = make_uint4(0u, 0u, 0u, 0u);
    list_txs<LIST, true>(s, lo, hi, nb, job.num_coeffs, tid, kHbdThreads,
             [&](const HbdBlk &b, int p, int &txl, int &nx, int &ny) {
                 int pbw;
                 plane_layout(b, job, sbx + b.x, sby + b.y, p, txl, nx, ny, pbw);
                 if (b.flags & 2) nx = ny = 0;
             },
             [&](const HbdBlk &b, int p, int txl) {
                 return (b.flags & 1) && p == 0 && !job.lossless && txl < 3 && b.ymode < 10 ? (int)c_tx_type[b.ymode] : 0;
             });
    if (tid == 0 && s.ntx[0] + s.ntx[1] + s.ntx[2] + s.ntx[3] > kMaxTasks) atomicOr(job.status, (unsigned)CVP9_JOB_TOO_MANY);
    const int n32 = s.ntx[3], n16 = s.ntx[2], n8 = s.ntx[1];
    deal_txs(s.ntx, 1, warp, kHbdWarps, [&](auto n, int first, int count, int) {
        constexpr int N = decltype(n)::value;
        const int before = N == 32 ? 0 : N == 16 ? n32 * 1024 : N == 8 ? n32 * 1024 + n16 * 256 : n32 * 1024 + n16 * 256 + n8 * 64;
        const int skip = N == 32 ? 0 : N == 16 ? n32 : N == 8 ? n32 + n16 : n32 + n16 + n8;
        hbd_tx_unit<N, LIST>(s, first, count, staged, c_base, before + (first - skip) * N * N, lane);
    });
    __syncthreads();
}

__device__ __forceinline__ IntraView<uint16_t> hbd_view(HbdSmem &s)
{
    IntraView<uint16_t> V;
    V.tile0 = &HT(s, 0, 0, 0);
    V.col0 = s.col;
    V.res = s.res;
    return V;
}

/* The intra TXs of the SB's nb blocks, their levels, the sorted quads. */
__device__ __noinline__ void hbd_plan(int nb, int sbx, int sby)
{
    HbdSmem &s = smem_as<HbdSmem>();
    const cvp9_job_t &job = s.jc;
    IntraWork &W = s.tmp.w;
    const int tid = threadIdx.x;
    intra_fill_cols(hbd_view(s), tid, kHbdThreads);
    int ntask;
    const int at = hbd_scan(s, tid < nb && (s.blk[tid].flags & 1) ? intra_tx_count(s.blk[tid], job, sbx, sby) : 0, &ntask);
    ntask = min(ntask, kMaxTasks);
    s.it_base[tid] = (uint16_t)min(at, 0xFFFF);
    for (int i = tid; i < kMaxTasks; i += kHbdThreads) W.own[i] = 0;
    if (tid < 96) (&W.prow[0][0])[tid] = 0u;
    __syncthreads();
    for (int t = tid; t < ntask; t += kHbdThreads) {
        const int b = find_base(s.it_base, nb, t);
        intra_tx_task(W, s.blk[b], job, sbx, sby, t - s.it_base[b], t, true);
    }
    __syncthreads();
    intra_tx_levels(W, ntask, tid, kHbdThreads);
    __syncthreads();
    intra_sort<CVP9_ARITH_FULL, uint16_t>(W, s.cell, ntask, tid, kHbdThreads);
}

/* Claim a block's coefficients [begin, end) of a span of at most kResidGrid, a
 * bit per four from base on; whether another block has one of them. */
__device__ __forceinline__ bool hbd_claim(uint32_t *map, unsigned begin, unsigned end, unsigned base)
{
    const unsigned g0 = (begin - base) >> 2, g1 = ((end - base) >> 2) - 1u;
    bool shared = false;
    for (unsigned w = g0 >> 5; w <= g1 >> 5; w++) {
        const unsigned a = w == g0 >> 5 ? g0 & 31u : 0u, z = w == g1 >> 5 ? g1 & 31u : 31u;
        const uint32_t m = ((2u << z) - 1u) & ~((1u << a) - 1u);
        shared |= (atomicOr(&map[w], m) & m) != 0u;
    }
    return shared;
}

/* Intra block b on its own, its residual in the grid. */
__device__ __noinline__ void hbd_ordered(int b, int sbx, int sby)
{
    HbdSmem &s = smem_as<HbdSmem>();
    IntraWork &W = s.tmp.w;
    const int tid = threadIdx.x;
    const IntraView<uint16_t> V = hbd_view(s);
    intra_fill_cols(V, tid, kHbdThreads);
    const int n = min(intra_tx_count(s.blk[b], s.jc, sbx, sby), kMaxTasks);
    for (int k = tid; k < n; k += kHbdThreads) intra_tx_task(W, s.blk[b], s.jc, sbx, sby, k, k, false);
    if (tid == 0) W.ntask = n;
    __syncthreads();
    intra_run_ordered<CVP9_ARITH_FULL, kHbdMax, uint16_t>(W, V, W.ntask, tid, kHbdThreads);
    __syncthreads();
}

__device__ __noinline__ void hbd_neighbours(unsigned need, int sb)
{
    HbdSmem &s = smem_as<HbdSmem>();
    wait_halo<HbdSmem, uint16_t>(s, hbd_view(s), need, sb, true, kHbdMid - 1, kHbdMid + 1, threadIdx.x, kHbdThreads);
}

__device__ __forceinline__ void hbd_publish(HbdSmem &s, int sb, int sbx, int sby, int tid)
{
    publish<uint16_t>(s.jc, sb, sbx, sby, tid, [&](int p, int x, int y) { return HT(s, p, x, y); });
}

__device__ __noinline__ void hbd_intra(unsigned need, int sb, int sbx, int sby)
{
    HbdSmem &s = smem_as<HbdSmem>();
    wait_halo<HbdSmem, uint16_t>(s, hbd_view(s), need, sb, true, kHbdMid - 1, kHbdMid + 1, threadIdx.x, kHbdThreads);
    intra_run<CVP9_ARITH_FULL, kHbdMax, uint16_t>(s.tmp.w, hbd_view(s), threadIdx.x, kHbdThreads);
    hbd_publish(s, sb, sbx, sby, threadIdx.x);
}

} /* namespace */

__global__ void __launch_bounds__(kHbdThreads, 3) k_hbd_recon(const cvp9_job_t *__restrict__ jobs,
                                                              const uint32_t *__restrict__ tickets,
                                                              uint32_t n_tickets, uint32_t *ticket_counter)
{
    HbdSmem &s = smem_as<HbdSmem>();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const cvp9_job_t &job = s.jc;
    uint32_t *const spans = reinterpret_cast<uint32_t *>(s.res);     /* two bit maps, until the predictions */
    for (;;) {
        __syncthreads();
        if (tid == 0) s.ticket = (int)atomicAdd(ticket_counter, 1u);
        __syncthreads();
        const int ticket = s.ticket;
        if (ticket >= (int)n_tickets) return;
        const uint32_t code = tickets[ticket];
        const cvp9_job_t *gj = jobs + (code >> 20);
        {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(gj);
            uint32_t *dst = reinterpret_cast<uint32_t *>(&s.jc);
            for (int i = tid; i < (int)(sizeof(cvp9_job_t) / 4); i += kHbdThreads) dst[i] = src[i];
        }
        const int sb = (int)(code & 0xFFFFFu);
        const int g_sb_cols = gj->sb_cols;
        const int sbr = sb / g_sb_cols, sbc = sb - sbr * g_sb_cols;
        const int sbx = sbc * 64, sby = sbr * 64;
        const uint32_t *rg = gj->sb_range + 4 * sb;
        const uint32_t start = rg[0], end = rg[1], groups = rg[2];
        const bool layout_bad = (*(volatile uint32_t *)gj->status & CVP9_JOB_BAD_BLOCK) != 0;
        const bool bad = groups > 1 || end < start || end > gj->num_blocks ||
                         (groups && end - start > (uint32_t)kHbdMaxBlocks);
        int nb = (groups && !bad && !layout_bad) ? (int)(end - start) : 0;
        /* the tile at 512, no cell claimed */
        {
            const uint4 mid = make_uint4(0x02000200u, 0x02000200u, 0x02000200u, 0x02000200u);
            uint4 *t4 = reinterpret_cast<uint4 *>(s.ty);
            for (int i = tid; i < (65 * kHYP + 2 * 33 * kHCP) / 8; i += kHbdThreads) t4[i] = mid;
        }
        for (int i = tid; i < 256; i += kHbdThreads) s.cell[i] = 0;
        if (tid < 16) s.rows[tid] = 0;
        if (tid < 64 + kResidGrid / 128) spans[tid] = 0;
        if (tid == 0) { s.needs = 0u; s.c_lo = 0xFFFFFFFFu; s.c_hi = 0u; s.c_sum = 0u; }
        __syncthreads();

        /* 1. blocks (each inside this SB, 4-aligned, 4..64 px, tx_size <= 3,
         * sub-8x8 ones on the 8x8 grid), and the 4x4 cells they write */
        bool my_intra = false, my_bad = false, my_seq = false;
        if (tid < nb) {
            const vp9_macroblock_info_t g = job.blocks[start + tid];
            const int lx = (int)g.x - sbx, ly = (int)g.y - sby;
            const bool sub8 = g.width < 8 || g.height < 8;
            const int bw = sub8 ? 8 : g.width, bh = sub8 ? 8 : g.height;
            /* ... and a transform no larger than the block */
            my_bad = lx < 0 || ly < 0 || (lx & 3) || (ly & 3) || (g.width & 3) || (g.height & 3) || g.width < 4 ||
                     g.height < 4 || lx + g.width > 64 || ly + g.height > 64 || g.x >= job.W || g.y >= job.H ||
                     g.tx_size > 3 || (sub8 && ((lx & 7) || (ly & 7))) || (4 << g.tx_size) > min(bw, bh);
            HbdBlk b;
            b.x = (uint8_t)(my_bad ? 0 : lx);
            b.y = (uint8_t)(my_bad ? 0 : ly);
            b.w = g.width;
            b.h = g.height;
            b.cw = (uint8_t)max(0, min(bw, job.W - (int)g.x));
            b.ch = (uint8_t)max(0, min(bh, job.H - (int)g.y));
            b.ccw = (uint8_t)max(0, min(max(bw / 2, 4), job.CW - (int)g.x / 2));
            b.cch = (uint8_t)max(0, min(max(bh / 2, 4), job.CH - (int)g.y / 2));
            b.txl = g.tx_size;
            b.flags = (uint8_t)((g.is_intra ? 1 : 0) | (g.skip ? 2 : 0));
            b.ymode = g.y_mode;
            b.uvmode = g.uv_mode;
            b.ref0 = g.ref_frame[0];
            b.ref1 = g.is_intra ? 0 : g.ref_frame[1];
            b.mvx = g.mv[0][0];
            b.mvy = g.mv[0][1];
            b.mv1x = g.mv[1][0];
            b.mv1y = g.mv[1][1];
            b.coeff = g.coeff_offset;
            s.blk[tid] = b;
            my_intra = g.is_intra != 0;
            /* TXs that do not tile their block, or whose chroma TXs straddle
             * 4x4 cells: list order */
            const int n = 4 << (g.tx_size & 3), m = min(n, 4 << max_tx_for(max(4, bw / 2), max(4, bh / 2)));
            my_seq = ((bw | bh) & (n - 1)) || (!sub8 && (((bw | bh) >> 1) & (m - 1))) || ((lx | ly) & 7);
        }
        if (__syncthreads_or(my_bad)) {
            if (tid == 0) atomicOr(job.status, (unsigned)CVP9_JOB_BAD_BLOCK);
            nb = 0;
            my_intra = my_seq = false;
        }
        if (tid < nb) {
            /* cells of the luma region a block writes (a sub-8x8 block its 8x8) */
            const HbdBlk &b = s.blk[tid];
            my_seq |= claim_cells(s.rows, b.x >> 2, (b.x + b.cw - 1) >> 2, b.y >> 2, (b.y + b.ch - 1) >> 2);
        }
        /* stage the coefficients in the permuted buffer, where 16-byte copies
         * can: every block's start a multiple of 4, the span no longer than the
         * SB's samples. The row passes go over the coefficients in place, so
         * only where no two blocks share any. A parser's spans follow one
         * another without gaps, which takes little to see: every one begins
         * at the first coefficient or where one ends (so there is no gap), and
         * they have as many coefficients as the whole (so none is there
         * twice). Other spans are compared coefficient by coefficient:
         * doing so for all took 1.6% of the kernel, leaving those with gaps or
         * out of order unstaged 14% of theirs. */
        bool odd = false;
        unsigned begin = 0u, ncoef = 0u;         /* this block's coefficients */
        if (tid < nb && !(s.blk[tid].flags & 2)) {
            const HbdBlk &b = s.blk[tid];
            for (int p = 0; p < 3; p++) {
                int txl, nx, ny, pbw;
                plane_layout(b, job, sbx + b.x, sby + b.y, p, txl, nx, ny, pbw);
                ncoef += (unsigned)(nx * ny) << (4 + 2 * txl);
            }
            begin = b.coeff;
            odd = ncoef && ((begin & 3u) || begin + ncoef < begin);
        }
        {
            const unsigned lo = __reduce_min_sync(0xffffffffu, ncoef ? begin : 0xFFFFFFFFu);
            const unsigned hi = __reduce_max_sync(0xffffffffu, ncoef ? begin + ncoef : 0u), sum = __reduce_add_sync(0xffffffffu, ncoef);
            if (lane == 0) { atomicMin(&s.c_lo, lo); atomicMax(&s.c_hi, hi); atomicAdd(&s.c_sum, sum); }
            /* ends by number of four, modulo 2048: the span has fewer */
            if (ncoef) atomicOr(&spans[((begin + ncoef) >> 7) & 63u], 1u << (((begin + ncoef) >> 2) & 31u));
        }
        const bool any_intra = __syncthreads_or(my_intra) != 0;
        const unsigned c_base = s.c_lo, c_hi = s.c_hi;
        const bool tight = !ncoef || begin == c_base || ((spans[(begin >> 7) & 63u] >> ((begin >> 2) & 31u)) & 1u);
        bool staged = c_hi > c_base && c_hi <= job.num_coeffs && c_hi - c_base <= (unsigned)kResidGrid &&
                      !((uintptr_t)job.coeffs32 & 15);
        if (staged && (__syncthreads_or(odd || !tight) || s.c_sum != c_hi - c_base))
            staged = !__syncthreads_or(odd || (ncoef && hbd_claim(spans + 64, begin, begin + ncoef, c_base)));
        if (staged)
            for (unsigned e = 4u * (unsigned)tid; e < c_hi - c_base; e += 4u * kHbdThreads)
                cp_async16(&s.tmp.i[tx_word((int)e)], job.coeffs32 + c_base + e);
        cp_async_commit();
        if (any_intra) {
            const int mb = lane * kHbdWarps + warp;     /* the blocks dealt over the warps */
            const HbdBlk &m = s.blk[mb];
            warp_spread(mb < nb ? (((m.x + m.cw + 3) >> 2) - (m.x >> 2)) * (((m.y + m.ch + 3) >> 2) - (m.y >> 2)) : 0, lane,
                        [&](int i, int k) {
                            const HbdBlk &b = s.blk[i * kHbdWarps + warp];
                            own_cell(s.cell, i * kHbdWarps + warp, b.x >> 2, (b.x + b.cw - 1) >> 2, b.y >> 2, k);
                        });
            __syncthreads();
        }
        /* an intra block reading samples of a block later in the list: the
         * superblock runs in list order */
        unsigned need = 0;
        if (tid < nb && my_intra) {
            const HbdBlk &b = s.blk[tid];
            const int cx0 = b.x >> 2, cy0 = b.y >> 2, cx1 = (b.x + b.cw - 1) >> 2, cy1 = (b.y + b.ch - 1) >> 2;
            if (cy0 > 0) for (int cx = max(0, cx0 - 1); cx <= cx1; cx++) my_seq |= s.cell[(cy0 - 1) * 16 + cx] > tid;
            if (cx0 > 0) for (int cy = cy0; cy <= cy1; cy++) my_seq |= s.cell[cy * 16 + cx0 - 1] > tid;
            need = intra_needs(b.x, b.y);
        }
        need = __reduce_or_sync(0xffffffffu, need);
        if (lane == 0 && need) atomicOr(&s.needs, need);
        const bool seq = __syncthreads_or(my_seq) != 0;

        /* 2. reconstruct: what reads no neighbour, then the intra blocks level
         * by level; or block by block in list order */
        if (!seq) {
            hbd_predict(0, nb, nb, sbx, sby);
            cp_async_wait_all();
            __syncthreads();
            hbd_residual<false>(0, nb, nb, staged, c_base, sbx, sby);
            if (any_intra) {
                hbd_plan(nb, sbx, sby);
                hbd_intra(s.needs, sb, sbx, sby);
            }
        } else {
            cp_async_wait_all();
            __syncthreads();
            if (any_intra) hbd_neighbours(7u, sb);
            for (int i = 0; i < nb; i++) {
                hbd_predict(i, i + 1, nb, sbx, sby);
                hbd_residual<true>(i, i + 1, nb, false, 0u, sbx, sby);
                if (s.blk[i].flags & 1) hbd_ordered(i, sbx, sby);
            }
        }

        /* 3. the samples the neighbours read, release the SB, then the whole
         * tile (clipped to the frame) */
        {
            uint16_t *out = reinterpret_cast<uint16_t *>(job.out);
            const int vw = min(64, job.W - sbx), vh = min(64, job.H - sby);
            if (seq || !any_intra) hbd_publish(s, sb, sbx, sby, tid);
            if (tid == 0 && bad)
                atomicOr(job.status, (unsigned)CVP9_JOB_BAD_ORDER |
                                     ((groups && end >= start && end - start > (uint32_t)kHbdMaxBlocks) ? (unsigned)CVP9_JOB_TOO_MANY : 0u));
            /* four samples a store: sizes are multiples of 8 */
            uint16_t *U = out + (size_t)job.W * job.H, *Vp = U + (size_t)job.CW * job.CH;
            for (int i = tid; i < 64 * 16; i += kHbdThreads) {
                const int r = i >> 4, c = (i & 15) * 4;
                if (r < vh && c < vw)
                    *reinterpret_cast<uint2 *>(out + (size_t)(sby + r) * job.W + sbx + c) =
                        *reinterpret_cast<const uint2 *>(&HT(s, 0, c, r));
            }
            const int cvw = min(32, job.CW - (sbx >> 1)), cvh = min(32, job.CH - (sby >> 1));
            for (int i = tid; i < 2 * 32 * 8; i += kHbdThreads) {
                const int p = i >> 8, r = (i >> 3) & 31, c = (i & 7) * 4;
                if (r < cvh && c < cvw)
                    *reinterpret_cast<uint2 *>((p ? Vp : U) + (size_t)((sby >> 1) + r) * job.CW + (sbx >> 1) + c) =
                        *reinterpret_cast<const uint2 *>(&HT(s, 1 + p, c, r));
            }
        }
    }
}

__global__ void k_nv12_pack(const cvp9_job_t *__restrict__ jobs)
{
    const cvp9_job_t &job = jobs[blockIdx.y];
    if ((job.lf_tiled && !job.full) || !job.nv12) return;
    size_t ny = (size_t)job.W * job.H, nc = (size_t)job.CW * job.CH;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ny) job.nv12[i] = job.out[i];
    if (i < nc) {
        size_t gy = i / job.CW, gx = i % job.CW;
        job.nv12[ny + gy * 2 * job.CW + 2 * gx] = job.out[ny + i];
        job.nv12[ny + gy * 2 * job.CW + 2 * gx + 1] = job.out[ny + nc + i];
    }
}

/* ── Coefficient upload over PCIe, REFCPU ────────────────────────────────
 * The dense coefficient array interleaves each block's luma TXs with its
 * chroma TXs; REFCPU reads only the luma ones (vp9_reconstruct.c:336-360).
 * A warp per block copies that span, [coeff_offset, + (cw/n)(ch/n) n^2),
 * from the page-locked host array to the same offset of the device array
 * with 16-byte reads when both sides share their alignment; the chroma
 * coefficients never cross the bus. */
__global__ void __launch_bounds__(256) k_gather_luma(const cvp9_job_t *__restrict__ jobs, uint32_t *bytes)
{
    const cvp9_job_t &job = jobs[blockIdx.y];
    const int16_t *src = job.coeffs_src;
    if (!src) return;
    int16_t *dst = const_cast<int16_t *>(job.coeffs);
    const int lane = threadIdx.x & 31;
    uint32_t moved = 0;
    for (uint32_t bi = blockIdx.x * 8u + (threadIdx.x >> 5); bi < job.num_blocks; bi += gridDim.x * 8u) {
        const uint32_t *g = reinterpret_cast<const uint32_t *>(job.blocks + bi);
        const uint32_t g0 = g[0], g1 = g[1], g5 = g[5], g6 = g[6];
        const int x = (int)(g0 & 0xffffu), y = (int)(g0 >> 16);
        const int w = (int)(g1 & 0xffu), h = (int)((g1 >> 8) & 0xffu), tx = (int)((g1 >> 16) & 0xffu);
        if ((g5 & 0xffu) || tx > 3 || x >= job.W || y >= job.H) continue;
        const int n = 4 << tx;
        const int cw = min(w, job.W - x), ch = min(h, job.H - y);
        const uint64_t a = g6;
        uint64_t e = a + (uint64_t)((cw / n) * (ch / n)) * (uint64_t)(n * n);
        if (e > job.num_coeffs) e = job.num_coeffs;
        if (a >= e) continue;
        const char *s = reinterpret_cast<const char *>(src + a);
        char *d = reinterpret_cast<char *>(dst + a);
        const uint64_t len = (e - a) * 2;
        if ((((uintptr_t)s ^ (uintptr_t)d) & 15) == 0) {
            const uint64_t head = (16 - ((uintptr_t)s & 15)) & 15;
            const uint64_t h2 = head < len ? head : len;
            for (uint64_t o = 2 * lane; o < h2; o += 64)
                *reinterpret_cast<int16_t *>(d + o) = *reinterpret_cast<const int16_t *>(s + o);
            const uint64_t nv = (len - h2) / 16;
            const uint4 *sv = reinterpret_cast<const uint4 *>(s + h2);
            uint4 *dv = reinterpret_cast<uint4 *>(d + h2);
            for (uint64_t v = lane; v < nv; v += 32) dv[v] = sv[v];
            for (uint64_t o = h2 + nv * 16 + 2 * lane; o < len; o += 64)
                *reinterpret_cast<int16_t *>(d + o) = *reinterpret_cast<const int16_t *>(s + o);
        } else {
            for (uint64_t o = 2 * lane; o < len; o += 64)
                *reinterpret_cast<int16_t *>(d + o) = *reinterpret_cast<const int16_t *>(s + o);
        }
        moved += (uint32_t)len;
    }
    if (lane == 0 && moved) atomicAdd(bytes, moved);
}

/* Sparse coefficient upload: the caller's (index, value) list of a frame
 * is scattered into its zeroed dense array, which the reconstruction then
 * reads exactly as if the dense array had been uploaded. */
__global__ void __launch_bounds__(256) k_scatter_coeffs(const cvp9_job_t *__restrict__ jobs)
{
    const cvp9_job_t &job = jobs[blockIdx.y];
    const uint32_t n = job.sp_n;
    if (job.sp_val32) {
        /* profile 2: int32 dequantised values into coeffs32 */
        int32_t *dst = const_cast<int32_t *>(job.coeffs32);
        for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
            const uint32_t p = job.sp_pos[k];
            if (p < job.num_coeffs) dst[p] = job.sp_val32[k];
        }
        return;
    }
    int16_t *dst = const_cast<int16_t *>(job.coeffs);
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t p = job.sp_pos[k];
        if (p < job.num_coeffs) dst[p] = job.sp_val[k];
    }
}

/* Packed coefficient upload (format of cvp9_pack_coeffs): a CTA per (page,
 * frame) rebuilds 65536 coefficients of the dense array — a dense page is
 * copied, an entry page is zero-filled and then scattered. A malformed
 * page (data past the buffer, counts out of range) is left alone and sets
 * bit (job index) % 32 of *err, which the host reads with the step. */
__global__ void __launch_bounds__(256) k_unpack_coeffs(const cvp9_job_t *__restrict__ jobs, uint32_t *err)
{
    const cvp9_job_t &job = jobs[blockIdx.y];
    const uint32_t *pk = job.packed;
    if (!pk) return;
    const uint32_t nw = job.packed_words, np = nw ? pk[0] : 0u;
    if (1u + 2u * (uint64_t)np > nw) {
        if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(err + blockIdx.y, 1u);
        return;
    }
    for (uint32_t p = blockIdx.x; p < np; p += gridDim.x) {
        const uint32_t base = p << 16;
        if (p >= 65536u || base >= job.num_coeffs) break;
        const uint32_t st = pk[1 + 2 * p], cnt = pk[2 + 2 * p];
        const uint32_t s0 = st & 0x7fffffffu;
        const uint32_t len = min(65536u, job.num_coeffs - base);
        const bool dense = st >> 31;
        const uint64_t words = dense ? ((uint64_t)len + 1) / 2 : cnt;
        if ((s0 & 3u) || (dense && cnt != len) || (!dense && cnt > (len + 1) / 2) || s0 + words > nw) {
            if (threadIdx.x == 0) atomicOr(err + blockIdx.y, 1u);
            continue;
        }
        int16_t *dst = const_cast<int16_t *>(job.coeffs) + base;     /* 16-byte aligned */
        const uint32_t *src = pk + s0;                               /* 16-byte aligned */
        uint4 *d4 = reinterpret_cast<uint4 *>(dst);
        const uint32_t nv = len >> 3;
        if (dense) {
            const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
            for (uint32_t v = threadIdx.x; v < nv; v += blockDim.x) d4[v] = __ldg(s4 + v);
            const int16_t *s16 = reinterpret_cast<const int16_t *>(src);
            for (uint32_t k = nv * 8 + threadIdx.x; k < len; k += blockDim.x) dst[k] = s16[k];
        } else {
            for (uint32_t v = threadIdx.x; v < nv; v += blockDim.x) d4[v] = make_uint4(0u, 0u, 0u, 0u);
            for (uint32_t k = nv * 8 + threadIdx.x; k < len; k += blockDim.x) dst[k] = 0;
            __syncthreads();
            for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x) {
                const uint32_t e = __ldg(src + k), o = e & 0xffffu;
                if (o < len) dst[o] = (int16_t)(e >> 16);
            }
        }
        __syncthreads();
    }
}

/* ── C-ABI launch shims ─────────────────────────────────────────────────── */

/* Launch a kernel that starts with grid_dependency_wait(): with `early`, its
 * CTAs may be placed before the kernel in front has ended. */
template <class... P, class... A>
static cudaError_t launch(bool early, void (*k)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute a = {};
    c.gridDim = grid;
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&c, k, (P)args...);
}

extern "C" {

size_t cvp9k_recon_smem_bytes(void) { return sizeof(ReconSmem); }

int cvp9k_launch_scatter(const cvp9_job_t *jobs, int njobs, uint32_t max_n, cudaStream_t st)
{
    if (njobs <= 0 || max_n == 0) return 0;
    unsigned gx = (max_n + 255u) / 256u;
    if (gx > 4096u) gx = 4096u;
    k_scatter_coeffs<<<dim3(gx, (unsigned)njobs), 256, 0, st>>>(jobs);
    return (int)cudaGetLastError();
}

int cvp9k_launch_unpack(const cvp9_job_t *jobs, int njobs, uint32_t max_pages, uint32_t *err, cudaStream_t st)
{
    if (njobs <= 0 || max_pages == 0) return 0;
    const unsigned gx = max_pages < 65535u ? max_pages : 65535u;
    k_unpack_coeffs<<<dim3(gx, (unsigned)njobs), 256, 0, st>>>(jobs, err);
    return (int)cudaGetLastError();
}

/* One job per blockIdx.y; 16-byte streaming copies (both ends are
 * 256-byte aligned arena ranges), the tail bytewise. */
__global__ void __launch_bounds__(256) k_collect(const cvp9_job_t *__restrict__ jobs)
{
    const cvp9_job_t &job = jobs[blockIdx.y];
    uint8_t *dst = job.dl;
    if (!dst) return;
    const uint8_t *src = job.out;
    const size_t n = (size_t)job.W * job.H + 2 * (size_t)job.CW * job.CH;
    const size_t n16 = n >> 4;
    const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
    uint4 *d4 = reinterpret_cast<uint4 *>(dst);
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n16; i += (size_t)gridDim.x * 256)
        __stcs(d4 + i, __ldcs(s4 + i));
    if (blockIdx.x == 0)
        for (size_t i = (n16 << 4) + threadIdx.x; i < n; i += 256) dst[i] = src[i];
}

int cvp9k_launch_collect(const cvp9_job_t *jobs, int njobs, size_t max_bytes, cudaStream_t st)
{
    if (njobs <= 0 || !max_bytes) return 0;
    /* about four CTAs per SM in all, at least one per 256 KB of a frame */
    size_t gx = (max_bytes + (256u << 10) - 1) >> 18;
    const size_t want = (size_t)(4 * 148 + njobs - 1) / (size_t)njobs;
    if (gx > want) gx = want;
    if (gx < 1) gx = 1;
    k_collect<<<dim3((unsigned)gx, (unsigned)njobs), 256, 0, st>>>(jobs);
    return (int)cudaGetLastError();
}

int cvp9k_launch_gather(const cvp9_job_t *jobs, int njobs, int max_blocks, uint32_t *bytes, cudaStream_t st)
{
    if (njobs <= 0 || max_blocks <= 0) return 0;
    int gx = (max_blocks + 7) / 8;
    if (gx > 2048) gx = 2048;
    k_gather_luma<<<dim3((unsigned)gx, (unsigned)njobs), 256, 0, st>>>(jobs, bytes);
    return (int)cudaGetLastError();
}

int cvp9k_upload_dct_basis(const double *basis, int count)
{
    if (count != 16 + 64 + 256 + 1024) return -1;
    if (cudaMemcpyToSymbol(c_dct, basis, sizeof(double) * (size_t)count) != cudaSuccess) return -1;
    return cudaMemcpyToSymbol(g_dct, basis, sizeof(double) * (size_t)count) == cudaSuccess ? 0 : -1;
}

int cvp9k_configure(void)
{
    {
        static const int taps[16][8] = CVP9_SUBPEL_REGULAR_INIT;
        uint32_t pk[16][2];
        for (int f = 0; f < 16; f++)
            for (int h = 0; h < 2; h++) {
                uint32_t w = 0;
                for (int t = 0; t < 4; t++) w |= (uint32_t)(uint8_t)(int8_t)taps[f][4 * h + t] << (8 * t);
                pk[f][h] = w;
            }
        if (cudaMemcpyToSymbol(c_subpel_pk, pk, sizeof(pk)) != cudaSuccess) return -1;
    }
    {
        static const int taps4[4][16][8] = { CVP9_SUBPEL_REGULAR_INIT, CVP9_SUBPEL_SMOOTH_INIT,
                                             CVP9_SUBPEL_SHARP_INIT, CVP9_SUBPEL_BILINEAR_INIT };
        uint32_t pk[4][16][2];
        for (int k = 0; k < 4; k++)
            for (int f = 0; f < 16; f++)
                for (int h = 0; h < 2; h++) {
                    uint32_t w = 0;
                    for (int t = 0; t < 4; t++) {
                        const int v = taps4[k][f][4 * h + t];
                        /* phase 0 (the centre tap alone, 128) is not packed:
                         * tap8 takes the centre sample for it */
                        if (f && (v < -128 || v > 127)) return -1;
                        w |= (uint32_t)(uint8_t)(int8_t)v << (8 * t);
                    }
                    pk[k][f][h] = w;
                }
        if (cudaMemcpyToSymbol(c_subpel4_pk, pk, sizeof(pk)) != cudaSuccess) return -1;
    }
    size_t smem = sizeof(ReconSmem);
    if (cudaFuncSetAttribute(k_recon<CVP9_ARITH_REFCPU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -1;
    if (cudaFuncSetAttribute(k_recon<CVP9_ARITH_SPEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -1;
    if (cudaFuncSetAttribute(k_recon<CVP9_ARITH_FULL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -1;
    /* all of the unified L1/shared storage as shared memory: three CTAs per SM */
    cudaFuncSetAttribute(k_recon<CVP9_ARITH_REFCPU>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(k_recon<CVP9_ARITH_SPEC>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(k_recon<CVP9_ARITH_FULL>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(k_inter<CVP9_ARITH_REFCPU, 5>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(k_inter<CVP9_ARITH_REFCPU, 6>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(k_inter<CVP9_ARITH_SPEC, 5>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaFuncSetAttribute(k_inter<CVP9_ARITH_SPEC, 6>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (cudaFuncSetAttribute(k_hbd_recon, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(HbdSmem)) != cudaSuccess)
        return -1;
    cudaFuncSetAttribute(k_hbd_recon, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (cudaFuncSetAttribute(k_lf_full<uint16_t, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(LfSmem<uint16_t>)) != cudaSuccess)
        return -1;
    /* Load every kernel the launcher can pick now. With lazy module loading
     * (the CUDA 12 default) a kernel's code is loaded at its first launch,
     * which stalls the device for tens of milliseconds; the tuner's first
     * trial of an inter path would otherwise take that stall inside a
     * serving step. */
    const void *fns[] = {
        (const void *)k_scan_blocks, (const void *)k_lf_mimap, (const void *)k_compact,
        (const void *)k_recon<CVP9_ARITH_REFCPU>, (const void *)k_recon<CVP9_ARITH_SPEC>,
        (const void *)k_recon<CVP9_ARITH_FULL>,
        (const void *)k_inter<CVP9_ARITH_REFCPU, 5>, (const void *)k_inter<CVP9_ARITH_REFCPU, 6>,
        (const void *)k_inter<CVP9_ARITH_SPEC, 5>, (const void *)k_inter<CVP9_ARITH_SPEC, 6>,
        (const void *)k_pred<CVP9_ARITH_SPEC, kPredMinB>, (const void *)k_pred<CVP9_ARITH_REFCPU, kPredMinB>,
        (const void *)k_pred<CVP9_ARITH_REFCPU, kPredMinB, true>,
        (const void *)k_resid<CVP9_ARITH_SPEC, kResidMinB, false>,
        (const void *)k_resid<CVP9_ARITH_REFCPU, kResidMinB, true>,
        (const void *)k_resid<CVP9_ARITH_REFCPU, kResidMinB, false>,
        (const void *)k_resid<CVP9_ARITH_REFCPU, kResid8MinB, true, 1>,
        (const void *)k_resid<CVP9_ARITH_REFCPU, kResidMinB, true, 2>,
        (const void *)k_lf_full<uint8_t, 0>, (const void *)k_nv12_pack,
        (const void *)k_loopfilter<CVP9_ARITH_SPEC, 32>, (const void *)k_loopfilter<CVP9_ARITH_REFCPU, 32>,
        (const void *)k_loopfilter<CVP9_ARITH_SPEC, 64>, (const void *)k_loopfilter<CVP9_ARITH_REFCPU, 64>,
        (const void *)k_lf_strip<CVP9_ARITH_SPEC>, (const void *)k_lf_strip<CVP9_ARITH_REFCPU>,
        (const void *)k_lf_flat_h, (const void *)k_lf_flat_v,
        (const void *)k_gather_luma, (const void *)k_scatter_coeffs, (const void *)k_unpack_coeffs,
        (const void *)k_collect, (const void *)k_hbd_recon, (const void *)k_lf_full<uint16_t, 2>,
    };
    for (size_t i = 0; i < sizeof(fns) / sizeof(fns[0]); i++) {
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, fns[i]) != cudaSuccess) return -1;
    }
    return 0;
}

int cvp9k_hbd_ctas_per_sm(void)
{
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_hbd_recon, kHbdThreads, sizeof(HbdSmem)) == cudaSuccess
        ? n : -1;
}

int cvp9k_lf_full_ctas_per_sm(void)
{
    int n = 0;
    /* the 10-bit kernel's, which holds more shared memory */
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_lf_full<uint16_t, 2>, kLfThreads,
                                                         sizeof(LfSmem<uint16_t>)) == cudaSuccess ? n : -1;
}

int cvp9k_recon_ctas_per_sm(int arith)
{
    int n = 0;
    auto *kr = arith == CVP9_ARITH_FULL ? k_recon<CVP9_ARITH_FULL>
                                        : arith == CVP9_ARITH_SPEC ? k_recon<CVP9_ARITH_SPEC> : k_recon<CVP9_ARITH_REFCPU>;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kr, kThreads, sizeof(ReconSmem)) == cudaSuccess ? n : -1;
}

/* Timing events become event-record nodes when the stream is being captured. */
static cudaError_t mark(cudaEvent_t ev, cudaStream_t st, bool capturing)
{
    if (!ev) return cudaSuccess;
    return capturing ? cudaEventRecordWithFlags(ev, st, cudaEventRecordExternal) : cudaEventRecord(ev, st);
}

int cvp9k_launch_frame(const cvp9k_launch_t *L, cudaStream_t st)
{
    if (!L || L->njobs <= 0) return (int)cudaErrorInvalidValue;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(st, &cap);
    if (e != cudaSuccess) return (int)e;
    const bool capturing = cap == cudaStreamCaptureStatusActive;
    /* no timing events in between, the regular chain: kernel after kernel
     * (a 352x288 picture of the allocation-free entry point 35 -> 27 us) */
    const bool early = !capturing && !L->ev[0] && !L->ev[1] && !L->ev[2] && !L->full && !L->hbd && !L->general;
    if ((e = mark(L->ev[0], st, capturing)) != cudaSuccess) return (int)e;
    if (L->hbd) {
        /* profile 2: scan, mode-info map, k_hbd_recon, the 10-bit VP9 filter */
        if (L->max_blocks > 0) {
            dim3 g((unsigned)((L->max_blocks + 255) / 256), (unsigned)L->njobs);
            k_scan_blocks<<<g, 256, 0, st>>>(L->jobs);
            k_lf_mimap<<<g, 256, 0, st>>>(L->jobs);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
        if ((e = mark(L->ev[1], st, capturing)) != cudaSuccess) return (int)e;
        if (L->n_tickets > 0) {
            int grid = L->recon_ctas > 0 ? L->recon_ctas : (int)L->n_tickets;
            if (grid > (int)L->n_tickets) grid = (int)L->n_tickets;
            k_hbd_recon<<<grid, kHbdThreads, sizeof(HbdSmem), st>>>(L->jobs, L->tickets, L->n_tickets,
                                                                    L->ticket_counter);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
        if ((e = mark(L->ev[2], st, capturing)) != cudaSuccess) return (int)e;
        if (L->lf_tickets > 0 && L->lf_counter) {
            const int grid = L->lf_ctas > 0 && L->lf_ctas < (int)L->lf_tickets ? L->lf_ctas : (int)L->lf_tickets;
            k_lf_full<uint16_t, 2><<<grid, kLfThreads, sizeof(LfSmem<uint16_t>), st>>>(L->jobs, L->njobs, L->lf_tickets, L->lf_counter);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
        return (int)mark(L->ev[3], st, capturing);
    }
    if (L->max_blocks > 0 || L->scan_ctas > 0) {
        int gx = L->scan_ctas > 0 ? L->scan_ctas : (L->max_blocks + 255) / 256;
        dim3 g((unsigned)gx, (unsigned)L->njobs);
        if ((e = launch(early, k_scan_blocks, g, 256, 0, st, L->jobs)) != cudaSuccess) return (int)e;
        if (L->full) k_lf_mimap<<<g, 256, 0, st>>>(L->jobs);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
    if ((e = mark(L->ev[1], st, capturing)) != cudaSuccess) return (int)e;
    if (L->n_tickets > 0) {
        int grid = L->recon_ctas > 0 ? L->recon_ctas : (int)L->n_tickets;
        if (grid > (int)L->n_tickets) grid = (int)L->n_tickets;
        size_t smem = sizeof(ReconSmem);
        const bool fast = L->general && L->general_tickets && L->n_general;
        if (fast) {
            const unsigned fg = (L->n_tickets + kFastWarps - 1) / kFastWarps;
            /* the count of general superblocks that k_inter raises */
            if ((e = cudaMemsetAsync(L->n_general + 1, 0, 4, st)) != cudaSuccess) return (int)e;
            const size_t fs = kFastWarps * sizeof(FastSmem);
            const bool spec = L->arith == CVP9_ARITH_SPEC;
            if (L->inter_variant >= 3 && spec) {       /* SPEC has one split (3; 4 and 5 are REFCPU forms) */
                k_pred<CVP9_ARITH_SPEC, kPredMinB><<<fg, kFastWarps * 32, kFastWarps * sizeof(PredSmem), st>>>(
                    L->jobs, L->tickets, L->n_tickets, L->general);
                k_resid<CVP9_ARITH_SPEC, kResidMinB, false><<<fg, kFastWarps * 32, kFastWarps * sizeof(ResidSmem), st>>>(
                    L->jobs, L->tickets, L->n_tickets, L->general);
            } else if (L->inter_variant == 5) {
                /* REFCPU: k_pred marks superblocks with TXs other than 8x8;
                 * the 8x8-only residual kernel carries no larger transform */
                k_pred<CVP9_ARITH_REFCPU, kPredMinB, true><<<fg, kFastWarps * 32, kFastWarps * sizeof(PredSmem), st>>>(
                    L->jobs, L->tickets, L->n_tickets, L->general);
                k_resid<CVP9_ARITH_REFCPU, kResid8MinB, true, 1>
                    <<<fg, kFastWarps * 32, kFastWarps * sizeof(ResidSmem), st>>>(L->jobs, L->tickets, L->n_tickets,
                                                                               L->general);
                k_resid<CVP9_ARITH_REFCPU, kResidMinB, true, 2>
                    <<<fg, kFastWarps * 32, kFastWarps * sizeof(ResidSmem), st>>>(L->jobs, L->tickets, L->n_tickets,
                                                                               L->general);
            } else if (L->inter_variant == 3 || L->inter_variant == 4) {
                k_pred<CVP9_ARITH_REFCPU, kPredMinB><<<fg, kFastWarps * 32, kFastWarps * sizeof(PredSmem), st>>>(
                    L->jobs, L->tickets, L->n_tickets, L->general);
                if (L->inter_variant == 4)
                    k_resid<CVP9_ARITH_REFCPU, kResidMinB, true><<<fg, kFastWarps * 32, kFastWarps * sizeof(ResidSmem), st>>>(
                        L->jobs, L->tickets, L->n_tickets, L->general);
                else
                    k_resid<CVP9_ARITH_REFCPU, kResidMinB, false><<<fg, kFastWarps * 32, kFastWarps * sizeof(ResidSmem), st>>>(
                        L->jobs, L->tickets, L->n_tickets, L->general);
            } else if (L->inter_variant == 2) {
                if (spec) k_inter<CVP9_ARITH_SPEC, 6><<<fg, kFastWarps * 32, fs, st>>>(L->jobs, L->tickets, L->n_tickets, L->general);
                else k_inter<CVP9_ARITH_REFCPU, 6><<<fg, kFastWarps * 32, fs, st>>>(L->jobs, L->tickets, L->n_tickets, L->general);
            } else {
                if (spec) k_inter<CVP9_ARITH_SPEC, 5><<<fg, kFastWarps * 32, fs, st>>>(L->jobs, L->tickets, L->n_tickets, L->general);
                else k_inter<CVP9_ARITH_REFCPU, 5><<<fg, kFastWarps * 32, fs, st>>>(L->jobs, L->tickets, L->n_tickets, L->general);
            }
            k_compact<<<1, 1024, 0, st>>>(L->tickets, L->general, L->n_tickets, L->general_tickets, L->n_general);
        }
        auto *kr = L->full ? k_recon<CVP9_ARITH_FULL>
                           : L->arith == CVP9_ARITH_SPEC ? k_recon<CVP9_ARITH_SPEC> : k_recon<CVP9_ARITH_REFCPU>;
        if ((e = launch(early, kr, dim3((unsigned)grid), kThreads, smem, st, L->jobs,
                        fast ? L->general_tickets : L->tickets, L->n_tickets, L->ticket_counter,
                        fast ? L->n_general : (uint32_t *)nullptr)) != cudaSuccess)
            return (int)e;
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
    if ((e = mark(L->ev[2], st, capturing)) != cudaSuccess) return (int)e;
    if (L->full) {
        if (L->lf_tickets > 0 && L->lf_counter) {
            const int grid = L->lf_ctas > 0 && L->lf_ctas < (int)L->lf_tickets ? L->lf_ctas : (int)L->lf_tickets;
            k_lf_full<uint8_t, 0><<<grid, kLfThreads, sizeof(LfSmem<uint8_t>), st>>>(L->jobs, L->njobs, L->lf_tickets, L->lf_counter);
        }
        if (L->full_nv12_max_px > 0) {
            long long n = L->full_nv12_max_px;
            k_nv12_pack<<<dim3((unsigned)((n + 255) / 256), (unsigned)L->njobs), 256, 0, st>>>(L->jobs);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
        return (int)mark(L->ev[3], st, capturing);
    }
    if (L->lf_tiles_x > 0 && L->lf_tiles_y > 0) {
        /* lf_tiles_y counts 64-row tiles; 32-row tiles need twice as many
         * (one more covers the 4-row shift) */
        if (L->lf_tile_h == 32) {
            dim3 g((unsigned)L->lf_tiles_x, (unsigned)(2 * L->lf_tiles_y), (unsigned)L->njobs);
            if ((e = launch(early, L->arith == CVP9_ARITH_SPEC ? k_loopfilter<CVP9_ARITH_SPEC, 32> : k_loopfilter<CVP9_ARITH_REFCPU, 32>,
                            g, 256, 0, st, L->jobs)) != cudaSuccess)
                return (int)e;
        } else {
            dim3 g((unsigned)L->lf_tiles_x, (unsigned)L->lf_tiles_y, (unsigned)L->njobs);
            if ((e = launch(early, L->arith == CVP9_ARITH_SPEC ? k_loopfilter<CVP9_ARITH_SPEC, 64> : k_loopfilter<CVP9_ARITH_REFCPU, 64>,
                            g, 256, 0, st, L->jobs)) != cudaSuccess)
                return (int)e;
        }
    }
    if (L->lf_strips_x > 0 && L->lf_strips_y > 0) {
        dim3 g((unsigned)L->lf_strips_x, (unsigned)L->lf_strips_y, (unsigned)L->njobs);
        if (L->arith == CVP9_ARITH_SPEC) k_lf_strip<CVP9_ARITH_SPEC><<<g, 128, 0, st>>>(L->jobs);
        else k_lf_strip<CVP9_ARITH_REFCPU><<<g, 128, 0, st>>>(L->jobs);
    }
    if (L->flat_lf_max_w > 0) {
        long long nh = (long long)((L->flat_lf_max_h + 7) / 8) * L->flat_lf_max_w;
        long long nv = (long long)((L->flat_lf_max_w + 7) / 8) * L->flat_lf_max_h;
        int refcpu = L->arith == CVP9_ARITH_REFCPU;
        k_lf_flat_h<<<dim3((unsigned)((nh + 255) / 256), (unsigned)L->njobs), 256, 0, st>>>(L->jobs, refcpu);
        k_lf_flat_v<<<dim3((unsigned)((nv + 255) / 256), (unsigned)L->njobs), 256, 0, st>>>(L->jobs, refcpu);
        if (L->flat_nv12) {
            long long n = (long long)L->flat_lf_max_w * L->flat_lf_max_h;
            k_nv12_pack<<<dim3((unsigned)((n + 255) / 256), (unsigned)L->njobs), 256, 0, st>>>(L->jobs);
        }
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
    return (int)mark(L->ev[3], st, capturing);
}

} /* extern "C" */
