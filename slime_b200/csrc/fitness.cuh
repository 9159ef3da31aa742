// Fitness reduction: per (grid, head) 64x64 Gram of the redistributed value V', its eigenvalues, exp-entropy rank, Pearson coherence between the last two steps, fitness = rank x coherence.
// Replaces gpu_svd_kernel / effective_rank_kernel / coherence_kernel / fitness_fused_kernel
// (slime/kernels/warp_ca.cu:66-226).  Gram and eigenvalues run in fp64: the small eigenvalues carry most of the
// entropy's sensitivity, and an fp32 Gram loses them.
#pragma once
#include "ca_aux.cuh"
#include "ca_bf16.cuh"
#include "common.cuh"

namespace slime {

constexpr int GRAM_CHUNK = 2048;   // cells per Gram partial, at most; populations too small to fill the GPU take less

// gram_part[((b*8+h)*splits + split)][64][64] (fp64) over cells [split*chunk, ...) of plane (b,h).
// The Gram matrix is symmetric: only the 136 4x4 blocks on or above the diagonal are accumulated (one thread
// each, 160 threads per block) and each is written to both places.  A chunk of 64 cells is converted to fp64
// once, on its way into shared memory (the conversion is the slow instruction here: converting at the point of
// use cost one conversion per two multiply-adds and made them the bottleneck).  Each 4-value block of a cell is
// kept as two 16-byte halves in two planes, so a warp's loads of consecutive blocks are consecutive 16-byte
// words: no bank conflicts.
constexpr int GRAM_THREADS = 160;
template <typename T>
__global__ void __launch_bounds__(GRAM_THREADS, 6)
k_gram(const T* __restrict__ vp, int cells, int chunk, double* __restrict__ gram_part) {
    __shared__ __align__(16) double2 flo[64][16];      // values 4 blk + 0, 4 blk + 1 of cell s
    __shared__ __align__(16) double2 fhi[64][16];      // values 4 blk + 2, 4 blk + 3
    const int split = blockIdx.x, h = blockIdx.y, b = blockIdx.z, splits = gridDim.x;
    const T* plane = vp + ((size_t)b * NH + h) * (size_t)cells * HD;
    // thread t -> block (bi, bj), bi <= bj, rows of the upper triangle laid end to end: row bi starts at
    // bi * 16 - bi * (bi - 1) / 2
    int bi = 0, rest = threadIdx.x;
    const bool live = threadIdx.x < 136;
    if (live) { while (rest >= 16 - bi) { rest -= 16 - bi; ++bi; } } else rest = 0;
    const int bj = bi + rest, ti = bi * 4, tj = bj * 4;
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    const int lo = split * chunk;
    const int hi = min(lo + chunk, cells);
    for (int s0 = lo; s0 < hi; s0 += 64) {
        __syncthreads();
        for (int i = threadIdx.x; i < 64 * 32; i += GRAM_THREADS) {       // one pair of adjacent values per step
            const int sl = i >> 5, pr = i & 31, s = s0 + sl;
            double2 v = make_double2(0.0, 0.0);
            if (s < hi) {
                v.x = (double)to_f32<T>(plane[(size_t)s * HD + 2 * pr]);
                v.y = (double)to_f32<T>(plane[(size_t)s * HD + 2 * pr + 1]);
            }
            if (pr & 1) fhi[sl][pr >> 1] = v; else flo[sl][pr >> 1] = v;
        }
        __syncthreads();
        if (live) {
#pragma unroll 8
            for (int s = 0; s < 64; ++s) {
                const double2 a0 = flo[s][bi], a1 = fhi[s][bi], c0 = flo[s][bj], c1 = fhi[s][bj];
                const double av[4] = {a0.x, a0.y, a1.x, a1.y};
                const double cv[4] = {c0.x, c0.y, c1.x, c1.y};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fma(av[i], cv[j], acc[i][j]);
            }
        }
    }
    if (!live) return;
    double* out = gram_part + (((size_t)b * NH + h) * splits + split) * (HD * HD);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            out[(ti + i) * HD + tj + j] = acc[i][j];
            if (ti != tj) out[(tj + j) * HD + ti + i] = acc[i][j];
        }
}

// The same Gram partials for bf16 planes on the tensor cores.  One CTA per (grid, head) plane (several where there are few planes) walks its chunks in tiles
// of 128 cells; a tile [128 cells][64 dims] lands in shared memory by TMA with the 128-byte swizzle, which is exactly
// the MN-major operand layout of tcgen05 (one 128-byte row of the 64 dims per cell), so the one tile is both operands of
// D[64 x 64] += F^T F: eight tcgen05.mma of M = 64, N = 64, K = 16 cells, fp32 accumulation in 64 TMEM columns (the
// products of bf16 values are exact in fp32).  After every chunk of cells the accumulator is written out as one fp64
// partial - the same [plane][split][64][64] layout the SIMT kernel fills - and cleared by the next chunk's first
// instruction, so chunks are still summed in fp64 by k_gram_rank.  An M = 64 accumulator keeps row r in TMEM lane
// 32 * (r / 16) + r % 16: warp w's first sixteen lanes hold rows 16 w .. 16 w + 15.
namespace gtc {
constexpr int TILE = 128, STAGES = 4, TILE_BYTES = TILE * 128;
constexpr int BARS = STAGES * TILE_BYTES, TMEM_PTR = BARS + (2 * STAGES + 2) * 8, BYTES = TMEM_PTR + 16, SMEM = BYTES + 1024;
constexpr uint32_t IDESC = ptx::umma_idesc_bf16(64, 64) | (1u << 15) | (1u << 16);     // both operands MN-major
}  // namespace gtc
__global__ void __launch_bounds__(128)
k_gram_tc(const __grid_constant__ CUtensorMap map_vp, int cells, int chunk, int splits, double* __restrict__ gram_part,
          int* __restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = align1024(smem_raw);
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + gtc::BARS);     // [4] tile landed            (waits: UMMA issuer)
    uint64_t* empty = full + gtc::STAGES;                             // [4] its UMMAs are done     (waits: TMA producer)
    uint64_t* acc_full = empty + gtc::STAGES;                         //     chunk accumulated      (waits: all)
    uint64_t* acc_empty = acc_full + 1;                               //     chunk written out      (waits: UMMA issuer)
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(sm + gtc::TMEM_PTR);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, plane = blockIdx.x;
    if (tid == 0) {
        for (int i = 0; i < gtc::STAGES; ++i) { ptx::mbar_init(&full[i], 1); ptx::mbar_init(&empty[i], 1); }
        ptx::mbar_init(acc_full, 1);
        ptx::mbar_init(acc_empty, 128);
        ptx::fence_barrier_init();
        ptx::prefetch_tmap(&map_vp);
    }
    if (warp == 0) ptx::tmem_alloc(tmem_ptr, 64);
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = *tmem_ptr;
    uint32_t it = 0;       // tiles so far (the producer and the issuer count the same way)
    const int split0 = (int)((long long)splits * blockIdx.y / gridDim.y), split1 = (int)((long long)splits * (blockIdx.y + 1) / gridDim.y);
    for (int split = split0; split < split1; ++split) {
        const int lo = split * chunk, hi = min(lo + chunk, cells), u = split - split0;
        const int n_tiles = (hi - lo + gtc::TILE - 1) / gtc::TILE;
        if (warp == 0 && lane == 0) {
            for (int t = 0; t < n_tiles; ++t) {
                const uint32_t i = it + t, s = i % gtc::STAGES;
                ptx::mbar_wait(&empty[s], ((i / gtc::STAGES) & 1) ^ 1, status, 410);
                ptx::mbar_expect_tx(&full[s], gtc::TILE_BYTES);
                // cells past the end of the plane read as zero and add nothing (the last chunk ends at the plane's end:
                // a tile never reaches into the next chunk)
                ptx::tma_load_3d(sm + s * gtc::TILE_BYTES, &map_vp, 0, lo + t * gtc::TILE, plane, &full[s]);
            }
        } else if (warp == 1 && lane == 0) {
            ptx::mbar_wait(acc_empty, (u & 1) ^ 1, status, 411);
            ptx::tc_fence_after();
            for (int t = 0; t < n_tiles; ++t) {
                const uint32_t i = it + t, s = i % gtc::STAGES;
                ptx::mbar_wait(&full[s], (i / gtc::STAGES) & 1, status, 412);
                ptx::tc_fence_after();
                const uint64_t d = ptx::umma_desc_sw128(ptx::smem_u32(sm + s * gtc::TILE_BYTES));
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)      // 16 cells per step: 2048 bytes = 128 sixteen-byte units further
                    ptx::umma_bf16(tmem, d + 128 * ks, d + 128 * ks, gtc::IDESC, t > 0 || ks > 0);
                ptx::umma_commit(&empty[s]);
            }
            ptx::umma_commit(acc_full);
        }
        it += n_tiles;
        __syncwarp();
        ptx::mbar_wait(acc_full, u & 1, status, 413);
        ptx::tc_fence_after();
        double* out = gram_part + ((size_t)plane * splits + split) * (HD * HD) + (size_t)(warp * 16 + (lane & 15)) * HD;
#pragma unroll
        for (int c = 0; c < HD; c += 16) {
            uint32_t r[16];
            ptx::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + c, r);
            ptx::tmem_ld_wait();
            if (lane < 16) {
#pragma unroll
                for (int k = 0; k < 16; k += 2)
                    *reinterpret_cast<double2*>(out + c + k) = make_double2((double)__uint_as_float(r[k]), (double)__uint_as_float(r[k + 1]));
            }
        }
        ptx::tc_fence_before();
        ptx::mbar_arrive(acc_empty);
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 0) ptx::tmem_dealloc(tmem, 64);
}

// Tensor map over a V' buffer [planes][cells][64] bf16 for k_gram_tc: box 64 dims x 128 cells x 1 plane, 128B swizzle.
inline int gram_tc_map(CUtensorMap* map, const void* vp, int planes, int cells) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn ||
        q != cudaDriverEntryPointSuccess)
        return -1;
    const cuuint64_t dims[3] = {64, (cuuint64_t)cells, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {128, (cuuint64_t)cells * 128};
    const cuuint32_t box[3] = {64, gtc::TILE, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = reinterpret_cast<EncodeTiledFn>(fn)(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(vp), dims,
                                                         strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -1;
    return cudaFuncSetAttribute(k_gram_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, gtc::SMEM) == cudaSuccess ? 0 : -1;
}

// One 256-thread block per (grid, head): the eigenvalues of the summed Gram matrix and the exp-entropy rank
// p = l/(sum l + 1e-7), rank = exp(-sum p ln(p + 1e-7))  (slime/kernels/warp_ca.cu:107-144).
//
// Householder reduction to tridiagonal form (Golub & Van Loan, Matrix Computations, 8.3.1), then every eigenvalue by
// multisection on Sturm counts (Wilkinson, The Algebraic Eigenvalue Problem, 5.37-5.39), all in fp64: absolute errors of a
// few 1e-15 of the trace from the first and 2e-14 from the second, where the entropy's sensitivity asks for 1e-9.
// It replaces a cyclic Jacobi iteration of 7 sweeps x 63 rounds, whose 440 rounds of three barriers took 610 us however
// few matrices there were, and 2.36 ms for 1024 of them; here 62 steps of two barriers and 18 of one.
//   The matrix lives in registers, row r = lane + 32 (warp & 1) and 16 columns per thread, so a step's matrix-vector
// product and rank-2 update touch shared memory only for the vectors, which every warp keeps a copy of.
constexpr int RANK_THREADS = 256;
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__global__ void __launch_bounds__(RANK_THREADS)
k_gram_rank(const double* __restrict__ gram_part, int splits, float* __restrict__ head_rank) {
    __shared__ __align__(16) double xrow[2][HD];          // row of the matrix that the next step eliminates
    __shared__ __align__(16) double vv[8][HD], ww[8][HD]; // per warp: the step's v and w
    __shared__ double part[4][HD];
    __shared__ __align__(16) double2 tri[HD];             // {d[i], e[i-1]^2} of the tridiagonal matrix over its trace
    __shared__ double dd[HD], ee[HD];
    __shared__ int cnt[RANK_THREADS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = lane + 32 * (warp & 1), c0 = (warp >> 1) * 16;
    double a[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) a[j] = 0.0;
    {
        // the matrix is symmetric: this thread's 16 values are read down a column, coalesced over the lanes
        const double* src = gram_part + (size_t)blockIdx.x * splits * (HD * HD) + c0 * HD + r;
        for (int k = 0; k < splits; ++k, src += HD * HD)
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] += __ldcs(src + j * HD);
    }
    if (r == 0) {
#pragma unroll
        for (int j = 0; j < 16; ++j) xrow[0][c0 + j] = a[j];
    }
    __syncthreads();
    double* v = vv[warp];
    double* w = ww[warp];
    for (int k = 0; k < HD - 2; ++k) {
        const double* x = xrow[k & 1];
        double x0 = lane > k ? x[lane] : 0.0, x1 = lane + 32 > k ? x[lane + 32] : 0.0;
        const double head = x[k + 1], diag = x[k];
        const double tail = warp_sum((lane == k + 1 ? 0.0 : x0 * x0) + (lane + 32 == k + 1 ? 0.0 : x1 * x1));
        double alpha = head, beta = 0.0;                   // tail = 0: nothing to eliminate
        if (tail != 0.0) {
            const double norm2 = fma(head, head, tail);
            alpha = head > 0.0 ? -sqrt(norm2) : sqrt(norm2);
            beta = 1.0 / fma(-head, alpha, norm2);
        }
        if (tid == 0) { dd[k] = diag; ee[k] = alpha; }
        if (lane == k + 1) x0 -= alpha;
        if (lane + 32 == k + 1) x1 -= alpha;
        if (tail == 0.0) x0 = x1 = 0.0;
        v[lane] = x0; v[lane + 32] = x1;
        __syncwarp();
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
            const double2 vc = *reinterpret_cast<const double2*>(v + c0 + j);
            s0 = fma(a[j], vc.x, s0);
            s1 = fma(a[j + 1], vc.y, s1);
        }
        part[warp >> 1][r] = s0 + s1;
        __syncthreads();
        const double p0 = beta * ((part[0][lane] + part[1][lane]) + (part[2][lane] + part[3][lane]));
        const double p1 = beta * ((part[0][lane + 32] + part[1][lane + 32]) + (part[2][lane + 32] + part[3][lane + 32]));
        const double half = 0.5 * beta * warp_sum(fma(p0, x0, p1 * x1));
        w[lane] = fma(-half, x0, p0); w[lane + 32] = fma(-half, x1, p1);
        __syncwarp();
        const double vr = v[r], wr = w[r];
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
            const double2 vc = *reinterpret_cast<const double2*>(v + c0 + j), wc = *reinterpret_cast<const double2*>(w + c0 + j);
            a[j] = fma(-vr, wc.x, fma(-wr, vc.x, a[j]));
            a[j + 1] = fma(-vr, wc.y, fma(-wr, vc.y, a[j + 1]));
        }
        if (r == k + 1) {
#pragma unroll
            for (int j = 0; j < 16; ++j) xrow[(k + 1) & 1][c0 + j] = a[j];
        }
        if (k == HD - 3 && r == HD - 1 && warp >> 1 == 3) dd[HD - 1] = a[15];
        __syncthreads();
    }
    if (tid == 0) { dd[HD - 2] = xrow[0][HD - 2]; ee[HD - 2] = xrow[0][HD - 1]; }
    __syncthreads();
    // over the trace: the eigenvalues of the (positive semidefinite) matrix then lie in [0, 1]
    const double trace = warp_sum(dd[lane] + dd[lane + 32]);
    const double inv = 1.0 / trace;
    if (tid < HD) {
        const double e = tid > 0 ? ee[tid - 1] * inv : 0.0;
        tri[tid] = make_double2(dd[tid] * inv, e * e);
    }
    __syncthreads();
    if (!(trace > 0.0) || !isfinite(trace) || !isfinite(inv)) {      // no spread to measure: one direction
        if (tid == 0) head_rank[blockIdx.x] = 1.f;
        return;
    }
    // Eigenvalues below x: sign changes of the leading minors p(i) = (d(i) - x) p(i-1) - e(i-1)^2 p(i-2).  The two last are
    // brought back to order 1 by a power of two every four steps; a minor that is exactly zero is taken as slightly of the
    // other sign (a perturbation of d(i) by 2^-60).
    auto below = [&](double x) {
        double p2 = 0.0, p1 = 1.0;
        int n = 0;
#pragma unroll 1
        for (int i = 0; i < HD; i += 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double2 t = tri[i + j];
                double p = fma(t.x - x, p1, -(t.y * p2));
                if (p == 0.0) p = p1 * -8.673617379884035e-19;
                n += (__double2hiint(p) ^ __double2hiint(p1)) < 0;
                p2 = p1; p1 = p;
            }
            const int e = max((__double2hiint(p1) >> 20) & 0x7ff, (__double2hiint(p2) >> 20) & 0x7ff);
            const double sc = __hiloint2double(min(max(2046 - e, 1), 2046) << 20, 0);
            p1 *= sc; p2 *= sc;
        }
        return n;
    };
    // all threads once, on a uniform grid: each eigenvalue within 1 / 256 ...
    const double step0 = 1.0 / RANK_THREADS;
    cnt[tid] = below((tid + 1) * step0);
    __syncthreads();
    // ... then four threads per eigenvalue, 16 rounds of five parts each (5^16 = 2^37)
    const int ev = tid >> 2, q = tid & 3;
    int lo_i = 0;                                          // first grid point with more than ev eigenvalues below it
#pragma unroll
    for (int b = RANK_THREADS / 2; b > 0; b >>= 1)
        if (cnt[lo_i + b - 1] <= ev) lo_i += b;
    double lo = lo_i * step0, width = step0;
    for (int round = 0; round < 16; ++round) {
        width *= 0.2;
        const bool above = below(fma(q + 1.0, width, lo)) <= ev;
        const unsigned m = (__ballot_sync(0xffffffffu, above) >> (lane & ~3)) & 15u;
        lo = fma((double)__popc(m), width, lo);
    }
    if (q == 0) dd[ev] = lo * trace;
    __syncthreads();
    if (tid >= 32) return;
    const double l0 = dd[lane], l1 = dd[lane + 32];
    const double sum = warp_sum(l0 + l1);
    const double e0 = l0 / (sum + 1e-7), e1 = l1 / (sum + 1e-7);
    const double ent = warp_sum(-(e0 * log(e0 + 1e-7) + e1 * log(e1 + 1e-7)));
    if (lane == 0) head_rank[blockIdx.x] = (float)exp(ent);
}

// Raw moments of (a, b) = (V' of step n-1, V' of step n) for one grid, fp64:
// part[(b*splits + split)][5] = {sum a, sum b, sum aa, sum bb, sum ab}.  Sixteen bytes per load (4 fp32 or 8 bf16
// values); per_grid is a multiple of 512.
template <typename T> struct PearsonVec;
template <> struct PearsonVec<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float* p, float (&f)[8]) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
    }
};
template <> struct PearsonVec<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&f)[8]) { unpack8(*reinterpret_cast<const uint4*>(p), f); }
};
template <typename T>
__global__ void __launch_bounds__(256)
k_pearson(const T* __restrict__ va, const T* __restrict__ vb, size_t per_grid, double* __restrict__ part) {
    __shared__ double red[5][256];
    constexpr int N = PearsonVec<T>::N;
    const int split = blockIdx.x, b = blockIdx.y, splits = gridDim.x;
    const size_t vecs = per_grid / N;
    const size_t chunk = (vecs + splits - 1) / splits;
    const size_t lo = (size_t)split * chunk;
    const size_t hi = lo + chunk < vecs ? lo + chunk : vecs;
    const T* a = va + (size_t)b * per_grid;
    const T* c = vb + (size_t)b * per_grid;
    double s[5] = {0, 0, 0, 0, 0};
    for (size_t i = lo + threadIdx.x; i < hi; i += 256) {
        float x[8], y[8];
        PearsonVec<T>::load(a + i * N, x);
        PearsonVec<T>::load(c + i * N, y);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const double xd = x[k], yd = y[k];
            s[0] += xd; s[1] += yd; s[2] = fma(xd, xd, s[2]); s[3] = fma(yd, yd, s[3]); s[4] = fma(xd, yd, s[4]);
        }
    }
    for (int k = 0; k < 5; ++k) red[k][threadIdx.x] = s[k];
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int k = 0; k < 5; ++k) red[k][threadIdx.x] += red[k][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 5) part[((size_t)b * splits + split) * 5 + threadIdx.x] = red[threadIdx.x][0];
}

// out[b] = {rank, coherence, fitness, hunger}: fitness = rank x coherence (slime/kernels/warp_ca.cu:219),
// hunger = 1 - coherence (slime/kernels/warp_ca.cu:238).  A warp per grid.
__global__ void __launch_bounds__(32)
k_fitness_final(const float* __restrict__ head_rank, const double* __restrict__ part, int splits, double n, float* __restrict__ out) {
    const int b = blockIdx.x, lane = threadIdx.x;
    double s[5] = {0, 0, 0, 0, 0};
    for (int k = lane; k < splits; k += 32)
#pragma unroll
        for (int j = 0; j < 5; ++j) s[j] += part[((size_t)b * splits + k) * 5 + j];
#pragma unroll
    for (int j = 0; j < 5; ++j) s[j] = warp_sum(s[j]);
    const double rk = warp_sum(lane < NH ? (double)head_rank[b * NH + lane] : 0.0) / NH;
    if (lane != 0) return;
    const double cov = s[4] - s[0] * s[1] / n;
    const double va = s[2] - s[0] * s[0] / n, vb = s[3] - s[1] * s[1] / n;
    const double coh = cov / sqrt(va * vb);
    out[b * 4 + 0] = (float)rk;
    out[b * 4 + 1] = (float)coh;
    out[b * 4 + 2] = (float)(rk * coh);
    out[b * 4 + 3] = (float)(1.0 - coh);
}

}  // namespace slime
