// Products with a sparse matrix by row tiles: a tile is R rows, the list of their distinct
// columns, and their entries as values and 16-bit local column ids.  A block owns a tile: it
// gathers the x entries of the tile's columns into shared memory by asynchronous copies, one
// each, while the first entries are on their way to registers, and then streams the entries
// against shared memory.  Included by solve.cu after the mbarrier helpers.
//
// The SELL-32 and CSR kernels wait for a column id and then for a 16-byte x value from L2 at
// every entry; the finest displacement level (28 entries a row, 4-wide vectors) was bound by
// that latency at half of the HBM bandwidth and its x traffic was four times the matrix.  Here a
// gathered x entry serves five or six matrix entries, these cost six (FP32) or ten (FP64) bytes,
// and no load waits for another one but column list -> x.  Lane layout: LPR = 256 / R lanes per
// row, entries in pairs (lane s of a row holds entries 2 (q LPR + s) and the next one at step q),
// rows of a tile by decreasing length.  (Bringing the entries to shared memory by bulk copies
// with two buffers a block measured 86 us at 48^3 against 70 for SELL-32: the three blocks that
// fit on an SM did not overlap their copies with their work.)
#pragma once

struct TileArgs {
    int64_t n;
    const int32_t* __restrict__ row;     // nt * R, -1 past the end; null: the vectors are in tile order
    const int32_t* __restrict__ col;     // nt * mc, padded with the tile's first column
    const int64_t* __restrict__ eoff;    // nt + 1, entries
    const uint16_t* __restrict__ steps;  // nt * 8
    const uint16_t* __restrict__ lc;
    const int32_t* __restrict__ skl;
    int mc;
};

template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES)
                     : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// x entries in shared memory, NV values each as in global memory
template <typename T, int NV>
struct TileX;
template <>
struct TileX<float, 4> {
    static __device__ __forceinline__ void copy(float* s, const float* x) { cp_async<16>(s, x); }
    static __device__ __forceinline__ void get(const float* s, int i, float* v) {
        const float4 q = reinterpret_cast<const float4*>(s)[i];
        v[0] = q.x;
        v[1] = q.y;
        v[2] = q.z;
    }
};
template <>
struct TileX<double, 4> {
    static __device__ __forceinline__ void copy(double* s, const double* x) {
        cp_async<16>(s, x);
        cp_async<8>(s + 2, x + 2);
    }
    static __device__ __forceinline__ void get(const double* s, int i, double* v) {
        const double2 q = reinterpret_cast<const double2*>(s)[2 * i];
        v[0] = q.x;
        v[1] = q.y;
        v[2] = s[4 * i + 2];
    }
};
template <typename T>
struct TileX<T, 1> {
    static __device__ __forceinline__ void copy(T* s, const T* x) { cp_async<sizeof(T)>(s, x); }
    static __device__ __forceinline__ void get(const T* s, int i, T* v) { v[0] = s[i]; }
};

template <typename T>
struct Pair;
template <>
struct Pair<float> {
    typedef float2 type;
};
template <>
struct Pair<double> {
    typedef double2 type;
};

template <typename T, int NV, int LPR, class Epi>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 4 : 5) k_spmv_tile(TileArgs A, const T* __restrict__ va,
                                                                          const T* x, Epi epi,
                                                                          const double* skip) {
    constexpr int RW = 32 / LPR, R = 256 / LPR, NC = ncomp<NV>(), PF = 4, CQ = TILE_MAX_COLS / 256;
    extern __shared__ __align__(128) unsigned char smem[];
    typedef typename Pair<T>::type P2;
    T* sx = reinterpret_cast<T*>(smem);
    const int64_t t = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, sub = lane % LPR;
    int cid[CQ];
#pragma unroll
    for (int q = 0; q < CQ; ++q)
        if (tid + q * 256 < A.mc) cid[q] = __ldg(A.col + t * A.mc + tid + q * 256);
    int64_t row = t * R + w * RW + lane / LPR;
    row = A.row ? __ldg(A.row + row) : (row < A.n ? row : -1);
    const int64_t e0 = __ldg(A.eoff + t);
    const uint4 s4 = __ldg(reinterpret_cast<const uint4*>(A.steps) + t);
    // steps of this warp and of those before it
    int base = 0, steps = 0;
    {
        const uint32_t s2[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int s = (int)((s2[q >> 1] >> (16 * (q & 1))) & 0xffffu);
            base += q < w ? s : 0;
            steps = q == w ? s : steps;
        }
    }
    const P2* pv = reinterpret_cast<const P2*>(va + e0) + base * 32 + lane;
    const uint32_t* pc = reinterpret_cast<const uint32_t*>(A.lc + e0) + base * 32 + lane;
    P2 a[PF];
    uint32_t cc[PF];
#pragma unroll
    for (int u = 0; u < PF; ++u)
        if (u < steps) {
            a[u] = __ldcs(pv + u * 32);
            cc[u] = __ldcs(pc + u * 32);
        }
    // (so far nothing that an earlier kernel writes)
    pdl_wait();
    if (skip && slice_frozen(A.skl, t, skip)) return;  // (the whole block)
#pragma unroll
    for (int q = 0; q < CQ; ++q) {
        const int i = tid + q * 256;
        if (i < A.mc) TileX<T, NV>::copy(sx + NV * i, x + NV * (int64_t)cid[q]);
    }
    cp_async_commit();
    const bool own = row >= 0 && sub == 0;
    typename Epi::Pre pre{};
    if (own) pre = epi.pre(row);
    cp_async_wait<0>();
    __syncthreads();
    T acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = T(0);
    for (int q = 0; q < steps; q += PF) {
        P2 an[PF];
        uint32_t cn[PF];
#pragma unroll
        for (int u = 0; u < PF; ++u)
            if (q + PF + u < steps) {
                an[u] = __ldcs(pv + (q + PF + u) * 32);
                cn[u] = __ldcs(pc + (q + PF + u) * 32);
            }
#pragma unroll
        for (int u = 0; u < PF; ++u)
            if (q + u < steps) {
                T x0[NV], x1[NV];
                TileX<T, NV>::get(sx, (int)(cc[u] & 0xffffu), x0);
                TileX<T, NV>::get(sx, (int)(cc[u] >> 16), x1);
#pragma unroll
                for (int k = 0; k < NC; ++k) acc[k] += a[u].x * x0[k];
#pragma unroll
                for (int k = 0; k < NC; ++k) acc[k] += a[u].y * x1[k];
            }
#pragma unroll
        for (int u = 0; u < PF; ++u) {
            a[u] = an[u];
            cc[u] = cn[u];
        }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NC; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    pdl_trigger();
    double r0 = 0.0, r1 = 0.0;
    if (own) epi.apply(row, acc, pre, r0, r1);
}

template <typename T, int NV, int LPR, class Epi>
static void launch_tile_l(mpet_ctx* c, const RowTiles& r, int64_t n, const T* x, const Epi& epi) {
    const size_t sm = (size_t)r.mc * NV * sizeof(T);
    auto kern = k_spmv_tile<T, NV, LPR, Epi>;
    if (sm > 48 * 1024) MPET_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM));
    const TileArgs A{n, r.perm ? nullptr : r.row, r.col, r.eoff, r.steps, r.lc, r.skl, r.mc};
    launch_k(c, kern, r.nt, 256, sm, A, (const T*)r.v, x, epi, r.skl ? c->skip_done : (const double*)nullptr);
    MPET_CHECK_LAUNCH();
    c->n_launch++;
}

template <typename T, int NV, class Epi>
static void launch_tile(mpet_ctx* c, const RowTiles& r, int64_t n, const T* x, const Epi& epi) {
    switch (r.R) {
        case 256: launch_tile_l<T, NV, 1, Epi>(c, r, n, x, epi); return;
        case 128: launch_tile_l<T, NV, 2, Epi>(c, r, n, x, epi); return;
        case 64: launch_tile_l<T, NV, 4, Epi>(c, r, n, x, epi); return;
        default: launch_tile_l<T, NV, 8, Epi>(c, r, n, x, epi); return;
    }
}
