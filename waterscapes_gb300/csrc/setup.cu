// Dofmap, adjacency, CSR sparsity pattern and Dirichlet DOF lists, all
// built on the GPU once per mesh.
//
// The pattern follows DOLFIN's SparsityPatternBuilder as used by
// assemble(self.a) in src/mpet/mpet/mpetsolver.py:335: for every cell the
// dense block over all (30 + 4J) mixed DOFs is inserted, so a row of a P2
// node i holds every displacement DOF of every P2 node sharing a cell with
// i, followed by every pressure DOF of every vertex sharing a cell with i
// (network-major).  Columns are ascending because displacement DOFs come
// first and each list is sorted.
//
// Everything is derived from sorted 64-bit keys (radix sort + unique), which
// keeps the construction deterministic.
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>

#include "mpet_internal.cuh"

namespace mpet {

typedef unsigned long long u64;


static inline int grid_for(int64_t n, int threads) {
    int64_t g = (n + threads - 1) / threads;
    if (g > 2147483647LL) g = 2147483647LL;
    return (int)(g < 1 ? 1 : g);
}

__device__ __forceinline__ int64_t lower_bound_u64(const u64* a, int64_t n, u64 key) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (a[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ int lower_bound_i32(const int32_t* a, int n, int32_t key) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (a[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Sort keys in place (ping-pong through a temporary) and keep the unique
// ones; returns a freshly allocated exact-size array from the pool.
static int64_t sort_unique(mpet_ctx* c, u64* keys, int64_t n, int end_bit, u64** out_keys) {
    if (n > 2147483647LL) fail(MPET_ERR_INVALID, "too many adjacency keys for one radix sort");
    int ni = (int)n;
    TmpBuf sorted(sizeof(u64) * (size_t)n);
    size_t tb = 0;
    MPET_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tb, keys, sorted.as<u64>(), ni, 0, end_bit, c->stream));
    {
        TmpBuf tmp(tb);
        MPET_CUDA(cub::DeviceRadixSort::SortKeys(tmp.p, tb, keys, sorted.as<u64>(), ni, 0, end_bit, c->stream));
    }
    TmpBuf nsel(sizeof(int64_t));
    tb = 0;
    MPET_CUDA(cub::DeviceSelect::Unique(nullptr, tb, sorted.as<u64>(), keys, nsel.as<int64_t>(), ni, c->stream));
    {
        TmpBuf tmp(tb);
        MPET_CUDA(cub::DeviceSelect::Unique(tmp.p, tb, sorted.as<u64>(), keys, nsel.as<int64_t>(), ni, c->stream));
    }
    int64_t cnt = 0;
    MPET_CUDA(cudaMemcpyAsync(&cnt, nsel.p, sizeof(int64_t), cudaMemcpyDeviceToHost, c->stream));
    MPET_CUDA(cudaStreamSynchronize(c->stream));
    u64* o = c->pool.alloc<u64>(cnt);
    MPET_CUDA(cudaMemcpyAsync(o, keys, sizeof(u64) * cnt, cudaMemcpyDeviceToDevice, c->stream));
    *out_keys = o;
    return cnt;
}

static int bits_for(u64 maxval) {
    int b = 1;
    while (b < 64 && (maxval >> b) != 0) ++b;
    return b;
}

// --- kernels ------------------------------------------------------------------

template <int D>
__global__ void k_edge_keys(const int32_t* __restrict__ cells, int64_t nc, int64_t nv, u64* keys) {
    constexpr int NV = Simplex<D>::NV, NE = Simplex<D>::NE;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= nc * NE) return;
    int64_t c = idx / NE;
    int e = (int)(idx % NE);
    int64_t a = cells[NV * c + edge_end<D>(e, 0)];
    int64_t b = cells[NV * c + edge_end<D>(e, 1)];
    int64_t lo = a < b ? a : b, hi = a < b ? b : a;
    keys[idx] = (u64)(lo * nv + hi);
}

template <int D>
__global__ void k_cell_nodes(const int32_t* __restrict__ cells, int64_t nc, int64_t nv,
                             const u64* __restrict__ ekey, int64_t ne, int32_t* cell_nodes) {
    constexpr int NV = Simplex<D>::NV, NN = Simplex<D>::NN;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= nc * NN) return;
    int64_t c = idx / NN;
    int j = (int)(idx % NN);
    if (j < NV) {
        cell_nodes[idx] = cells[NV * c + j];
        return;
    }
    int e = j - NV;
    int64_t a = cells[NV * c + edge_end<D>(e, 0)];
    int64_t b = cells[NV * c + edge_end<D>(e, 1)];
    int64_t lo = a < b ? a : b, hi = a < b ? b : a;
    int64_t pos = lower_bound_u64(ekey, ne, (u64)(lo * nv + hi));
    cell_nodes[idx] = (int32_t)(nv + pos);
}

// Triangles: gradients of the barycentric coordinates (x, y in slots 3r, 3r+1
// of the 16-double record, z slot 0) and the area in slot 12.
__global__ void k_geometry2(const double* __restrict__ x, const int32_t* __restrict__ cells, int64_t nc,
                            double* geo) {
    int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= nc) return;
    double p[3][2];
    for (int i = 0; i < 3; ++i)
        for (int k = 0; k < 2; ++k) p[i][k] = x[3 * (int64_t)cells[3 * c + i] + k];
    const double e1[2] = {p[1][0] - p[0][0], p[1][1] - p[0][1]};
    const double e2[2] = {p[2][0] - p[0][0], p[2][1] - p[0][1]};
    const double det = e1[0] * e2[1] - e1[1] * e2[0];
    const double id = 1.0 / det;
    // rows of the inverse Jacobian: grad lambda_1 = ( e2y, -e2x)/det, grad lambda_2 = (-e1y, e1x)/det
    double* g = geo + 16 * c;
    for (int q = 0; q < 16; ++q) g[q] = 0.0;
    g[3] = e2[1] * id;
    g[4] = -e2[0] * id;
    g[6] = -e1[1] * id;
    g[7] = e1[0] * id;
    g[0] = -(g[3] + g[6]);
    g[1] = -(g[4] + g[7]);
    g[12] = fabs(det) / 2.0;
}

__global__ void k_geometry(const double* __restrict__ x, const int32_t* __restrict__ cells, int64_t nc,
                           double* geo) {
    int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= nc) return;
    double p[4][3];
    for (int i = 0; i < 4; ++i)
        for (int k = 0; k < 3; ++k) p[i][k] = x[3 * (int64_t)cells[4 * c + i] + k];
    double e1[3], e2[3], e3[3];
    for (int k = 0; k < 3; ++k) {
        e1[k] = p[1][k] - p[0][k];
        e2[k] = p[2][k] - p[0][k];
        e3[k] = p[3][k] - p[0][k];
    }
    double c23[3] = {e2[1] * e3[2] - e2[2] * e3[1], e2[2] * e3[0] - e2[0] * e3[2], e2[0] * e3[1] - e2[1] * e3[0]};
    double c31[3] = {e3[1] * e1[2] - e3[2] * e1[1], e3[2] * e1[0] - e3[0] * e1[2], e3[0] * e1[1] - e3[1] * e1[0]};
    double c12[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    double det = e1[0] * c23[0] + e1[1] * c23[1] + e1[2] * c23[2];
    double id = 1.0 / det;
    double* g = geo + 16 * c;
    for (int k = 0; k < 3; ++k) {
        double b1 = c23[k] * id, b2 = c31[k] * id, b3 = c12[k] * id;
        g[3 + k] = b1;
        g[6 + k] = b2;
        g[9 + k] = b3;
        g[k] = -(b1 + b2 + b3);
    }
    g[12] = fabs(det) / 6.0;
    g[13] = g[14] = g[15] = 0.0;
}

template <int D>
__global__ void k_pairs_n2(const int32_t* __restrict__ cn, int64_t nc, int64_t nnodes, u64* keys) {
    constexpr int NN = Simplex<D>::NN;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= nc * NN * NN) return;
    int64_t c = idx / (NN * NN);
    int r = (int)(idx % (NN * NN));
    int m = r / NN, j = r % NN;
    keys[idx] = (u64)cn[NN * c + m] * (u64)nnodes + (u64)cn[NN * c + j];
}

template <int D>
__global__ void k_pairs_n1(const int32_t* __restrict__ cn, const int32_t* __restrict__ cells, int64_t nc,
                           int64_t nv, u64* keys) {
    constexpr int NN = Simplex<D>::NN, NV = Simplex<D>::NV;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= nc * NN * NV) return;
    int64_t c = idx / (NN * NV);
    int r = (int)(idx % (NN * NV));
    int m = r / NV, w = r % NV;
    keys[idx] = (u64)cn[NN * c + m] * (u64)nv + (u64)cells[NV * c + w];
}

template <int D>
__global__ void k_pairs_inc(const int32_t* __restrict__ cn, int64_t nc, u64* keys) {
    constexpr int NN = Simplex<D>::NN;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= nc * NN) return;
    int64_t c = idx / NN;
    int m = (int)(idx % NN);
    keys[idx] = ((u64)cn[idx] << 32) | (u64)(c * 16 + m);
}

__global__ void k_ptr_from_keys(const u64* __restrict__ keys, int64_t nkeys, int64_t nrows, u64 stride,
                                int64_t* ptr) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i > nrows) return;
    ptr[i] = lower_bound_u64(keys, nkeys, (u64)i * stride);
}

__global__ void k_low_from_keys(const u64* __restrict__ keys, int64_t nkeys, u64 stride, int32_t* out) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= nkeys) return;
    out[p] = (int32_t)(keys[p] % stride);
}

__global__ void k_low32_from_keys(const u64* __restrict__ keys, int64_t nkeys, int32_t* out) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= nkeys) return;
    out[p] = (int32_t)(keys[p] & 0xffffffffULL);
}

__global__ void k_max_degree(const int64_t* __restrict__ ptr, int64_t n, int* out) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    atomicMax(out, (int)(ptr[i + 1] - ptr[i]));
}

template <int D>
__global__ void k_ranks(const int32_t* __restrict__ cn, const int32_t* __restrict__ cells, int64_t nc,
                        const int64_t* __restrict__ n2_ptr, const int32_t* __restrict__ n2_col,
                        const int64_t* __restrict__ n1_ptr, const int32_t* __restrict__ n1_col,
                        uint16_t* rank2, uint16_t* rank1) {
    constexpr int NN = Simplex<D>::NN, NV = Simplex<D>::NV, R2 = NN * NN, R1 = NN * NV;
    int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= nc * (R2 + R1)) return;
    int64_t c = idx / (R2 + R1);
    int r = (int)(idx % (R2 + R1));
    if (r < R2) {
        int m = r / NN, j = r % NN;
        int32_t i = cn[NN * c + m];
        int64_t s = n2_ptr[i];
        int d = (int)(n2_ptr[i + 1] - s);
        rank2[R2 * c + r] = (uint16_t)lower_bound_i32(n2_col + s, d, cn[NN * c + j]);
    } else {
        r -= R2;
        int m = r / NV, w = r % NV;
        int32_t i = cn[NN * c + m];
        int64_t s = n1_ptr[i];
        int d = (int)(n1_ptr[i + 1] - s);
        rank1[R1 * c + r] = (uint16_t)lower_bound_i32(n1_col + s, d, cells[NV * c + w]);
    }
}

__global__ void k_row_len(int64_t N, int64_t Nu, int64_t nv, int J, int dim, const int64_t* __restrict__ n2_ptr,
                          const int64_t* __restrict__ n1_ptr, int64_t* len) {
    int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r > N) return;
    if (r == N) {
        len[r] = 0;
        return;
    }
    int64_t node = r < Nu ? r / dim : (r - Nu) % nv;
    len[r] = dim * (n2_ptr[node + 1] - n2_ptr[node]) + (int64_t)J * (n1_ptr[node + 1] - n1_ptr[node]);
}

__global__ void k_fill_cols(int64_t N, int64_t Nu, int64_t nv, int J, int dim, const int64_t* __restrict__ row_ptr,
                            const int64_t* __restrict__ n2_ptr, const int32_t* __restrict__ n2_col,
                            const int64_t* __restrict__ n1_ptr, const int32_t* __restrict__ n1_col,
                            int32_t* col) {
    int lane = threadIdx.x & 31;
    int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = warp; r < N; r += nwarps) {
        int64_t node = r < Nu ? r / dim : (r - Nu) % nv;
        int64_t s2 = n2_ptr[node], s1 = n1_ptr[node];
        int d2 = (int)(n2_ptr[node + 1] - s2), d1 = (int)(n1_ptr[node + 1] - s1);
        int L = dim * d2 + J * d1;
        int64_t base = row_ptr[r];
        for (int e = lane; e < L; e += 32) {
            int32_t cidx;
            if (e < dim * d2) {
                cidx = dim * n2_col[s2 + e / dim] + e % dim;
            } else {
                int e2 = e - dim * d2;
                int a = e2 / d1;
                cidx = (int32_t)(Nu + (int64_t)a * nv + n1_col[s1 + e2 % d1]);
            }
            col[base + e] = cidx;
        }
    }
}

// a facet has D vertices and D(D-1)/2 edges (every vertex pair)
template <int D>
__global__ void k_bc_flags(const int32_t* __restrict__ bf, const int32_t* __restrict__ mk, int64_t nf, int J,
                           int64_t nv, const u64* __restrict__ ekey, int64_t ne, uint8_t* node_bc,
                           uint8_t* vert_bc) {
    int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (f >= nf) return;
    int64_t v[D];
    for (int k = 0; k < D; ++k) v[k] = bf[D * f + k];
    if (mk[f] == 0) {
        for (int k = 0; k < D; ++k) node_bc[v[k]] = 1;
        for (int i = 0; i < D; ++i)
            for (int j = i + 1; j < D; ++j) {
                int64_t a = v[i], b = v[j];
                int64_t lo = a < b ? a : b, hi = a < b ? b : a;
                int64_t pos = lower_bound_u64(ekey, ne, (u64)(lo * nv + hi));
                if (pos < ne && ekey[pos] == (u64)(lo * nv + hi)) node_bc[nv + pos] = 1;
            }
    }
    for (int a = 0; a < J; ++a)
        if (mk[(int64_t)(1 + a) * nf + f] == 0)
            for (int k = 0; k < D; ++k) vert_bc[(int64_t)a * nv + v[k]] = 1;
}

__global__ void k_bc_dofs_u(const int32_t* __restrict__ nodes, int64_t n, int dim, int32_t* dofs, uint8_t* dof_bc) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int k = 0; k < dim; ++k) {
        int32_t d = dim * nodes[i] + k;
        dofs[dim * i + k] = d;
        dof_bc[d] = 1;
    }
}

__global__ void k_bc_dofs_p(const int32_t* __restrict__ verts, int64_t n, int64_t base, int32_t* dofs,
                            uint8_t* dof_bc) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int32_t d = (int32_t)(base + verts[i]);
    dofs[i] = d;
    dof_bc[d] = 1;
}

// --- host drivers -------------------------------------------------------------------

template <int D>
static void build_topology_d(mpet_ctx* c) {
    constexpr int NE = Simplex<D>::NE, NN = Simplex<D>::NN, NV = Simplex<D>::NV;
    cudaStream_t s = c->stream;
    const int T = 256;
    int64_t nc = c->nc, nv = c->nv;
    // edges
    {
        TmpBuf keys(sizeof(u64) * nc * NE);
        k_edge_keys<D><<<grid_for(nc * NE, T), T, 0, s>>>(c->cells, nc, nv, keys.as<u64>());
        MPET_CHECK_LAUNCH();
        u64* ek = nullptr;
        c->ne = sort_unique(c, keys.as<u64>(), nc * NE, bits_for((u64)nv * (u64)nv), &ek);
        c->edge_key = (int64_t*)ek;
    }
    c->nnodes = nv + c->ne;
    c->cell_nodes = c->pool.alloc<int32_t>(nc * NN);
    k_cell_nodes<D><<<grid_for(nc * NN, T), T, 0, s>>>(c->cells, nc, nv, (const u64*)c->edge_key, c->ne,
                                                     c->cell_nodes);
    MPET_CHECK_LAUNCH();
    c->geo = c->pool.alloc<double>(nc * 16);
    if (D == 3) k_geometry<<<grid_for(nc, T), T, 0, s>>>(c->x, c->cells, nc, c->geo);
    else k_geometry2<<<grid_for(nc, T), T, 0, s>>>(c->x, c->cells, nc, c->geo);
    MPET_CHECK_LAUNCH();
    int64_t nn = c->nnodes;
    // P2 node adjacency
    {
        TmpBuf keys(sizeof(u64) * nc * NN * NN);
        k_pairs_n2<D><<<grid_for(nc * NN * NN, T), T, 0, s>>>(c->cell_nodes, nc, nn, keys.as<u64>());
        MPET_CHECK_LAUNCH();
        u64* uk = nullptr;
        c->n2_nnz = sort_unique(c, keys.as<u64>(), nc * NN * NN, bits_for((u64)nn * (u64)nn), &uk);
        c->n2_ptr = c->pool.alloc<int64_t>(nn + 1);
        c->n2_col = c->pool.alloc<int32_t>(c->n2_nnz);
        k_ptr_from_keys<<<grid_for(nn + 1, T), T, 0, s>>>(uk, c->n2_nnz, nn, (u64)nn, c->n2_ptr);
        k_low_from_keys<<<grid_for(c->n2_nnz, T), T, 0, s>>>(uk, c->n2_nnz, (u64)nn, c->n2_col);
        MPET_CHECK_LAUNCH();
        MPET_CUDA(cudaStreamSynchronize(s));
        c->pool.release(uk);
    }
    // vertices adjacent to each node
    {
        TmpBuf keys(sizeof(u64) * nc * NN * NV);
        k_pairs_n1<D><<<grid_for(nc * NN * NV, T), T, 0, s>>>(c->cell_nodes, c->cells, nc, nv, keys.as<u64>());
        MPET_CHECK_LAUNCH();
        u64* uk = nullptr;
        c->n1_nnz = sort_unique(c, keys.as<u64>(), nc * NN * NV, bits_for((u64)nn * (u64)nv), &uk);
        c->n1_ptr = c->pool.alloc<int64_t>(nn + 1);
        c->n1_col = c->pool.alloc<int32_t>(c->n1_nnz);
        k_ptr_from_keys<<<grid_for(nn + 1, T), T, 0, s>>>(uk, c->n1_nnz, nn, (u64)nv, c->n1_ptr);
        k_low_from_keys<<<grid_for(c->n1_nnz, T), T, 0, s>>>(uk, c->n1_nnz, (u64)nv, c->n1_col);
        MPET_CHECK_LAUNCH();
        MPET_CUDA(cudaStreamSynchronize(s));
        c->pool.release(uk);
    }
    // node -> cell incidence (cells ascending within a node)
    {
        if (nc >= (1LL << 27)) fail(MPET_ERR_INVALID, "too many cells (limit 2^27: cell * 16 + local fits int32)");
        TmpBuf keys(sizeof(u64) * nc * NN);
        k_pairs_inc<D><<<grid_for(nc * NN, T), T, 0, s>>>(c->cell_nodes, nc, keys.as<u64>());
        MPET_CHECK_LAUNCH();
        u64* uk = nullptr;
        int64_t n = sort_unique(c, keys.as<u64>(), nc * NN, 32 + bits_for((u64)nn), &uk);
        if (n != nc * NN) fail(MPET_ERR_INVALID, "degenerate cell (repeated vertex)");
        c->inc_ptr = c->pool.alloc<int64_t>(nn + 1);
        c->inc = c->pool.alloc<int32_t>(n);
        k_ptr_from_keys<<<grid_for(nn + 1, T), T, 0, s>>>(uk, n, nn, 1ULL << 32, c->inc_ptr);
        k_low32_from_keys<<<grid_for(n, T), T, 0, s>>>(uk, n, c->inc);
        MPET_CHECK_LAUNCH();
        MPET_CUDA(cudaStreamSynchronize(s));
        c->pool.release(uk);
    }
    // degree limits of the 16-bit rank tables
    {
        TmpBuf mx(sizeof(int) * 2);
        MPET_CUDA(cudaMemsetAsync(mx.p, 0, sizeof(int) * 2, s));
        k_max_degree<<<grid_for(nn, T), T, 0, s>>>(c->n2_ptr, nn, mx.as<int>());
        k_max_degree<<<grid_for(nn, T), T, 0, s>>>(c->inc_ptr, nn, mx.as<int>() + 1);
        MPET_CHECK_LAUNCH();
        int h[2];
        MPET_CUDA(cudaMemcpyAsync(h, mx.p, sizeof(h), cudaMemcpyDeviceToHost, s));
        MPET_CUDA(cudaStreamSynchronize(s));
        if (h[0] >= 65535) fail(MPET_ERR_INVALID, "node degree too large for 16-bit ranks");
    }
    c->rank2 = c->pool.alloc<uint16_t>(nc * NN * NN);
    c->rank1 = c->pool.alloc<uint16_t>(nc * NN * NV);
    k_ranks<D><<<grid_for(nc * (NN * NN + NN * NV), T), T, 0, s>>>(c->cell_nodes, c->cells, nc, c->n2_ptr, c->n2_col, c->n1_ptr,
                                                 c->n1_col, c->rank2, c->rank1);
    MPET_CHECK_LAUNCH();
}

void build_topology(mpet_ctx* c) {
    if (c->dim == 2) build_topology_d<2>(c);
    else build_topology_d<3>(c);
}

void build_pattern(mpet_ctx* c) {
    cudaStream_t s = c->stream;
    const int T = 256;
    int J = c->J;
    c->Nu = (int64_t)c->dim * c->nnodes;
    c->N = c->Nu + (int64_t)J * c->nv;
    if (c->N >= 2147483647LL) fail(MPET_ERR_INVALID, "too many DOFs for 32-bit column ids");
    int64_t N = c->N;
    c->A.n = c->A.m = N;
    c->A.rp = c->pool.alloc<int64_t>(N + 1);
    {
        TmpBuf len(sizeof(int64_t) * (N + 1));
        k_row_len<<<grid_for(N + 1, T), T, 0, s>>>(N, c->Nu, c->nv, J, c->dim, c->n2_ptr, c->n1_ptr,
                                                   len.as<int64_t>());
        MPET_CHECK_LAUNCH();
        size_t tb = 0;
        MPET_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, len.as<int64_t>(), c->A.rp, (int)(N + 1), s));
        TmpBuf tmp(tb);
        MPET_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, len.as<int64_t>(), c->A.rp, (int)(N + 1), s));
    }
    MPET_CUDA(cudaMemcpyAsync(&c->nnz, c->A.rp + N, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    MPET_CUDA(cudaStreamSynchronize(s));
    c->A.nnz = c->nnz;
    c->A.ci = c->pool.alloc<int32_t>(c->nnz);
    k_fill_cols<<<152 * 16, 256, 0, s>>>(N, c->Nu, c->nv, J, c->dim, c->A.rp, c->n2_ptr, c->n2_col, c->n1_ptr,
                                         c->n1_col, c->A.ci);
    MPET_CHECK_LAUNCH();
    c->A.lpr = choose_lpr(N, c->nnz);
    {
        std::vector<int64_t> rp(N + 1);
        MPET_CUDA(cudaMemcpyAsync(rp.data(), c->A.rp, sizeof(int64_t) * (N + 1), cudaMemcpyDeviceToHost, s));
        MPET_CUDA(cudaStreamSynchronize(s));
        build_tiles(c, c->A, rp.data());
        for (int64_t i = 0; i < c->nnodes; ++i) {
            const int64_t len = rp[c->dim * i + 1] - rp[c->dim * i], rows = c->dim + (i < c->nv ? J : 0);
            int& m = c->asm_rows[i < c->nv ? 0 : 1];
            m = (int)std::max<int64_t>(m, std::min<int64_t>(len * rows, 1 << 20));
        }
    }
    // preconditioner block patterns: u-Laplacian on n2, P1 blocks on the vertex rows of n1
    c->Lu.n = c->Lu.m = c->nnodes;
    c->Lu.nnz = c->n2_nnz;
    c->Lu.rp = c->n2_ptr;
    c->Lu.ci = c->n2_col;
    c->Lu.lpr = choose_lpr(c->nnodes, c->n2_nnz);
    int64_t p1nnz = 0;
    MPET_CUDA(cudaMemcpyAsync(&p1nnz, c->n1_ptr + c->nv, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    MPET_CUDA(cudaStreamSynchronize(s));
    for (int a = 0; a < J; ++a) {
        c->Pp[a].n = c->Pp[a].m = c->nv;
        c->Pp[a].nnz = p1nnz;
        c->Pp[a].rp = c->n1_ptr;
        c->Pp[a].ci = c->n1_col;
        c->Pp[a].lpr = choose_lpr(c->nv, p1nnz);
    }
}

static int64_t compact_flags(mpet_ctx* c, const uint8_t* flags, int64_t n, int32_t** out) {
    TmpBuf buf(sizeof(int32_t) * (n > 0 ? n : 1));
    TmpBuf nsel(sizeof(int));
    size_t tb = 0;
    thrust::counting_iterator<int32_t> it(0);
    MPET_CUDA(cub::DeviceSelect::Flagged(nullptr, tb, it, flags, buf.as<int32_t>(), nsel.as<int>(), (int)n, c->stream));
    {
        TmpBuf tmp(tb);
        MPET_CUDA(cub::DeviceSelect::Flagged(tmp.p, tb, it, flags, buf.as<int32_t>(), nsel.as<int>(), (int)n,
                                             c->stream));
    }
    int cnt = 0;
    MPET_CUDA(cudaMemcpyAsync(&cnt, nsel.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    MPET_CUDA(cudaStreamSynchronize(c->stream));
    int32_t* o = c->pool.alloc<int32_t>(cnt);
    if (cnt) MPET_CUDA(cudaMemcpyAsync(o, buf.p, sizeof(int32_t) * cnt, cudaMemcpyDeviceToDevice, c->stream));
    MPET_CUDA(cudaStreamSynchronize(c->stream));
    *out = o;
    return cnt;
}

void build_bc(mpet_ctx* c) {
    cudaStream_t s = c->stream;
    const int T = 256;
    int J = c->J;
    c->node_bc = c->pool.alloc<uint8_t>(c->nnodes);
    c->vert_bc = c->pool.alloc<uint8_t>((int64_t)J * c->nv);
    c->dof_bc = c->pool.alloc<uint8_t>(c->N);
    MPET_CUDA(cudaMemsetAsync(c->node_bc, 0, c->nnodes, s));
    MPET_CUDA(cudaMemsetAsync(c->vert_bc, 0, (size_t)J * c->nv, s));
    MPET_CUDA(cudaMemsetAsync(c->dof_bc, 0, c->N, s));
    if (c->nf > 0) {
        if (c->dim == 2)
            k_bc_flags<2><<<grid_for(c->nf, T), T, 0, s>>>(c->bfacets, c->markers, c->nf, J, c->nv,
                                                            (const u64*)c->edge_key, c->ne, c->node_bc, c->vert_bc);
        else
            k_bc_flags<3><<<grid_for(c->nf, T), T, 0, s>>>(c->bfacets, c->markers, c->nf, J, c->nv,
                                                            (const u64*)c->edge_key, c->ne, c->node_bc, c->vert_bc);
        MPET_CHECK_LAUNCH();
    }
    c->nbc_nodes[0] = compact_flags(c, c->node_bc, c->nnodes, &c->bc_nodes[0]);
    for (int a = 0; a < J; ++a)
        c->nbc_nodes[1 + a] = compact_flags(c, c->vert_bc + (int64_t)a * c->nv, c->nv, &c->bc_nodes[1 + a]);
    c->bc_off[0] = 0;
    c->bc_off[1] = (int64_t)c->dim * c->nbc_nodes[0];
    for (int a = 0; a < J; ++a) c->bc_off[2 + a] = c->bc_off[1 + a] + c->nbc_nodes[1 + a];
    c->nbc_dofs = c->bc_off[1 + J];
    c->bc_dofs = c->pool.alloc<int32_t>(c->nbc_dofs);
    c->bc_vals = c->pool.alloc<double>(c->nbc_dofs);
    MPET_CUDA(cudaMemsetAsync(c->bc_vals, 0, sizeof(double) * (c->nbc_dofs > 0 ? c->nbc_dofs : 1), s));
    if (c->nbc_nodes[0])
        k_bc_dofs_u<<<grid_for(c->nbc_nodes[0], T), T, 0, s>>>(c->bc_nodes[0], c->nbc_nodes[0], c->dim,
                                                                c->bc_dofs, c->dof_bc);
    for (int a = 0; a < J; ++a)
        if (c->nbc_nodes[1 + a])
            k_bc_dofs_p<<<grid_for(c->nbc_nodes[1 + a], T), T, 0, s>>>(
                c->bc_nodes[1 + a], c->nbc_nodes[1 + a], c->Nu + (int64_t)a * c->nv, c->bc_dofs + c->bc_off[1 + a],
                c->dof_bc);
    MPET_CHECK_LAUNCH();
    MPET_CUDA(cudaStreamSynchronize(s));
}


// ---- patches of cells --------------------------------------------------------------
//
// Cells in Morton order of their centroids (instance by instance in a batch), cut into
// patches of at most P cells; per patch its node list, the cells' local ids, the places of
// their contributions and, for nodes of several patches, the slots of their partial sums.  All
// from sorted 64-bit keys, as above: the numbering is the same in every run.

__device__ __forceinline__ u64 spread3(u64 v) {
    u64 r = 0;
    for (int b = 0; b < 14; ++b) r |= ((v >> b) & 1ULL) << (3 * b);
    return r;
}

__global__ void k_cell_morton(const double* __restrict__ x, const int32_t* __restrict__ cells, int64_t nc,
                              const int32_t* __restrict__ inst, double lo0, double lo1, double lo2, double scale,
                              u64* key, int32_t* idx) {
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const double lo[3] = {lo0, lo1, lo2};
    u64 m = 0;
    for (int k = 0; k < 3; ++k) {
        double s = 0.0;
        for (int v = 0; v < 4; ++v) s += x[3 * (int64_t)cells[4 * c + v] + k];
        double q = (0.25 * s - lo[k]) * scale;
        q = q < 0.0 ? 0.0 : (q > 16383.0 ? 16383.0 : q);
        m |= spread3((u64)q) << k;
    }
    key[c] = ((u64)(inst ? inst[c] : 0) << 42) | m;
    idx[c] = (int32_t)c;
}

__global__ void k_patch_slots(int64_t np, int P, const int32_t* __restrict__ pstart,
                              const int32_t* __restrict__ order, int32_t* cell) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= np * P) return;
    const int64_t p = s / P;
    const int l = (int)(s % P);
    cell[s] = l < pstart[p + 1] - pstart[p] ? order[pstart[p] + l] : -1;
}

__global__ void k_patch_node_keys(int64_t np, int P, const int32_t* __restrict__ cell,
                                  const int32_t* __restrict__ cn, u64* key) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= np * P * 10) return;
    const int64_t s = r / 10;
    const int32_t c = cell[s];
    // (padding repeats the patch's first node)
    const int64_t cc = c >= 0 ? c : cell[s / P * P];
    key[r] = ((u64)(s / P) << 32) | (u64)cn[10 * cc + (c >= 0 ? r % 10 : 0)];
}

__global__ void k_patch_ptr(const u64* __restrict__ key, int64_t n, int64_t np, int64_t nv, int32_t* ptr,
                            int32_t* pnv) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p > np) return;
    const int64_t b = lower_bound_u64(key, n, (u64)p << 32);
    ptr[p] = (int32_t)b;
    if (p < np) pnv[p] = (int32_t)(lower_bound_u64(key, n, ((u64)p << 32) | (u64)nv) - b);
}

// cells of the patch at each of its nodes
__global__ void k_patch_valence(int64_t np, int P, const int32_t* __restrict__ cell, const int32_t* __restrict__ cn,
                                const u64* __restrict__ key, const int32_t* __restrict__ ptr, int32_t* val) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= np * P * 10) return;
    const int64_t s = r / 10, p = s / P;
    const int32_t c = cell[s];
    if (c < 0) return;
    const int32_t b = ptr[p];
    const u64 k = ((u64)p << 32) | (u64)cn[10 * (int64_t)c + r % 10];
    atomicAdd(val + b + lower_bound_u64(key + b, ptr[p + 1] - b, k), 1);
}

// order of a patch's nodes: vertices, then edges, each by decreasing valence (a warp's
// threads then add about equally many contributions), then by node
__global__ void k_patch_order_keys(int64_t npn, const u64* __restrict__ key, const int32_t* __restrict__ val,
                                   int64_t nv, u64* okey, int32_t* idx) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= npn) return;
    const u64 node = key[i] & 0xffffffffu;
    const int v = val[i] < 255 ? val[i] : 255;
    okey[i] = ((key[i] >> 32) << 40) | ((node < (u64)nv ? 0ULL : 1ULL) << 39) | ((u64)(255 - v) << 31) | node;
    idx[i] = (int32_t)i;
}

__global__ void k_patch_reorder(int64_t npn, const int32_t* __restrict__ idx, const u64* __restrict__ key,
                                u64* okey, int32_t* inv) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= npn) return;
    okey[i] = key[idx[i]];
    inv[idx[i]] = (int32_t)i;
}

// local ids of every slot's cell, and the contribution keys (patch node << 16) | (j P + lane)
__global__ void k_patch_lids(int64_t np, int P, const int32_t* __restrict__ cell, const int32_t* __restrict__ cn,
                             const u64* __restrict__ key, const int32_t* __restrict__ inv,
                             const int32_t* __restrict__ ptr, uint32_t* lid, u64* gkey) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= np * P) return;
    const int64_t p = s / P;
    const int l = (int)(s % P);
    const int32_t c = cell[s];
    const int32_t b = ptr[p];
    const int64_t n = ptr[p + 1] - b;
    for (int w = 0; w < 5; ++w) {
        uint32_t v = 0;
        for (int h = 0; h < 2; ++h) {
            const int j = 2 * w + h;
            uint32_t i = 0;
            if (c >= 0)
                i = (uint32_t)(inv[b + lower_bound_u64(key + b, n, ((u64)p << 32) | (u64)cn[10 * (int64_t)c + j])] - b);
            v |= i << (16 * h);
            gkey[s * 10 + j] = c >= 0 ? (((u64)b + i) << 16) | (u64)(j * P + l) : ~0ULL;
        }
        lid[(p * 5 + w) * P + l] = v;
    }
}

// place of each slot's values among its patch's contributions (sorted by node, then lane)
__global__ void k_patch_pos(int64_t np, int P, const int32_t* __restrict__ cell, const u64* __restrict__ gkey,
                            int64_t n, const int32_t* __restrict__ ptr, const uint32_t* __restrict__ lid,
                            const int32_t* __restrict__ pstart, uint32_t* pos) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= np * P) return;
    const int64_t p = s / P;
    const int l = (int)(s % P);
    const int32_t c = cell[s];
    const int64_t g0 = 10 * (int64_t)pstart[p];
    const int64_t gn = 10 * (int64_t)(pstart[p + 1] - pstart[p]);
    for (int w = 0; w < 5; ++w) {
        const uint32_t ids = lid[(p * 5 + w) * P + l];
        uint32_t v = 0;
        for (int h = 0; h < 2; ++h) {
            const int j = 2 * w + h;
            uint32_t q = 0xffffu;  // (padding)
            if (c >= 0)
                q = (uint32_t)lower_bound_u64(gkey + g0, gn,
                                              (((u64)ptr[p] + ((ids >> (16 * h)) & 0xffffu)) << 16) | (u64)(j * P + l));
            v |= q << (16 * h);
        }
        pos[(p * 5 + w) * P + l] = v;
    }
}

__global__ void k_patch_gl_ptr(const u64* __restrict__ gkey, int64_t n, const u64* __restrict__ key, int64_t npn,
                               const int32_t* __restrict__ ptr, const int32_t* __restrict__ pstart,
                               uint16_t* gl_ptr) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= npn) return;
    const int64_t p = (int64_t)(key[i] >> 32);
    gl_ptr[i + p] = (uint16_t)(lower_bound_u64(gkey, n, (u64)i << 16) - 10 * (int64_t)pstart[p]);
    if (i + 1 == ptr[p + 1]) gl_ptr[i + p + 1] = (uint16_t)(10 * (pstart[p + 1] - pstart[p]));
}

__global__ void k_patch_node_major(int64_t npn, const u64* __restrict__ key, u64* nkey) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < npn) nkey[i] = (key[i] << 32) | (u64)i;
}

// per node: whether several patches hold it, and its number of partial sums; *none: some node is in no
// patch
__global__ void k_patch_shared(int64_t nnodes, const u64* __restrict__ nkey, int64_t npn, int32_t* shared,
                               int32_t* slots, int32_t* none) {
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (v >= nnodes) return;
    const int n = (int)(lower_bound_u64(nkey, npn, (u64)(v + 1) << 32) - lower_bound_u64(nkey, npn, (u64)v << 32));
    shared[v] = n > 1;
    slots[v] = n > 1 ? n : 0;
    if (n == 0) *none = 1;
}

__global__ void k_patch_fill_shared(int64_t npn, const u64* __restrict__ nkey,
                                    const int32_t* __restrict__ shared, const int32_t* __restrict__ sid,
                                    const int32_t* __restrict__ sbase, const int32_t* __restrict__ slots,
                                    const uint8_t* __restrict__ node_bc, int32_t* pn_node, int32_t* pn_sh,
                                    int32_t* sh_ptr, int32_t* sh_node) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= npn) return;
    const int64_t v = (int64_t)(nkey[i] >> 32), pn = (int64_t)(nkey[i] & 0xffffffffu);
    pn_node[pn] = (int32_t)v | (node_bc[v] ? (int32_t)0x80000000 : 0);
    if (!shared[v]) {
        pn_sh[pn] = -1;
        return;
    }
    const int rank = (int)(i - lower_bound_u64(nkey, npn, (u64)v << 32));
    pn_sh[pn] = sbase[v] + rank;
    if (rank == 0) {
        sh_node[sid[v]] = pn_node[pn];
        sh_ptr[sid[v]] = sbase[v];
        sh_ptr[sid[v] + 1] = sbase[v] + slots[v];  // (the next shared node writes the same value)
    }
}

// lower corner and longest side of the vertices' bounding box
static void bounding_box(mpet_ctx* c, double lo[3], double& ext) {
    std::vector<double> xyz((size_t)c->nv * 3);
    MPET_CUDA(cudaMemcpyAsync(xyz.data(), c->x, sizeof(double) * xyz.size(), cudaMemcpyDeviceToHost, c->stream));
    MPET_CUDA(cudaStreamSynchronize(c->stream));
    ext = 0.0;
    for (int k = 0; k < 3; ++k) {
        double hi = -1e300;
        lo[k] = 1e300;
        for (int64_t v = 0; v < c->nv; ++v) {
            lo[k] = xyz[3 * v + k] < lo[k] ? xyz[3 * v + k] : lo[k];
            hi = xyz[3 * v + k] > hi ? xyz[3 * v + k] : hi;
        }
        ext = hi - lo[k] > ext ? hi - lo[k] : ext;
    }
}

void release_patches(mpet_ctx* c) {
    PatchSet& s = c->patch;
    for (void* p : {(void*)s.cell, (void*)s.lid, (void*)s.pn_ptr, (void*)s.pn_nv, (void*)s.pn_node, (void*)s.pn_sh,
                    (void*)s.sh_ptr, (void*)s.sh_node, (void*)s.gl_ptr, (void*)s.pos, (void*)s.inst, (void*)s.part,
                    (void*)s.part_p, (void*)s.sys, (void*)s.coef})
        c->pool.release(p);
    s = PatchSet();
    c->sys_patch = false;
}

void build_patches(mpet_ctx* c) {
    PatchSet& s = c->patch;
    if (s.tried) return;
    s.tried = true;
    const int64_t nc = c->nc;
    if (c->dim != 3 || nc < 1 || c->prm.precision != MPET_PRECISION_MIXED) return;
    // cells per patch: 256 once every SM gets two patches of them, else smaller patches so that
    // a small mesh still spreads over the chip
    const int P = nc >= 256 * 304 ? 256 : (nc >= 128 * 152 ? 128 : 64);
    const int J = c->J;
    if (!device_fits(c, (size_t)nc * (200 + 4 * (10 + J * J + J)) + (size_t)c->nnodes * (16 + 4 * J) * 2)) return;
    cudaStream_t st = c->stream;
    const int T = 256;
    // patch boundaries (host): instance by instance, patches of equal size
    std::vector<int64_t> ncell(c->ninst > 0 ? c->ninst : 1, 0);
    if (c->ninst > 0) {
        std::vector<int32_t> ci(nc);
        MPET_CUDA(cudaMemcpyAsync(ci.data(), c->cell_inst, sizeof(int32_t) * nc, cudaMemcpyDeviceToHost, st));
        MPET_CUDA(cudaStreamSynchronize(st));
        for (int32_t i : ci) ncell[i]++;
    } else {
        ncell[0] = nc;
    }
    std::vector<int32_t> pstart, pinst;
    int64_t base = 0;
    for (size_t i = 0; i < ncell.size(); ++i) {
        const int64_t k = (ncell[i] + P - 1) / P;
        for (int64_t q = 0; q < k; ++q) {
            pstart.push_back((int32_t)(base + ncell[i] * q / k));
            pinst.push_back((int32_t)i);
        }
        base += ncell[i];
    }
    const int64_t np = (int64_t)pstart.size();
    pstart.push_back((int32_t)nc);
    if (np * P * 10 >= 2147483647LL || c->nnodes >= (1LL << 30)) return;  // (32-bit keys, flag bits)
    TmpBuf d_pstart(sizeof(int32_t) * (np + 1));
    MPET_CUDA(cudaMemcpyAsync(d_pstart.p, pstart.data(), sizeof(int32_t) * (np + 1), cudaMemcpyHostToDevice, st));
    double lo[3], ext;
    bounding_box(c, lo, ext);
    const double scale = ext > 0.0 ? 16384.0 / ext : 0.0;
    s.cell = c->pool.alloc<int32_t>(np * P);
    {
        TmpBuf k0(sizeof(u64) * nc), k1(sizeof(u64) * nc), i0(sizeof(int32_t) * nc), i1(sizeof(int32_t) * nc);
        k_cell_morton<<<grid_for(nc, T), T, 0, st>>>(c->x, c->cells, nc, c->ninst > 0 ? c->cell_inst : nullptr, lo[0],
                                                     lo[1], lo[2], scale, k0.as<u64>(), i0.as<int32_t>());
        MPET_CHECK_LAUNCH();
        size_t tb = 0;
        const int eb = 42 + bits_for((u64)ncell.size());
        MPET_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, k0.as<u64>(), k1.as<u64>(), i0.as<int32_t>(),
                                                  i1.as<int32_t>(), (int)nc, 0, eb, st));
        TmpBuf tmp(tb);
        MPET_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, k0.as<u64>(), k1.as<u64>(), i0.as<int32_t>(),
                                                  i1.as<int32_t>(), (int)nc, 0, eb, st));
        k_patch_slots<<<grid_for(np * P, T), T, 0, st>>>(np, P, d_pstart.as<int32_t>(), i1.as<int32_t>(), s.cell);
        MPET_CHECK_LAUNCH();
        MPET_CUDA(cudaStreamSynchronize(st));
    }
    // patch nodes
    const int64_t nref = np * P * 10;
    u64* key = nullptr;
    {
        TmpBuf keys(sizeof(u64) * nref);
        k_patch_node_keys<<<grid_for(nref, T), T, 0, st>>>(np, P, s.cell, c->cell_nodes, keys.as<u64>());
        MPET_CHECK_LAUNCH();
        s.npn = sort_unique(c, keys.as<u64>(), nref, 32 + bits_for((u64)np), &key);
    }
    s.pn_ptr = c->pool.alloc<int32_t>(np + 1);
    s.pn_nv = c->pool.alloc<int32_t>(np);
    k_patch_ptr<<<grid_for(np + 1, T), T, 0, st>>>(key, s.npn, np, c->nv, s.pn_ptr, s.pn_nv);
    MPET_CHECK_LAUNCH();
    std::vector<int32_t> ptr(np + 1), pnv(np);
    MPET_CUDA(cudaMemcpyAsync(ptr.data(), s.pn_ptr, sizeof(int32_t) * (np + 1), cudaMemcpyDeviceToHost, st));
    MPET_CUDA(cudaMemcpyAsync(pnv.data(), s.pn_nv, sizeof(int32_t) * np, cudaMemcpyDeviceToHost, st));
    // the patch nodes in their order within the patch
    TmpBuf inv(sizeof(int32_t) * s.npn), okey(sizeof(u64) * s.npn);
    {
        TmpBuf val(sizeof(int32_t) * s.npn), k0(sizeof(u64) * s.npn), i0(sizeof(int32_t) * s.npn),
            i1(sizeof(int32_t) * s.npn);
        MPET_CUDA(cudaMemsetAsync(val.p, 0, sizeof(int32_t) * s.npn, st));
        k_patch_valence<<<grid_for(nref, T), T, 0, st>>>(np, P, s.cell, c->cell_nodes, key, s.pn_ptr,
                                                         val.as<int32_t>());
        k_patch_order_keys<<<grid_for(s.npn, T), T, 0, st>>>(s.npn, key, val.as<int32_t>(), c->nv, k0.as<u64>(),
                                                             i0.as<int32_t>());
        MPET_CHECK_LAUNCH();
        size_t tb = 0;
        const int eb = 40 + bits_for((u64)np);
        MPET_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, k0.as<u64>(), okey.as<u64>(), i0.as<int32_t>(),
                                                  i1.as<int32_t>(), (int)s.npn, 0, eb, st));
        TmpBuf tmp(tb);
        MPET_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, k0.as<u64>(), okey.as<u64>(), i0.as<int32_t>(),
                                                  i1.as<int32_t>(), (int)s.npn, 0, eb, st));
        k_patch_reorder<<<grid_for(s.npn, T), T, 0, st>>>(s.npn, i1.as<int32_t>(), key, okey.as<u64>(),
                                                          inv.as<int32_t>());
        MPET_CHECK_LAUNCH();
        MPET_CUDA(cudaStreamSynchronize(st));
    }
    // local ids and places of the contributions
    s.lid = c->pool.alloc<uint32_t>(np * P * 5);
    s.pos = c->pool.alloc<uint32_t>(np * P * 5);
    s.gl_ptr = c->pool.alloc<uint16_t>(s.npn + np);
    {
        TmpBuf keys(sizeof(u64) * nref);
        k_patch_lids<<<grid_for(np * P, T), T, 0, st>>>(np, P, s.cell, c->cell_nodes, key, inv.as<int32_t>(),
                                                        s.pn_ptr, s.lid, keys.as<u64>());
        MPET_CHECK_LAUNCH();
        u64* gk = nullptr;
        sort_unique(c, keys.as<u64>(), nref, 64, &gk);
        k_patch_pos<<<grid_for(np * P, T), T, 0, st>>>(np, P, s.cell, gk, nc * 10, s.pn_ptr, s.lid,
                                                       d_pstart.as<int32_t>(), s.pos);
        k_patch_gl_ptr<<<grid_for(s.npn, T), T, 0, st>>>(gk, nc * 10, okey.as<u64>(), s.npn, s.pn_ptr,
                                                         d_pstart.as<int32_t>(), s.gl_ptr);
        MPET_CHECK_LAUNCH();
        MPET_CUDA(cudaStreamSynchronize(st));
        c->pool.release(gk);
    }
    for (int64_t p = 0; p < np; ++p) {
        s.max_pn = std::max(s.max_pn, ptr[p + 1] - ptr[p]);
        s.max_pv = std::max(s.max_pv, pnv[p]);
    }
    // nodes of several patches
    s.pn_node = c->pool.alloc<int32_t>(s.npn);
    s.pn_sh = c->pool.alloc<int32_t>(s.npn);
    {
        const int64_t nn = c->nnodes;
        TmpBuf keys(sizeof(u64) * s.npn), shared(sizeof(int32_t) * (nn + 1)), slots(sizeof(int32_t) * (nn + 1)),
            sid(sizeof(int32_t) * (nn + 1)), sbase(sizeof(int32_t) * (nn + 1));
        k_patch_node_major<<<grid_for(s.npn, T), T, 0, st>>>(s.npn, okey.as<u64>(), keys.as<u64>());
        MPET_CHECK_LAUNCH();
        u64* nk = nullptr;
        sort_unique(c, keys.as<u64>(), s.npn, 32 + bits_for((u64)nn), &nk);
        for (TmpBuf* b : {&shared, &slots}) MPET_CUDA(cudaMemsetAsync(b->p, 0, sizeof(int32_t) * (nn + 1), st));
        TmpBuf none(sizeof(int32_t));
        MPET_CUDA(cudaMemsetAsync(none.p, 0, sizeof(int32_t), st));
        k_patch_shared<<<grid_for(nn, T), T, 0, st>>>(nn, nk, s.npn, shared.as<int32_t>(), slots.as<int32_t>(),
                                                      none.as<int32_t>());
        MPET_CHECK_LAUNCH();
        size_t tb = 0;
        MPET_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, shared.as<int32_t>(), sid.as<int32_t>(), (int)(nn + 1), st));
        TmpBuf tmp(tb);
        MPET_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, shared.as<int32_t>(), sid.as<int32_t>(), (int)(nn + 1), st));
        MPET_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, slots.as<int32_t>(), sbase.as<int32_t>(), (int)(nn + 1), st));
        int32_t tot[5];
        MPET_CUDA(cudaMemcpyAsync(&tot[4], none.p, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        MPET_CUDA(cudaMemcpyAsync(&tot[0], sid.as<int32_t>() + nn, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        MPET_CUDA(cudaMemcpyAsync(&tot[1], sbase.as<int32_t>() + nn, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        MPET_CUDA(cudaMemcpyAsync(&tot[2], sid.as<int32_t>() + c->nv, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        MPET_CUDA(cudaMemcpyAsync(&tot[3], sbase.as<int32_t>() + c->nv, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        MPET_CUDA(cudaStreamSynchronize(st));
        if (tot[4]) {  // a vertex of no cell: no patch would write its rows of the product
            c->pool.release(nk);
            c->pool.release(key);
            release_patches(c);
            s.tried = true;
            return;
        }
        s.nsh = tot[0];
        s.nslot = tot[1];
        s.nshv = tot[2];
        s.nslotv = tot[3];
        s.sh_ptr = c->pool.alloc<int32_t>(s.nsh + 1);
        s.sh_node = c->pool.alloc<int32_t>(s.nsh);
        MPET_CUDA(cudaMemsetAsync(s.sh_ptr, 0, sizeof(int32_t) * (s.nsh + 1), st));
        k_patch_fill_shared<<<grid_for(s.npn, T), T, 0, st>>>(s.npn, nk, shared.as<int32_t>(), sid.as<int32_t>(),
                                                              sbase.as<int32_t>(), slots.as<int32_t>(), c->node_bc,
                                                              s.pn_node, s.pn_sh, s.sh_ptr, s.sh_node);
        MPET_CHECK_LAUNCH();
        MPET_CUDA(cudaStreamSynchronize(st));
        c->pool.release(nk);
    }
    c->pool.release(key);
    // shared memory of a block (patch.cuh): x at the nodes and the contributions
    if (4 * (5 * s.max_pn + J * s.max_pv + (30 + 4 * J) * P) > PATCH_SMEM) {
        release_patches(c);
        c->patch.tried = true;
        return;
    }
    if (c->ninst > 0) {
        s.inst = c->pool.alloc<int32_t>(np);
        MPET_CUDA(cudaMemcpyAsync(s.inst, pinst.data(), sizeof(int32_t) * np, cudaMemcpyHostToDevice, st));
    }
    s.part = c->pool.alloc<float>(s.nslot * 4);
    s.part_p = c->pool.alloc<float>(s.nslotv * J);
    s.sys = c->pool.alloc<float>(np * P * 10);
    MPET_CUDA(cudaStreamSynchronize(st));
    s.P = P;
    s.np = np;
    launch_patch_geometry(c);
}


// ---- row tiles --------------------------------------------------------------------

__global__ void k_node_morton(const double* __restrict__ x, const int64_t* __restrict__ ekey, int64_t nn, int64_t nv,
                              const int32_t* __restrict__ inst, double lo0, double lo1, double lo2, double scale,
                              u64* key, int32_t* idx) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nn) return;
    const double lo[3] = {lo0, lo1, lo2};
    u64 m = 0;
    for (int k = 0; k < 3; ++k) {
        const double p = i < nv ? x[3 * i + k]
                                : 0.5 * (x[3 * (ekey[i - nv] / nv) + k] + x[3 * (ekey[i - nv] % nv) + k]);
        double q = (p - lo[k]) * scale;
        q = q < 0.0 ? 0.0 : (q > 16383.0 ? 16383.0 : q);
        m |= spread3((u64)q) << k;
    }
    key[i] = ((u64)(inst ? inst[i] : 0) << 42) | m;
    idx[i] = (int32_t)i;
}

const int32_t* node_order(mpet_ctx* c) {
    if (c->node_order) return c->node_order;
    const int64_t nn = c->nnodes;
    double lo[3], ext;
    bounding_box(c, lo, ext);
    int32_t* o = c->pool.alloc<int32_t>(nn);
    TmpBuf k0(sizeof(u64) * nn), k1(sizeof(u64) * nn), i0(sizeof(int32_t) * nn);
    k_node_morton<<<grid_for(nn, 256), 256, 0, c->stream>>>(c->x, c->edge_key, nn, c->nv,
                                                            c->ninst > 0 ? c->node_inst : nullptr, lo[0], lo[1], lo[2],
                                                            ext > 0.0 ? 16384.0 / ext : 0.0, k0.as<u64>(),
                                                            i0.as<int32_t>());
    MPET_CHECK_LAUNCH();
    size_t tb = 0;
    const int eb = 42 + bits_for((u64)(c->ninst > 0 ? c->ninst : 1));
    MPET_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, k0.as<u64>(), k1.as<u64>(), i0.as<int32_t>(), o, (int)nn, 0,
                                              eb, c->stream));
    TmpBuf tmp(tb);
    MPET_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, k0.as<u64>(), k1.as<u64>(), i0.as<int32_t>(), o, (int)nn, 0,
                                              eb, c->stream));
    MPET_CUDA(cudaStreamSynchronize(c->stream));
    c->node_order = o;
    return o;
}

__global__ void k_tile_row_keys(int64_t n, int R, const int32_t* __restrict__ order, const int64_t* __restrict__ rp,
                                u64* key, int32_t* row) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t r = order ? order[i] : (int32_t)i;
    key[i] = ((u64)(i / R) << 32) | (u64)(0xffffffffu - (unsigned)(rp[r + 1] - rp[r]));
    row[i] = r;
}

__global__ void k_tile_perm(int64_t n, const int32_t* __restrict__ row, int32_t* perm) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) perm[row[i]] = (int32_t)i;
}

// steps of every warp (its first row is its longest) and the entries of every tile
__global__ void k_tile_steps(int64_t nt, int R, int lpr, const int32_t* __restrict__ row,
                             const int64_t* __restrict__ rp, uint16_t* steps, int64_t* ent) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const int rw = 32 / lpr;
    int64_t sum = 0;
    for (int w = 0; w < 8; ++w) {
        const int32_t r = row[t * R + w * rw];
        const int64_t len = r >= 0 ? rp[r + 1] - rp[r] : 0;
        const int64_t s = (len + 2 * lpr - 1) / (2 * lpr);
        steps[t * 8 + w] = (uint16_t)(s < 65535 ? s : 65535);
        sum += s;
    }
    ent[t] = sum * 64;
}

__global__ void k_tile_col_keys(int64_t nrows, int R, const int32_t* __restrict__ row, const int64_t* __restrict__ rp,
                                const int32_t* __restrict__ ci, const int32_t* __restrict__ perm, u64* key) {
    const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3;  // eight lanes per row
    const int l = threadIdx.x & 7;
    if (i >= nrows || row[i] < 0) return;
    const int32_t r = row[i];
    for (int64_t e = rp[r] + l; e < rp[r + 1]; e += 8) key[e] = ((u64)(i / R) << 32) | (u64)(unsigned)(perm ? perm[ci[e]] : ci[e]);
}

__global__ void k_tile_cptr(const u64* __restrict__ key, int64_t n, int64_t nt, int32_t* cptr) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t <= nt) cptr[t] = (int32_t)lower_bound_u64(key, n, (u64)t << 32);
}

// the tiles' column lists, mc apart, padded with the first column
__global__ void k_tile_cols(int64_t nt, int mc, const u64* __restrict__ key, const int32_t* __restrict__ cptr,
                            int32_t* col) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nt * mc) return;
    const int64_t t = i / mc;
    const int q = (int)(i % mc), n = cptr[t + 1] - cptr[t];
    col[i] = n > 0 ? (int32_t)(key[cptr[t] + (q < n ? q : 0)] & 0xffffffffu) : 0;
}

template <typename T>
__global__ void k_tile_fill(int64_t nt, int R, int lpr, const int32_t* __restrict__ row,
                            const int64_t* __restrict__ rp, const int32_t* __restrict__ ci,
                            const int32_t* __restrict__ perm, const double* __restrict__ v,
                            const int32_t* __restrict__ cptr, int mc, const int32_t* __restrict__ col,
                            const int64_t* __restrict__ eoff, const uint16_t* __restrict__ steps, T* tv,
                            uint16_t* tl) {
    const int64_t th = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (th >= nt * 256) return;
    const int64_t t = th >> 8;
    const int w = (int)(th >> 5) & 7, lane = (int)th & 31;
    const int rw = 32 / lpr, sub = lane % lpr;
    int base = 0;
    for (int q = 0; q < w; ++q) base += steps[t * 8 + q];
    const int n = steps[t * 8 + w];
    const int32_t r = row[t * R + w * rw + lane / lpr];
    const int64_t b = r >= 0 ? rp[r] : 0, len = r >= 0 ? rp[r + 1] - b : 0;
    const int32_t* cs = col + t * mc;
    const int nc = cptr[t + 1] - cptr[t];
    // padding: value 0 at the row's last column (a valid place, as in the SELL copy)
    auto place = [&](int64_t e) { return (uint16_t)lower_bound_i32(cs, nc, perm ? perm[ci[e]] : ci[e]); };
    const uint16_t pad = len > 0 ? place(b + len - 1) : 0;
    for (int q = 0; q < n; ++q)
        for (int h = 0; h < 2; ++h) {
            const int64_t e = 2 * ((int64_t)q * lpr + sub) + h;
            const int64_t o = eoff[t] + 2 * ((int64_t)(base + q) * 32 + lane) + h;
            tv[o] = e < len ? (T)v[b + e] : T(0);
            tl[o] = e < len ? place(b + e) : pad;
        }
}

void release_row_tiles(mpet_ctx* c, RowTiles& r) {
    for (void* p : {(void*)r.row, (void*)r.perm, (void*)r.col, (void*)r.eoff, (void*)r.steps, r.v, (void*)r.lc,
                    (void*)r.skl})
        c->pool.release(p);
    r = RowTiles();
}

// false: a tile of R rows does not fit in shared memory
static bool build_tiles_of(mpet_ctx* c, Csr& A, const int32_t* order, int nvec, bool fp32, int R) {
    const int lpr = 256 / R;
    RowTiles& r = A.rt;
    const int64_t n = A.n, nnz = A.nnz;
    cudaStream_t st = c->stream;
    const int64_t nt = (n + R - 1) / R;
    const int T = 256;
    r.row = c->pool.alloc<int32_t>(nt * R);
    MPET_CUDA(cudaMemsetAsync(r.row, 0xff, sizeof(int32_t) * nt * R, st));
    {
        TmpBuf k0(sizeof(u64) * n), k1(sizeof(u64) * n), i0(sizeof(int32_t) * n);
        k_tile_row_keys<<<grid_for(n, T), T, 0, st>>>(n, R, order, A.rp, k0.as<u64>(), i0.as<int32_t>());
        MPET_CHECK_LAUNCH();
        size_t tb = 0;
        const int eb = 32 + bits_for((u64)nt);
        MPET_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, k0.as<u64>(), k1.as<u64>(), i0.as<int32_t>(), r.row,
                                                  (int)n, 0, eb, st));
        TmpBuf tmp(tb);
        MPET_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, k0.as<u64>(), k1.as<u64>(), i0.as<int32_t>(), r.row,
                                                  (int)n, 0, eb, st));
        MPET_CUDA(cudaStreamSynchronize(st));
    }
    if (order) {
        r.perm = c->pool.alloc<int32_t>(n);
        k_tile_perm<<<grid_for(n, T), T, 0, st>>>(n, r.row, r.perm);
        MPET_CHECK_LAUNCH();
    }
    r.steps = c->pool.alloc<uint16_t>(nt * 8);
    r.eoff = c->pool.alloc<int64_t>(nt + 1);
    k_tile_steps<<<grid_for(nt, T), T, 0, st>>>(nt, R, lpr, r.row, A.rp, r.steps, r.eoff);
    MPET_CHECK_LAUNCH();
    std::vector<int64_t> eo(nt + 1);
    MPET_CUDA(cudaMemcpyAsync(eo.data(), r.eoff, sizeof(int64_t) * nt, cudaMemcpyDeviceToHost, st));
    MPET_CUDA(cudaStreamSynchronize(st));
    int64_t total = 0, max_ent = 0;
    for (int64_t t = 0; t < nt; ++t) {
        const int64_t e = eo[t];
        max_ent = std::max(max_ent, e);
        eo[t] = total;
        total += e;
    }
    eo[nt] = total;
    MPET_CUDA(cudaMemcpyAsync(r.eoff, eo.data(), sizeof(int64_t) * (nt + 1), cudaMemcpyHostToDevice, st));
    if (max_ent > 65536) {  // (bounds the steps of a warp)
        release_row_tiles(c, r);
        return false;
    }
    // distinct columns
    u64* key = nullptr;
    int64_t ncol = 0;
    {
        TmpBuf keys(sizeof(u64) * nnz);
        k_tile_col_keys<<<grid_for(nt * R * 8, T), T, 0, st>>>(nt * R, R, r.row, A.rp, A.ci, r.perm, keys.as<u64>());
        MPET_CHECK_LAUNCH();
        ncol = sort_unique(c, keys.as<u64>(), nnz, 32 + bits_for((u64)nt), &key);
    }
    TmpBuf cptr(sizeof(int32_t) * (nt + 1));
    k_tile_cptr<<<grid_for(nt + 1, T), T, 0, st>>>(key, ncol, nt, cptr.as<int32_t>());
    MPET_CHECK_LAUNCH();
    std::vector<int32_t> cp(nt + 1);
    MPET_CUDA(cudaMemcpyAsync(cp.data(), cptr.p, sizeof(int32_t) * (nt + 1), cudaMemcpyDeviceToHost, st));
    MPET_CUDA(cudaStreamSynchronize(st));
    for (int64_t t = 0; t < nt; ++t) r.mc = std::max(r.mc, cp[t + 1] - cp[t]);
    r.mc = (r.mc + 31) / 32 * 32;
    // (x in shared memory: three blocks per SM at least)
    if ((size_t)r.mc * nvec * (fp32 ? 4 : 8) > TILE_SMEM || r.mc > TILE_MAX_COLS) {
        c->pool.release(key);
        release_row_tiles(c, r);
        return false;
    }
    r.col = c->pool.alloc<int32_t>(nt * r.mc);
    k_tile_cols<<<grid_for(nt * r.mc, T), T, 0, st>>>(nt, r.mc, key, cptr.as<int32_t>(), r.col);
    MPET_CHECK_LAUNCH();
    MPET_CUDA(cudaStreamSynchronize(st));
    c->pool.release(key);
    r.lc = c->pool.alloc<uint16_t>(total);
    if (fp32) {
        r.v = c->pool.alloc<float>(total);
        k_tile_fill<float><<<grid_for(nt * 256, T), T, 0, st>>>(nt, R, lpr, r.row, A.rp, A.ci, r.perm, A.v64,
                                                                     cptr.as<int32_t>(), r.mc,
                                                                r.col, r.eoff, r.steps, (float*)r.v, r.lc);
    } else {
        r.v = c->pool.alloc<double>(total);
        k_tile_fill<double><<<grid_for(nt * 256, T), T, 0, st>>>(nt, R, lpr, r.row, A.rp, A.ci, r.perm, A.v64,
                                                                     cptr.as<int32_t>(), r.mc,
                                                                 r.col, r.eoff, r.steps, (double*)r.v, r.lc);
    }
    MPET_CHECK_LAUNCH();
    MPET_CUDA(cudaStreamSynchronize(st));
    r.fp32 = fp32;
    r.R = R;
    r.nt = nt;
    return true;
}

void build_row_tiles(mpet_ctx* c, Csr& A, const int32_t* order, int nvec, bool fp32) {
    const int64_t n = A.n, nnz = A.nnz;
    if (n == 0 || nnz == 0 || nnz >= 2147483647LL || !A.v64) return;
    const size_t ev = (fp32 ? 4 : 8) + 2;
    if (!device_fits(c, (size_t)nnz * (24 + ev + ev / 4) + (size_t)n * 24)) return;
    // Rows per tile: 256 on a large level (the more rows, the fewer x entries per row: the
    // displacement level at 64^3 takes 1650, 1237 and 1071 us with 64, 128 and 256, 1157 with 512);
    // 128 below 400,000 rows, where the tiles are few waves of blocks (24^3, 118,000 rows: 205 us
    // per iteration against 237 with 256); less on a small level so that every SM has two tiles.
    int R = n >= 400000 ? 256 : 128;
    while (R > 32 && n < (int64_t)R * 304) R >>= 1;
    for (; R >= 32; R >>= 1)
        if (build_tiles_of(c, A, order, nvec, fp32, R)) return;
}

// ---- a level's transfers in tile order -----------------------------------------------

__global__ void k_perm_len(int64_t n, const int32_t* __restrict__ row, const int64_t* __restrict__ rp, int64_t* len) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i <= n) len[i] = i < n ? rp[row[i] + 1] - rp[row[i]] : 0;
}

__global__ void k_perm_rows(int64_t n, const int32_t* __restrict__ row, const int64_t* __restrict__ rp,
                            const int32_t* __restrict__ ci, const double* __restrict__ v,
                            const int64_t* __restrict__ rpt, int32_t* cit, double* vt,
                            const double* __restrict__ dinv, double* dinvt) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t b = rp[row[i]], len = rp[row[i] + 1] - b;
    for (int64_t e = 0; e < len; ++e) {
        cit[rpt[i] + e] = ci[b + e];
        vt[rpt[i] + e] = v[b + e];
    }
    dinvt[i] = dinv[row[i]];
}

__global__ void k_perm_cols(int64_t nnz, const int32_t* __restrict__ ci, const int32_t* __restrict__ perm,
                            int32_t* cit) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e < nnz) cit[e] = perm[ci[e]];
}

void permute_transfers(mpet_ctx* c, const int32_t* perm, const int32_t* row, const Csr& P, const Csr& R,
                       const double* dinv, Csr& Pt, Csr& Rt, double** dinvt) {
    cudaStream_t st = c->stream;
    Pt.n = P.n;
    Pt.m = P.m;
    Pt.nnz = P.nnz;
    Pt.rp = c->pool.alloc<int64_t>(P.n + 1);
    Pt.ci = c->pool.alloc<int32_t>(P.nnz);
    Pt.v64 = c->pool.alloc<double>(P.nnz);
    *dinvt = c->pool.alloc<double>(P.n);
    {
        TmpBuf len(sizeof(int64_t) * (P.n + 1));
        k_perm_len<<<grid_for(P.n + 1, 256), 256, 0, st>>>(P.n, row, P.rp, len.as<int64_t>());
        MPET_CHECK_LAUNCH();
        size_t tb = 0;
        MPET_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, len.as<int64_t>(), Pt.rp, (int)(P.n + 1), st));
        TmpBuf tmp(tb);
        MPET_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, len.as<int64_t>(), Pt.rp, (int)(P.n + 1), st));
        k_perm_rows<<<grid_for(P.n, 256), 256, 0, st>>>(P.n, row, P.rp, P.ci, P.v64, Pt.rp, Pt.ci, Pt.v64, dinv,
                                                        *dinvt);
        MPET_CHECK_LAUNCH();
        MPET_CUDA(cudaStreamSynchronize(st));
    }
    Rt.n = R.n;
    Rt.m = R.m;
    Rt.nnz = R.nnz;
    Rt.rp = c->pool.alloc<int64_t>(R.n + 1);
    Rt.ci = c->pool.alloc<int32_t>(R.nnz);
    Rt.v64 = c->pool.alloc<double>(R.nnz);
    MPET_CUDA(cudaMemcpyAsync(Rt.rp, R.rp, sizeof(int64_t) * (R.n + 1), cudaMemcpyDeviceToDevice, st));
    MPET_CUDA(cudaMemcpyAsync(Rt.v64, R.v64, sizeof(double) * R.nnz, cudaMemcpyDeviceToDevice, st));
    k_perm_cols<<<grid_for(R.nnz, 256), 256, 0, st>>>(R.nnz, R.ci, perm, Rt.ci);
    MPET_CHECK_LAUNCH();
}

}  // namespace mpet
