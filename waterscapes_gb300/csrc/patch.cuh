// FP32 product with the MPET system on patches of tetrahedra, cell by cell without a stored
// matrix (the inner Krylov products of the mixed-precision solves).  Included by solve.cu
// after the epilogues.
//
// A block owns a patch: up to P cells that are neighbours in a space-filling order
// (build_patches in setup.cu).  It gathers x at the patch's nodes into shared memory,
// one thread per cell forms the cell's product and stores each of its values at the
// place that the value has among the contributions to its node (the order of the patch's
// cells), and one thread per row group adds them up.  A node with all its cells in the patch
// is finished at once; a node shared by several patches gets one partial sum per patch, and
// a second kernel adds these in patch order and finishes it.  No value is accumulated by
// atomics: every sum has a fixed order.
//
// P2 gradients are linear on a cell, so with W_c the coefficients of grad u at vertex c over
// the barycentric gradients,
//   W_cc = 3 u_c,   W_cv = 4 u_cv - u_v,
// a cell needs the stress at its four vertices and the P1 mass matrix between them: about 700
// operations with four networks, for 40 bytes of geometry, 40 bytes of local numbering and
// the cell's share of its nodes, where the stored node-block matrix costs 2900 bytes per cell.
//
// Rounding: FP32 like the stored copy that it replaces, in other places.  Differences of u and p are
// taken before anything is scaled, so smooth vectors, whose products cancel, come out closer than from
// rounded entries.  Error against the FP64 matrix relative to || A x || (48^3, A=4; elements, stored):
// Lanczos-like vectors (M^-1 A)^5 v, displacement rows 4.9e-6, 1.7e-5, pressure rows 1e-7, 2e-6; smooth
// interpolants 2.7e-5, 7.0e-5 and 9e-12, 2.5e-11; random vectors 1.0e-7, 1.2e-7 and 4e-11, 6e-11.
// Further off only in the displacement rows of vectors that are nearly all pressure, where the stress is
// the pressure's rounding: M^-1 of random vectors 2.1e-7, 1.1e-7, of smooth ones 1.4e-6, 4.5e-7 (their
// pressure rows 8e-8, 2.4e-6).
#pragma once

struct PatchArgs {
    int P, max_pn, max_pv;
    int64_t np;
    const int32_t* __restrict__ pn_ptr;
    const int32_t* __restrict__ pn_nv;
    const int32_t* __restrict__ pn_node;
    const int32_t* __restrict__ pn_sh;
    const int32_t* __restrict__ sh_ptr;
    const uint32_t* __restrict__ lid;
    const uint32_t* __restrict__ pos;
    const uint16_t* __restrict__ gl_ptr;
    const int32_t* __restrict__ inst;
    float* part;
};

static PatchArgs patch_args(const mpet_ctx* c) {
    const PatchSet& s = c->patch;
    return PatchArgs{s.P,      s.max_pn, s.max_pv, s.np,  s.pn_ptr, s.pn_nv, s.pn_node,
                     s.pn_sh,  s.sh_ptr, s.lid,    s.pos, s.gl_ptr, s.inst,  s.part};
}

// first local node of edge (a, b), a != b: nodes 4..9 are the edges (2,3), (1,3), (1,2), (0,3), (0,2), (0,1)
__host__ __device__ constexpr int edge_node(int a, int b) {
    return a + b == 5 ? 4 : a + b == 4 ? 5 : a + b == 1 ? 9 : a + b == 2 ? 8 : (a == 0 || b == 0) ? 7 : 6;
}
static_assert(edge_node(2, 3) == 4 && edge_node(1, 3) == 5 && edge_node(1, 2) == 6 && edge_node(0, 3) == 7 &&
                  edge_node(0, 2) == 8 && edge_node(0, 1) == 9 && edge_node(3, 0) == 7 && edge_node(2, 1) == 6,
              "local edge numbering");

// ten 16-bit values of a thread's cell (five 32-bit words, two values each)
__device__ __forceinline__ void patch_u16x10(const uint32_t* __restrict__ w, int64_t p, int P, int (&id)[10]) {
    w += (p * 5) * P + threadIdx.x;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const uint32_t v = __ldg(w + q * P);
        id[2 * q] = (int)(v & 0xffffu);
        id[2 * q + 1] = (int)(v >> 16);
    }
}

// The contributions of one component of a cell.  With T_c = R_c + s and F_cv = T_c . b_v (b_0 = -(b_1 +
// b_2 + b_3)): edge (a, b): 4 w (F_ab + F_ba); vertex v: w (4 F_vv - sum_c F_cv) = w (4 R_v - s) . b_v, in
// the second form, whose large parts cancel before they are rounded.
__device__ __forceinline__ void patch_scatter(const float (&R)[4][3], const float (&s)[3], const float (&b)[3][3],
                                              float w, float* sc, const int (&pos)[10]) {
    float F[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float g[3];
#pragma unroll
        for (int l = 0; l < 3; ++l)
            g[l] = c > 0 ? b[c > 0 ? c - 1 : 0][l] : -(b[0][l] + b[1][l] + b[2][l]);
        sc[pos[c]] = w * ((4.f * R[c][0] - s[0]) * g[0] + (4.f * R[c][1] - s[1]) * g[1] + (4.f * R[c][2] - s[2]) * g[2]);
        const float t0 = R[c][0] + s[0], t1 = R[c][1] + s[1], t2 = R[c][2] + s[2];
#pragma unroll
        for (int v = 1; v < 4; ++v) F[c][v] = t0 * b[v - 1][0] + t1 * b[v - 1][1] + t2 * b[v - 1][2];
        F[c][0] = -(F[c][1] + F[c][2] + F[c][3]);
    }
    const float w4 = 4.f * w;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int e = a + 1; e < 4; ++e) sc[pos[edge_node(a, e)]] = w4 * (F[a][e] + F[e][a]);
}

// y = A x; DOT: y = A x - (beta / oldb) r1 with the partial sums of x . y (EpiMinres)
struct PatchOut {
    float* y;
    const float* r1;
    MinresScalars* sc;
};

template <bool DOT>
__device__ __forceinline__ void patch_row(const PatchOut& O, int64_t row, float acc, float r1, float xv, float c,
                                          DotAcc& dot) {
    if (DOT) {
        acc -= c * r1;
        dot.add(xv, acc);
    }
    O.y[row] = acc;
}

// this block's partial of x . y; the block of the second kernel (first > 0) that arrives last
// adds the partials of both and takes the scalar step (alfa)
template <bool DOT>
__device__ __forceinline__ void patch_dot_finish(const DotAcc& dot, double* partials, int first, unsigned* cnt,
                                                 MinresScalars* sc) {
    if (DOT) {
        __shared__ double sh[8];
        const double s = block_sum256(dot.value(), sh);
        if (threadIdx.x == 0) partials[first + blockIdx.x] = s;
        if (first == 0 || !last_block(cnt)) return;
        const double t = sum_partials_n(partials, first + gridDim.x, sh);
        if (threadIdx.x == 0) mr_alfa_one(sc, t);
    }
}

struct PatchDims {
    int64_t nv, Nu;
    int nshv;           // shared vertices (the first shared nodes)
    int64_t nslotv;     // their slots (the first slots)
    float* part_p;      // J planes of nslotv
    const uint8_t* dof_bc;
    const float* geo;   // (p * 10 + q) * P + l: b_1, b_2, b_3, |T| / 20
    const float* coef;  // per-cell coefficients, (p * nc + q) * P + l, or null
    const int64_t* bn_ptr;  // Robin matrix: entries 3 bn_ptr[v] .. 3 bn_ptr[v + 1] - 1 of vertex v
    const int32_t* rob_col;
    const float* rob_val;   // J planes of rob_n
    int64_t rob_n;
};

// the Robin matrix's part of network a's row at vertex v
__device__ __forceinline__ float patch_robin(const PatchDims& D, int a, int64_t v, const float* x) {
    const int64_t e1 = 3 * __ldg(D.bn_ptr + v + 1);
    float s = 0.f;
    for (int64_t e = 3 * __ldg(D.bn_ptr + v); e < e1; ++e)
        s += __ldg(D.rob_val + a * D.rob_n + e) * x[D.Nu + a * D.nv + __ldg(D.rob_col + e)];
    return s;
}

template <int J, bool DOT>
__global__ void __launch_bounds__(256, J <= 4 ? 3 : 2) k_patch_sys(PatchArgs A, PatchDims D, PatchCoef C,
                                                      const float* x, PatchOut O, double* partials,
                                                      const double* skip) {
    extern __shared__ float psm[];
    const int P = A.P, t = threadIdx.x, M = A.max_pn, V = A.max_pv;
    float* sx = psm;                // three planes of max_pn: u
    float* sp = sx + 3 * M;         // J planes of max_pv: p
    float* sc = sp + J * V;         // three planes of 10 P: contributions to u rows
    float* scp = sc + 30 * P;       // J planes of 4 P (the vertices' places come first): contributions to p rows
    // node (bit 30: displacement Dirichlet), or sign bit and partial-sum slot of a shared node
    unsigned* snd = reinterpret_cast<unsigned*>(scp + 4 * J * P);
    unsigned* sgp = snd + M;  // first and past-the-last contribution
    float4* part = reinterpret_cast<float4*>(A.part);
    pdl_wait();
    const float cr = DOT ? O.sc->f_c_r1 : 0.f;
    DotAcc dot;
    for (int64_t p = blockIdx.x; p < A.np; p += gridDim.x) {
        const int n0 = A.pn_ptr[p], nn = A.pn_ptr[p + 1] - n0, nvp = A.pn_nv[p];
        if (skip && skip[A.inst[p]] != 0.0) {
            // (the whole block) a converged instance: zeros, since the next iterations feed y to
            // preconditioner products that skip by 32-row slices, some of which also hold rows of
            // other instances, and rows that nothing rewrites would grow from one to the next
            for (int i = t; i < nn; i += P) {
                const int nd = __ldg(A.pn_node + n0 + i) & 0x7fffffff;
                if (__ldg(A.pn_sh + n0 + i) >= 0) continue;
#pragma unroll
                for (int k = 0; k < 3; ++k) O.y[3 * (int64_t)nd + k] = 0.f;
                if (i < nvp)
#pragma unroll
                    for (int a = 0; a < J; ++a) O.y[D.Nu + a * D.nv + nd] = 0.f;
            }
            continue;
        }
        for (int i = t; i < nn; i += P) {
            const int nd0 = __ldg(A.pn_node + n0 + i), nd = nd0 & 0x7fffffff, sh = __ldg(A.pn_sh + n0 + i);
            snd[i] = sh >= 0 ? 0x80000000u | (unsigned)sh : (unsigned)nd | (nd0 < 0 ? 1u << 30 : 0u);
            sgp[i] = (unsigned)__ldg(A.gl_ptr + n0 + p + i) | ((unsigned)__ldg(A.gl_ptr + n0 + p + i + 1) << 16);
#pragma unroll
            for (int k = 0; k < 3; ++k) sx[k * M + i] = x[3 * (int64_t)nd + k];
            if (i < nvp)
#pragma unroll
                for (int a = 0; a < J; ++a) sp[a * V + i] = x[D.Nu + a * D.nv + nd];
        }
        int id[10], pos[10];
        patch_u16x10(A.lid, p, P, id);
        patch_u16x10(A.pos, p, P, pos);
        const bool live = pos[0] != 0xffff;  // padding lanes have no cell
        float b[3][3], w;
#pragma unroll
        for (int q = 0; q < 9; ++q) b[q / 3][q % 3] = __ldg(D.geo + (p * 10 + q) * P + t);
        w = __ldg(D.geo + (p * 10 + 9) * P + t);
        __syncthreads();
        // stress (xx, yy, zz, xy, xz, yz) and divergence at the vertices
        float S[4][6], tr[4];
        {
            float H[4][3][3];  // H_c[k][l] = d u_k / d x_l at vertex c
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                float u[10];
#pragma unroll
                for (int j = 0; j < 10; ++j) u[j] = sx[k * M + id[j]];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float w0 = c == 0 ? 3.f * u[0] : 4.f * u[edge_node(c, c == 0 ? 1 : 0)] - u[0];
                    float d[3];
#pragma unroll
                    for (int v = 1; v < 4; ++v)
                        d[v - 1] = (v == c ? 3.f * u[c] : 4.f * u[edge_node(c, v == c ? (c + 1) % 4 : v)] - u[v]) - w0;
#pragma unroll
                    for (int l = 0; l < 3; ++l) H[c][k][l] = d[0] * b[0][l] + d[1] * b[1][l] + d[2] * b[2][l];
                }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                tr[c] = H[c][0][0] + H[c][1][1] + H[c][2][2];
                float dg = C.lam * tr[c];
#pragma unroll
                for (int a = 0; a < J; ++a) dg += C.cpl[a] * sp[a * V + id[c]];
#pragma unroll
                for (int k = 0; k < 3; ++k) S[c][k] = 2.f * C.mu * H[c][k][k] + dg;
                S[c][3] = C.mu * (H[c][0][1] + H[c][1][0]);
                S[c][4] = C.mu * (H[c][0][2] + H[c][2][0]);
                S[c][5] = C.mu * (H[c][1][2] + H[c][2][1]);
            }
        }
        // The P1 mass matrix between the vertices is |T| / 20 (1 + delta); the factor w comes last, as
        // on a small cell it is far smaller than the products that it scales.
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float R[4][3], s[3];  // row k of the stress at the vertices and its sum over them
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const int q = k == l ? k : k + l + 2;
#pragma unroll
                for (int c = 0; c < 4; ++c) R[c][l] = S[c][q];
                s[l] = R[0][l] + R[1][l] + R[2][l] + R[3][l];
            }
            if (live) patch_scatter(R, s, b, w, sc + k * 10 * P, pos);
        }
        // pressure rows: coupling, mass-type and stiffness terms
        {
            const float ts = tr[0] + tr[1] + tr[2] + tr[3];
            float pv[J][4], ps[J];
#pragma unroll
            for (int a = 0; a < J; ++a) {
#pragma unroll
                for (int c = 0; c < 4; ++c) pv[a][c] = sp[a * V + id[c]];
                ps[a] = pv[a][0] + pv[a][1] + pv[a][2] + pv[a][3];
            }
#pragma unroll
            for (int a = 0; a < J; ++a) {
                const float d1 = pv[a][1] - pv[a][0], d2 = pv[a][2] - pv[a][0], d3 = pv[a][3] - pv[a][0];
                float kd = C.Kd[a];
                if (C.ncell > 0) kd = __ldg(D.coef + (p * C.ncell + a) * P + t);
                kd *= 20.f;
                float gr[3];
#pragma unroll
                for (int l = 0; l < 3; ++l) gr[l] = kd * (d1 * b[0][l] + d2 * b[1][l] + d3 * b[2][l]);
                float o[4];
#pragma unroll
                for (int v = 1; v < 4; ++v) o[v] = gr[0] * b[v - 1][0] + gr[1] * b[v - 1][1] + gr[2] * b[v - 1][2];
                o[0] = -(o[1] + o[2] + o[3]);
#pragma unroll
                for (int c = 0; c < 4; ++c) o[c] += C.cpl[a] * (tr[c] + ts);
#pragma unroll
                for (int e = 0; e < J; ++e) {  // (p_e, lambda_c) = w (p_e(c) + sum)
                    float cm = C.Cm[a * MPET_MAX_NETWORKS + e];
                    if (C.ncell > J) cm = __ldg(D.coef + (p * C.ncell + J + a * J + e) * P + t);
#pragma unroll
                    for (int c = 0; c < 4; ++c) o[c] += cm * (pv[e][c] + ps[e]);
                }
                if (live)
#pragma unroll
                    for (int c = 0; c < 4; ++c) scp[a * 4 * P + pos[c]] = w * o[c];
            }
        }
        __syncthreads();
        for (int i = t; i < nn; i += P) {
            const unsigned nd = snd[i];
            const bool shared = nd >> 31;
            const int e0 = (int)(sgp[i] & 0xffffu), e1 = (int)(sgp[i] >> 16);
            const int64_t row = 3 * (int64_t)(nd & 0x3fffffffu);
            float r1[3];
            if (DOT && !shared)
#pragma unroll
                for (int k = 0; k < 3; ++k) r1[k] = O.r1[row + k];
            float a[3] = {0.f, 0.f, 0.f};
#pragma unroll 4
            for (int e = e0; e < e1; ++e) {
#pragma unroll
                for (int k = 0; k < 3; ++k) a[k] += sc[k * 10 * P + e];
            }
            if (shared) {
                part[nd & 0x7fffffffu] = make_float4(a[0], a[1], a[2], 0.f);
            } else {
                const bool bc = (nd >> 30) && C.bc;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float xv = sx[k * M + i];
                    patch_row<DOT>(O, row + k, bc ? xv : a[k], r1[k], xv, cr, dot);
                }
            }
        }
        // vertex places come first (the patch's vertices are its first nodes), all below 4 P
        for (int m = t; m < J * nvp; m += P) {
            const int net = m / nvp, i = m - net * nvp;
            const unsigned nd = snd[i];
            const bool shared = nd >> 31;
            const int e0 = (int)(sgp[i] & 0xffffu), e1 = (int)(sgp[i] >> 16);
            const int64_t row = D.Nu + net * D.nv + (nd & 0x3fffffffu);
            float r1 = 0.f;
            if (DOT && !shared) r1 = O.r1[row];
            float a = 0.f;
#pragma unroll 4
            for (int e = e0; e < e1; ++e) a += scp[net * 4 * P + e];
            if (shared) {
                D.part_p[net * D.nslotv + (nd & 0x7fffffffu)] = a;
            } else {
                const float xv = sp[net * V + i];
                if (C.robin) a += patch_robin(D, net, nd & 0x3fffffffu, x);
                patch_row<DOT>(O, row, C.bc && D.dof_bc[row] ? xv : a, r1, xv, cr, dot);
            }
        }
        __syncthreads();  // the next patch reuses the shared arrays
    }
    pdl_trigger();
    patch_dot_finish<DOT>(dot, partials, 0, nullptr, nullptr);
}

// rows of the nodes of several patches: items 0..nsh-1 the u rows of a shared node, then the
// p rows of the shared vertices, network by network
template <int J, bool DOT>
__global__ void __launch_bounds__(256) k_patch_sys_shared(int64_t nsh, const int32_t* __restrict__ sh_node,
                                                          const int32_t* __restrict__ sh_ptr,
                                                          const float4* part, PatchDims D, int bc, int robin,
                                                          const float* x, PatchOut O, double* partials,
                                                          int first, unsigned* cnt,
                                                          const int32_t* __restrict__ node_inst,
                                                          const double* skip) {
    pdl_wait();
    const float cr = DOT ? O.sc->f_c_r1 : 0.f;
    DotAcc dot;
    const int64_t items = nsh + (int64_t)J * D.nshv;
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < items; m += (int64_t)gridDim.x * blockDim.x) {
        const bool urow = m < nsh;
        const int net = urow ? 0 : (int)((m - nsh) / D.nshv);
        const int64_t i = urow ? m : m - nsh - (int64_t)net * D.nshv;
        const int nd0 = __ldg(sh_node + i), b = __ldg(sh_ptr + i), n = __ldg(sh_ptr + i + 1) - b;
        const int64_t nd = nd0 & 0x7fffffff;
        if (skip && skip[node_inst[nd]] != 0.0) {  // a converged instance: zeros, as above
            if (urow)
#pragma unroll
                for (int k = 0; k < 3; ++k) O.y[3 * nd + k] = 0.f;
            else
                O.y[D.Nu + net * D.nv + nd] = 0.f;
            continue;
        }
        if (urow) {
            float r1[3], xv[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                r1[k] = DOT ? O.r1[3 * nd + k] : 0.f;
                xv[k] = x[3 * nd + k];
            }
            float a[3] = {0.f, 0.f, 0.f};
            for (int r = 0; r < n; r += 4) {
                float4 v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = r + q < n ? part[b + r + q] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    a[0] += v[q].x;
                    a[1] += v[q].y;
                    a[2] += v[q].z;
                }
            }
            const bool fixed = nd0 < 0 && bc;
#pragma unroll
            for (int k = 0; k < 3; ++k) patch_row<DOT>(O, 3 * nd + k, fixed ? xv[k] : a[k], r1[k], xv[k], cr, dot);
        } else {
            const int64_t row = D.Nu + net * D.nv + nd;
            const float r1 = DOT ? O.r1[row] : 0.f, xv = x[row];
            float a = 0.f;
            for (int r = 0; r < n; ++r) a += D.part_p[net * D.nslotv + b + r];
            if (robin) a += patch_robin(D, net, nd, x);
            patch_row<DOT>(O, row, bc && D.dof_bc[row] ? xv : a, r1, xv, cr, dot);
        }
    }
    pdl_trigger();
    patch_dot_finish<DOT>(dot, partials, first, cnt, O.sc);
}

template <int J, bool DOT>
static void launch_patch_sys_j(mpet_ctx* c, const float* x, const PatchOut& O) {
    const PatchSet& s = c->patch;
    const size_t sm = sizeof(float) * ((size_t)5 * s.max_pn + (size_t)J * s.max_pv + (size_t)(30 + 4 * J) * s.P);
    const double* skip = s.inst ? c->skip_done : nullptr;
    const PatchDims D{c->nv, c->Nu, (int)s.nshv, s.nslotv, s.part_p, c->dof_bc, s.sys, s.coef, c->bn_ptr, c->rob_col,
                      c->rob_val, 3 * c->rob_n};
    // (reduction partials: one per block, at most NB_RED over both kernels)
    const int64_t items = s.nsh + (int64_t)J * s.nshv;
    const int g1 = (int)std::min<int64_t>(s.np, 456);
    const int g2 = (int)std::min<int64_t>(std::max<int64_t>((items + 255) / 256, 1), NB_RED - 456);
    MPET_CUDA(cudaFuncSetAttribute(k_patch_sys<J, DOT>, cudaFuncAttributeMaxDynamicSharedMemorySize, PATCH_SMEM));
    launch_k(c, k_patch_sys<J, DOT>, g1, s.P, sm, patch_args(c), D, c->patch_coef, x, O, c->partials, skip);
    launch_k(c, k_patch_sys_shared<J, DOT>, g2, 256, 0, s.nsh, s.sh_node, s.sh_ptr, (const float4*)s.part, D,
                                                          c->patch_coef.bc, c->patch_coef.robin, x, O, c->partials, g1, c->red_cnt,
                                                          c->node_inst, skip);
    MPET_CHECK_LAUNCH();
    c->n_launch += 2;
}

template <bool DOT>
static void launch_patch_sys(mpet_ctx* c, const float* x, const PatchOut& O) {
    switch (c->J) {
        case 1: launch_patch_sys_j<1, DOT>(c, x, O); return;
        case 2: launch_patch_sys_j<2, DOT>(c, x, O); return;
        case 3: launch_patch_sys_j<3, DOT>(c, x, O); return;
        case 4: launch_patch_sys_j<4, DOT>(c, x, O); return;
        case 5: launch_patch_sys_j<5, DOT>(c, x, O); return;
        case 6: launch_patch_sys_j<6, DOT>(c, x, O); return;
        case 7: launch_patch_sys_j<7, DOT>(c, x, O); return;
        default: launch_patch_sys_j<8, DOT>(c, x, O); return;
    }
}

// products of the system matrix in the Krylov iterations: element patches where they serve
// (c->sys_patch: mixed precision, tetrahedra, no forced SpMV variant, not a small matrix),
// else the stored matrix
template <typename T>
static void krylov_product(mpet_ctx* c, const T* x, T* y) {
    if constexpr (sizeof(T) == 4) {
        if (c->sys_patch) {
            launch_patch_sys<false>(c, x, PatchOut{y, nullptr, nullptr});
            return;
        }
    }
    launch_spmv<T, 1>(c, c->A, vals<T>(c->A), x, EpiStore<T, 1>{y});
}

// the Lanczos step of MINRES: y = A v - (beta / oldb) r1 and alfa = v . y
template <typename T>
static void minres_product(mpet_ctx* c, const EpiMinres<T>& e) {
    if constexpr (sizeof(T) == 4) {
        if (c->sys_patch) {
            launch_patch_sys<true>(c, e.v, PatchOut{e.y, e.r1, c->sc});
            return;
        }
    }
    launch_spmv<T, 1>(c, c->A, vals<T>(c->A), e.v, e);
    launch_k(c, k_mr_alfa, 1, 256, 0, c->sc, c->partials);
    MPET_CHECK_LAUNCH();
    c->n_launch++;
}
