// nnp_tc.cu -- atomic networks on the tensor cores (tcgen05, sm_100a).
//
// Replaces k_nn_fp32 for NNP_PREC_BF16 / NNP_PREC_BF16X3: ANN::fpbp plus
// DODZ::grad (ml/nn.cpp:1402-1420, 1836-1859) for tiles of 128 atoms of one
// element.  Each hidden layer is one M=128 MMA chain per tile,
//     Z_h = A_h W_h^T          (A_0 = inpw * (G + inpb)),
// with the bias and activation applied by the thread that owns the row while
// it reads the FP32 accumulator out of TMEM.  The output layer (one neuron,
// linear) is a dot product on the CUDA cores.  The input gradient runs the
// same chain backwards,
//     D_{h-1} = (D_h W_h) * f'(z_{h-1}),   dE/dG = (D_0 W_0) * inpw,
// so a tile costs 2 (L-1) MMA chains.  Operands are BF16 in shared memory; with
// BF16X3 every operand is split into hi + lo BF16 parts and each product is
// hi*hi + hi*lo + lo*hi (FP32 accumulation), which keeps ~16 significant bits.
//
// A tile is a chain of dependent MMAs and epilogues, so what matters is how many
// tiles an SM has in flight.  A CTA (one per SM) has up to four warpgroups, each
// with its own tile, sharing the element's weights; a tile keeps one operand
// region in shared memory (an epilogue overwrites the operand its MMA has
// consumed) and its f'(z) in TMEM columns behind the accumulator.  With weights
// and f'(z) in every tile's shared memory 2 (56-32-32-1), 1 (64-48-48-1) and 1
// (80-64-64-1) tiles fitted an SM, now 4, 3 and 2.  With the layer count as a
// template parameter (plan and widths in registers) and TMEM read 16 columns at
// a time: 1,088,749 atoms of three elements (56-32-32-1) 768 -> 433 us, 353,589
// of four (64-48-48-1) 562 -> 251 us, 131,072 of two (80-64-64-1) 301 -> 175 us.
// Other counts, split BF16, with weights and f'(z) in every tile's shared memory /
// the count at run time / as a template parameter, 4000 and 400,000 atoms: one hidden
// layer of 32: 24.5, 187 / 24.6, 127 / 20.5, 115 us; three: 43, 609 / 47, 293 / 41,
// 254; elements with two and three (always at run time): 43, 529 / 46, 254.
// Bound: the serial chain of MMAs and epilogues of a tile.
// Thread r of a warpgroup owns row r of its tile (TMEM lane r).  Tiles are taken
// in groups of one per warpgroup, all of one element, element by element over
// the element-sorted atom order; the CTA meets only to restage the weights when
// the element changes.
#include <cuda_bf16.h>

#include "nnp_device.cuh"
#include "nnp_engine.h"
#include "nnp_tc.cuh"

namespace nnp {

namespace {

constexpr int TILE = 128;
constexpr uint32_t TMEM_COLS = 512;           // allocated: all of the SM's
constexpr int MAX_GROUPS = 4;                 // tiles in flight per CTA
constexpr uint32_t WAIT_POLLS = 1u << 26;     // default bound of one MMA-chain wait (~0.1-1 s); the final drain always uses it
constexpr int HEADER = 128;                   // mbarriers (8 B each) and TMEM address slot (4 B); operands follow

__host__ __device__ inline int pad16(int n) { return (n + 15) & ~15; }
__host__ __device__ inline int pad8(int n) { return (n + 7) & ~7; }

// Shared-memory and TMEM plan of one network shape (identical on host and device).
struct TcPlan {
    int P[NNP_MAX_LAYERS + 1];   // padded widths of every layer's input
    int wf[NNP_MAX_LAYERS];      // bf16 offset of W_h   [P_{h+1} x P_h]  (forward B operand)
    int wb[NNP_MAX_LAYERS];      // bf16 offset of W_h^T [P_h x P_{h+1}]  (backward B operand)
    int dcol[NNP_MAX_LAYERS];    // TMEM column of f'(z_h), behind the accumulator
    int wbytes;                  // bytes of one copy (hi or lo) of all weight operands
    int tbytes;                  // bytes of one copy of a tile's operand region
    int cols;                    // TMEM columns of one tile
    int vfloats;                 // inpw, inpb, hidden biases, output-layer weights (FP32)
    int copies;
    __host__ __device__ int total(int groups) const { return HEADER + copies * (wbytes + groups * tbytes) + 4 * vfloats; }
};

__host__ __device__ __forceinline__ void make_plan(int L, const int *nodes, bool split, TcPlan &p)
{
    int w = 0, wide = 0;
#pragma unroll
    for (int l = 0; l < L; ++l) {
        p.P[l] = pad16(nodes[l]);
        wide = wide > p.P[l] ? wide : p.P[l];
    }
    int col = (wide + 31) & ~31;
#pragma unroll
    for (int h = 0; h + 1 < L; ++h) {
        p.wf[h] = w;
        w += p.P[h + 1] * p.P[h];
        p.wb[h] = w;
        w += p.P[h] * p.P[h + 1];
        p.dcol[h] = col;
        col += pad8(nodes[h + 1]);
    }
    p.wbytes = w * 2;
    p.tbytes = TILE * wide * 2;
    p.cols = (col + 31) & ~31;
    int v = 2 * nodes[0] + nodes[L - 1];
#pragma unroll
    for (int h = 0; h + 1 < L; ++h) v += nodes[h + 1];
    p.vfloats = (v + 3) & ~3;
    p.copies = split ? 2 : 1;
}

struct Smem {
    __nv_bfloat16 *w_hi, *w_lo, *t_hi, *t_lo;
    float *vec;        // [inpw | inpb | bias of hidden layer 0, 1, ... | W_out[0][n]]
    uint64_t *bar;     // this warpgroup's
};

__device__ inline Smem carve(unsigned char *base, const TcPlan &p, bool split, int group, int groups)
{
    Smem s;
    s.bar = reinterpret_cast<uint64_t *>(base) + group;
    unsigned char *q = base + HEADER;
    s.w_hi = reinterpret_cast<__nv_bfloat16 *>(q); q += p.wbytes;
    s.w_lo = split ? reinterpret_cast<__nv_bfloat16 *>(q) : nullptr; q += split ? p.wbytes : 0;
    s.t_hi = reinterpret_cast<__nv_bfloat16 *>(q + (size_t)group * p.copies * p.tbytes);
    s.t_lo = split ? reinterpret_cast<__nv_bfloat16 *>(q + (size_t)group * p.copies * p.tbytes + p.tbytes) : nullptr;
    s.vec = reinterpret_cast<float *>(q + (size_t)groups * p.copies * p.tbytes);
    return s;
}

// 8 consecutive values -> one 16-byte store of BF16 (hi, and the lo remainder when split)
__device__ __forceinline__ void store8(__nv_bfloat16 *hi, __nv_bfloat16 *lo, int off, const float *v)
{
    __align__(16) __nv_bfloat16 h[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        h[i] = __float2bfloat16_rn(v[i]);
        l[i] = __float2bfloat16_rn(v[i] - __bfloat162float(h[i]));
    }
    *reinterpret_cast<uint4 *>(hi + off) = *reinterpret_cast<const uint4 *>(h);
    if (lo) *reinterpret_cast<uint4 *>(lo + off) = *reinterpret_cast<const uint4 *>(l);
}

// Bias and transposed weights of layer l of a network in the wpar layout
// (net_view's layout), found by walking the layers: no per-thread pointer
// arrays, which the compiler would keep in local memory for a run-time l.
__device__ __forceinline__ void layer_ptrs(const float *net, const DevType &T, int l, const float *&b, const float *&wt,
                                           int &ws)
{
    const float *q = net + 2 * T.nodes[0] + 2 * T.nodes[T.nlayer];
    for (int m = 0; m < l; ++m) q += T.nodes[m + 1] + (i64)T.nodes[m] * wt_stride(T.nodes[m + 1]);
    b = q;
    wt = q + T.nodes[l + 1];
    ws = wt_stride(T.nodes[l + 1]);
}

// Activation and slope in the epilogues: tanh inline, the other forms through
// one out-of-line copy of the generic switch, so the unrolled epilogue loops
// stay small (instruction fetch limited the kernel).
__device__ __noinline__ void activation_call(int neuron, float c, float z, float &a, float &d)
{
    float d2;
    activation(neuron, c, z, a, d, d2);
}

__device__ __forceinline__ void tc_activation(int neuron, float c, float z, float &a, float &d)
{
    if (neuron == NEU_TANH) {
        const float t = tanhf(c * z);
        a = t;
        d = c * (1.f - t * t);
    } else {
        activation_call(neuron, c, z, a, d);
    }
}

// One MMA chain D[128 x N] = A[128 x K] * B[N x K]^T issued by the warpgroup's
// first thread and waited for by every one of its threads, at most `polls`
// tests of the barrier each.  The result is the same in every thread of the
// group (a wait that gave up in any thread fails it for all), so the group
// leaves its tile as one and no thread is left at a barrier the others skip.
// On failure the phase is not advanced: the drain before the TMEM release
// waits for that chain.
__device__ bool gemm(const Smem &s, int group, int b_off, int K, int N, bool split, uint32_t tmem, uint32_t &phase,
                     uint32_t polls)
{
    tc::fence_async_smem();
    tc::fence_before_sync();
    tc::group_sync(group + 1);
    if ((threadIdx.x & (TILE - 1)) == 0) {
        tc::fence_after_sync();
        const uint32_t id = tc::idesc_bf16(TILE, N);
        const uint32_t sbo = (K / 8) * 128;
        const uint32_t a_hi = tc::smem_u32(s.t_hi), b_hi = tc::smem_u32(s.w_hi + b_off);
        uint32_t acc = 0;
        for (int kk = 0; kk < K / 16; ++kk) {
            const uint64_t ad = tc::sdesc(a_hi + kk * 256, 128, sbo);
            const uint64_t bd = tc::sdesc(b_hi + kk * 256, 128, sbo);
            tc::mma_bf16(tmem, ad, bd, id, acc);
            acc = 1;
            if (split) {
                const uint32_t a_lo = tc::smem_u32(s.t_lo), b_lo = tc::smem_u32(s.w_lo + b_off);
                tc::mma_bf16(tmem, ad, tc::sdesc(b_lo + kk * 256, 128, sbo), id, 1);
                tc::mma_bf16(tmem, tc::sdesc(a_lo + kk * 256, 128, sbo), bd, id, 1);
            }
        }
        tc::mma_commit(s.bar);
    }
    const bool ok = tc::group_sync_and(group + 1, tc::mbar_wait(s.bar, phase, polls));
    if (ok) phase ^= 1u;
    tc::fence_after_sync();
    return ok;
}

}  // namespace

// LT: number of layers when every element has that many (plan and widths are then
// registers; 0: any)
template <bool SPLIT, int LT>
__global__ void __launch_bounds__(MAX_GROUPS * TILE) k_nn_tc(const DevPot *__restrict__ pot,
                                                             const float *__restrict__ wpar,
                                                             const int *__restrict__ type_count,
                                                             const int *__restrict__ order, const float *__restrict__ G,
                                                             int gstride, float *__restrict__ e_atom,
                                                             float *__restrict__ dEdG, DevErr *err, uint32_t polls)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const DevPot &P = *pot;
    const int group = threadIdx.x / TILE, groups = blockDim.x / TILE, t = threadIdx.x & (TILE - 1);
    const int warp = threadIdx.x >> 5;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw);
    uint32_t *slot = reinterpret_cast<uint32_t *>(smem_raw + 8 * MAX_GROUPS);
    if (threadIdx.x == 0) {
        for (int q = 0; q < groups; ++q) tc::mbar_init(bars + q, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(slot, TMEM_COLS);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *slot;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t phase = 0;
    int staged = -1, T = 0, first = 0, base = 0;   // element, its first tile group and atom
    bool ok = true;
    for (int g = blockIdx.x;; g += gridDim.x) {
        while (T < P.ntypes) {
            const int n = (type_count[T] + groups * TILE - 1) / (groups * TILE);
            if (g < first + n) break;
            first += n;
            base += type_count[T];
            ++T;
        }
        if (T == P.ntypes) break;                  // uniform over the CTA
        const DevType &DT = P.t[T];
        const int L = LT ? LT : DT.nlayer;
        int nd[LT ? LT + 1 : NNP_MAX_LAYERS + 1];
#pragma unroll
        for (int l = 0; l <= (LT ? LT : L); ++l) nd[l] = DT.nodes[l];
        TcPlan p;
        make_plan(L, nd, SPLIT, p);
        const Smem s = carve(smem_raw, p, SPLIT, group, groups);
        const uint32_t tmem = tmem_base + group * p.cols;
        const float *net = wpar + DT.woff;
        const int nin = nd[0], nout = nd[L];
        const float *inpw = net, *inpb = net + nin, *outw = net + 2 * nin, *outb = outw + nout;
        const float *b_out, *w_out;
        int ws_out;
        layer_ptrs(net, DT, L - 1, b_out, w_out, ws_out);
        // ---- weights of this element in the operand layouts (zero padded)
        if (staged != T) {
            __syncthreads();                       // every group is done with the previous element
#pragma unroll
            for (int h = 0; h + 1 < L; ++h) {
                const int ni = nd[h], no = nd[h + 1], Pi = p.P[h], Po = p.P[h + 1];
                const float *bh, *wth;
                int ws;
                layer_ptrs(net, DT, h, bh, wth, ws);
#pragma unroll 4
                for (int q = threadIdx.x; q < Po * Pi; q += blockDim.x) {
                    const int m = q / Po, n = q - m * Po;       // W[n][m], n < Po (out), m < Pi (in)
                    const float w = (n < no && m < ni) ? wth[m * ws + n] : 0.f;
                    const __nv_bfloat16 hi = __float2bfloat16_rn(w);
                    s.w_hi[p.wf[h] + tc::kmaj(n, m, Pi)] = hi;
                    s.w_hi[p.wb[h] + tc::kmaj(m, n, Po)] = hi;
                    if (SPLIT) {
                        const __nv_bfloat16 lo = __float2bfloat16_rn(w - __bfloat162float(hi));
                        s.w_lo[p.wf[h] + tc::kmaj(n, m, Pi)] = lo;
                        s.w_lo[p.wb[h] + tc::kmaj(m, n, Po)] = lo;
                    }
                }
            }
            // per-element vectors, read by every thread in the epilogues
            {
                float *vb = s.vec + 2 * nin;
                for (int q = threadIdx.x; q < nin; q += blockDim.x) {
                    s.vec[q] = inpw[q];
                    s.vec[nin + q] = inpb[q];
                }
                for (int h = 0; h + 1 < L; ++h) {
                    const float *bh, *wth;
                    int ws;
                    layer_ptrs(net, DT, h, bh, wth, ws);
                    for (int q = threadIdx.x; q < nd[h + 1]; q += blockDim.x) vb[q] = bh[q];
                    vb += nd[h + 1];
                }
                for (int q = threadIdx.x; q < nd[L - 1]; q += blockDim.x) vb[q] = w_out[q * ws_out];
            }
            staged = T;
            tc::fence_async_smem();
            __syncthreads();
        }
        const int a0 = ((g - first) * groups + group) * TILE;    // this group's tile of the element
        if (!ok || a0 >= type_count[T]) continue;                // (uniform over the group)
        const int neuron = DT.neuron;
        const float cn = DT.c, outw0 = outw[0], eoff = outb[0] + b_out[0] * outw[0];
        const float *v_inpw = s.vec, *v_inpb = s.vec + nin, *v_bias = s.vec + 2 * nin;
        const float *v_wout = v_bias;
#pragma unroll
        for (int h = 0; h + 1 < L; ++h) v_wout += nd[h + 1];
        // ---- this thread's atom
        const bool live = a0 + t < type_count[T];
        const i64 i = live ? order[base + a0 + t] : 0;
        // A_0 = inpw * (G + inpb), zero padded; the row is read as float4
        // (gstride is a multiple of 4 and rows start 16-byte aligned)
        {
            const float *Gi = G + i * gstride;
#pragma unroll 4
            for (int k0 = 0; k0 < p.P[0]; k0 += 8) {
                float4 lo4 = make_float4(0.f, 0.f, 0.f, 0.f), hi4 = lo4;
                if (live && k0 + 4 <= gstride) lo4 = *reinterpret_cast<const float4 *>(Gi + k0);
                if (live && k0 + 8 <= gstride) hi4 = *reinterpret_cast<const float4 *>(Gi + k0 + 4);
                const float g8[8] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w};
                float v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int k = k0 + q;
                    v[q] = (live && k < nin) ? v_inpw[k] * (g8[q] + v_inpb[k]) : 0.f;
                }
                store8(s.t_hi, SPLIT ? s.t_lo : nullptr, tc::kmaj(t, k0, p.P[0]), v);
            }
        }
        // ---- forward through the hidden layers
        float e = 0.f;
        const float *bh = v_bias;
#pragma unroll
        for (int h = 0; h + 1 < L; ++h) {
            if (!ok) break;
            const int no = nd[h + 1], Po = p.P[h + 1];
            ok = gemm(s, group, p.wf[h], p.P[h], Po, SPLIT, tmem, phase, polls);
            if (!ok) break;
            const bool last = (h + 2 == L);
#pragma unroll 1
            for (int c0 = 0; c0 < Po; c0 += 16) {
                uint32_t r[2][8];
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (c0 + 8 * u < Po) tc::tmem_ld8_raw(tmem + lane_base + c0 + 8 * u, r[u]);
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (c0 + 8 * u < Po) tc::tmem_wait_tie(r[u]);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int cb = c0 + 8 * u;
                    if (cb >= Po) break;
                    float out[8], d8[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int n = cb + q;
                        out[q] = 0.f;
                        d8[q] = 0.f;
                        if (n < no) {
                            float a;
                            tc_activation(neuron, cn, __uint_as_float(r[u][q]) + bh[n], a, d8[q]);
                            if (last) {
                                // output layer: e = b + sum_n W[0][n] a_n; D = outw W[0][n] f'(z_n)
                                const float wo = v_wout[n];
                                e = fmaf(wo, a, e);
                                out[q] = outw0 * wo * d8[q];
                            } else {
                                out[q] = a;
                            }
                        }
                    }
                    if (!last && cb < pad8(no)) tc::tmem_st8(tmem + lane_base + p.dcol[h] + cb, d8);
                    // next layer's input A_{h+1}, or (last hidden layer) the first
                    // backward operand D_h; both have K = P_{h+1}
                    store8(s.t_hi, SPLIT ? s.t_lo : nullptr, tc::kmaj(t, cb, Po), out);
                }
            }
            if (!last) tc::tmem_wait_st();
            bh += no;
            if (last && live) e_atom[i] = eoff + e * outw0;
        }
        // ---- backward: D_{h-1} = (D_h W_h) * f'(z_{h-1}), dE/dG = (D_0 W_0) * inpw
#pragma unroll
        for (int h = L - 2; h >= 0; --h) {
            if (!ok) break;
            const int Pi = p.P[h], Po = p.P[h + 1];
            ok = gemm(s, group, p.wb[h], Po, Pi, SPLIT, tmem, phase, polls);
            if (!ok) break;
            const int ni = nd[h];
            float *o = dEdG + i * gstride;
#pragma unroll 1
            for (int c0 = 0; c0 < Pi; c0 += 16) {
                uint32_t r[2][8], f[2][8];
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (c0 + 8 * u < Pi) {
                        tc::tmem_ld8_raw(tmem + lane_base + c0 + 8 * u, r[u]);
                        if (h > 0 && c0 + 8 * u < pad8(ni)) tc::tmem_ld8_raw(tmem + lane_base + p.dcol[h > 0 ? h - 1 : 0] + c0 + 8 * u, f[u]);
                    }
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (c0 + 8 * u < Pi) {
                        tc::tmem_wait_tie(r[u]);
                        if (h > 0 && c0 + 8 * u < pad8(ni)) tc::tmem_wait_tie(f[u]);
                    }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int cb = c0 + 8 * u;
                    if (cb >= Pi) break;
                    float w[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int n = cb + q;
                        w[q] = (n < ni) ? __uint_as_float(r[u][q]) * (h > 0 ? __uint_as_float(f[u][q]) : v_inpw[n]) : 0.f;
                    }
                    if (h > 0) {
                        store8(s.t_hi, SPLIT ? s.t_lo : nullptr, tc::kmaj(t, cb, Pi), w);
                    } else if (live) {
                        // dE/dG row, written as float4 (gstride is a multiple of 4)
                        if (cb + 4 <= gstride) *reinterpret_cast<float4 *>(o + cb) = make_float4(w[0], w[1], w[2], w[3]);
                        if (cb + 8 <= gstride) *reinterpret_cast<float4 *>(o + cb + 4) = make_float4(w[4], w[5], w[6], w[7]);
                    }
                }
            }
        }
    }
    if (!ok && t == 0) atomicMax(&err->nonfinite, 2);
    // every issued MMA chain was waited for unless a wait gave up (in every
    // thread of the group alike); then the chain still in flight is waited for
    // once more, with the full default bound, before the TMEM is released
    if (!ok) tc::mbar_wait(bars + group, phase, WAIT_POLLS);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem_base, TMEM_COLS);
}

// Bytes of a tile that keeps every layer's operands and f'(z) to itself.  A
// network is computed in BF16 if those fit an SM's shared memory: larger ones
// have always kept FP32 networks under every precision setting, and a result
// that was FP32 stays so although the shared plan would hold more.
static int64_t tc_plain_bytes(const DevType &T, const TcPlan &p)
{
    int64_t tile = 0, slope = 0;
    for (int h = 0; h + 1 < T.nlayer; ++h) {
        tile += 2 * TILE * std::max(p.P[h], p.P[h + 1]);
        slope += 4 * TILE * T.nodes[h + 1];
    }
    return HEADER + p.copies * (p.wbytes + tile) + slope + 4 * p.vfloats;
}

// Tiles in flight that the networks' largest shapes allow in one CTA (shared
// memory, TMEM columns), at most `most`; 0 when they do not fit the tensor-core
// path (output layer wider than one neuron, no hidden layer, a layer wider than
// 128, a tile of more than an SM's shared memory).
static int tc_groups(const Engine &E, bool split, int most, int *bytes)
{
    int groups = std::min(most, MAX_GROUPS), big = 0;
    for (int T = 0; T < E.dpot.ntypes; ++T) {
        const DevType &DT = E.dpot.t[T];
        if (DT.nlayer < 2 || DT.nodes[DT.nlayer] != 1) return 0;
        for (int l = 0; l < DT.nlayer; ++l)
            if (pad16(DT.nodes[l]) > 128) return 0;
        TcPlan p;
        make_plan(DT.nlayer, DT.nodes, split, p);
        if (tc_plain_bytes(DT, p) > 227 * 1024) return 0;
        groups = std::min(groups, (int)TMEM_COLS / p.cols);
        while (groups > 0 && p.total(groups) > 227 * 1024) --groups;
    }
    for (int T = 0; T < E.dpot.ntypes; ++T) {
        TcPlan p;
        make_plan(E.dpot.t[T].nlayer, E.dpot.t[T].nodes, split, p);
        big = std::max(big, p.total(groups));
    }
    if (bytes) *bytes = big;
    return groups;
}

int tc_fits(const Engine &E, bool split) { return tc_groups(E, split, 1, nullptr); }

std::string run_nn_tc(Engine &E, bool split)
{
    const int64_t N = E.n_atoms;
    if (N == 0) return "";
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // a tile per SM before a second one on any
    const int64_t tiles = (N + TILE - 1) / TILE + E.dpot.ntypes;
    int most = (int)std::min<int64_t>(MAX_GROUPS, (tiles + nsm - 1) / nsm), sm = 0;
    if (E.tune.tc_per_sm > 0) most = std::min(most, E.tune.tc_per_sm);   // autotuned (nnp_tune.cpp)
    const int groups = tc_groups(E, split, most, &sm);
    if (groups == 0) return "networks do not fit the tensor-core path";
    const int grid = (int)std::min<int64_t>((tiles + groups - 1) / groups + E.dpot.ntypes, nsm);
    const uint32_t polls = E.mma_wait_polls > 0 ? E.mma_wait_polls : WAIT_POLLS;
    int L = E.dpot.t[0].nlayer;
    for (int T = 1; T < E.dpot.ntypes; ++T) L = E.dpot.t[T].nlayer == L ? L : 0;
    auto kern = split ? (L == 2 ? k_nn_tc<true, 2> : L == 3 ? k_nn_tc<true, 3> : L == 4 ? k_nn_tc<true, 4> : k_nn_tc<true, 0>)
                      : (L == 2 ? k_nn_tc<false, 2> : L == 3 ? k_nn_tc<false, 3> : L == 4 ? k_nn_tc<false, 4> : k_nn_tc<false, 0>);
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, NNP_SMEM_MAX);
    kern<<<grid, groups * TILE, sm, E.stream>>>(E.d_pot, E.wpar.p, E.type_fill.p, E.order.p, E.G.p, E.gstride,
                                                E.e_atom.p, E.dEdG.p, E.err.p, polls);
    E.launches += 1;
    E.mark(3);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? "" : std::string("tensor-core networks: ") + cudaGetErrorString(e);
}

}  // namespace nnp
