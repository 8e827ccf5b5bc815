// Prologue of the streaming matvec: builds the int8 B operands of the MMAs in shared memory.
//
// int8 levels: per activation row m and per block of 256 k (one weight super-block) the values are
// written as  x ~ alpha * (l0 + l1/254 + l2/254^2),  l_i in [-127, 127], alpha = max|x| / 127 over the
// block; every level is the rounded residual of the previous ones, so three levels carry ~23 bits
// and the integer MMAs downstream are exact.  Level l of row m is column m*nl + l, stored at
//   xq[col][256*lb + 64*G + 16*c + 8*sub + 4*h + byte]   for k = 256*blk + 64*G + 32*sub + 16*h + 4*c + byte,
// i.e. the two words a lane needs for one m16n8k32 MMA are adjacent.  lb = blk - blk0 is the block
// index local to the CTA: a CTA quantises only the blocks its K-slices cover.  alam[lb][col] =
// alpha * 254^-l (0 for unused columns).  Also written: per-32 sums of x as an (hi, lo) pair of f16
// scaled by a per-block power of two whose inverse goes to minv[lb][m] (Q4_K mins), per-16 sums of
// the levels as f16 (Q6_K offset term) or per-32 sums as int32 (Q4_0 offset term).
//
// Rounding uses the 1.5 * 2^23 trick: t = x * inv + MAGIC rounds to the nearest integer in the
// FMA pipe, the level is the low byte of t's bit pattern, and no conversion instruction is issued.
#pragma once
#include "qmv_common.cuh"

namespace tlb {

#define MAGIC_RN 12582912.0f

// A block (mrow, blk) is quantised by a group of 64 threads (index j in the group) in two steps with a
// group barrier between them, so that a group can run the steps of two blocks side by side:
// warp_absmax() gives the largest magnitude among a warp's 128 values; quantise_block() takes the
// block's maximum and writes the shared tables at local block index lb.
__device__ __forceinline__ float warp_absmax(const float4 v)
{
    float mx = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    return mx;
}

template <int FMT, bool ONE>
__device__ __forceinline__ void quantise_block(const MvParams &p, uint8_t *smem, const float amax, const float4 v,
                                               int mrow, int lb, int j, int lane)
{
    const int M = ONE ? 1 : p.m, NL = ONE ? 3 : p.nl;
    // blocks whose largest magnitude is below 2^-100 (or not finite) quantise to zero levels: their
    // contribution is below f32 resolution of any realistic result, and 1 / alpha stays finite
    const float alpha = (amax > 7.9e-31f && amax < 3.0e38f) ? amax * (1.f / 127.f) : 1.f;
    float res[4] = {v.x, v.y, v.z, v.w};
    float scale = alpha, inv = __frcp_rn(alpha);
    uint32_t words[3] = {0u, 0u, 0u};
    float lsum[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int l = 0; l < 3; l++) {
        if (l < NL) {
            uint32_t tb[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                // |res * inv| <= 127 by construction at every level (alpha = max / 127; a residual is at most
                // half a step of the level before), so no clamp is needed
                const float t = fmaf(res[e], inv, MAGIC_RN);
                const float qf = t - MAGIC_RN;
                res[e] = fmaf(-qf, scale, res[e]);
                lsum[l] += qf;
                tb[e] = __float_as_uint(t);     // low byte = the level as two's-complement int8
            }
            words[l] = prmt(prmt(tb[0], tb[1], 0x0040u), prmt(tb[2], tb[3], 0x0040u), 0x5410u);
            scale *= (1.f / 254.f);
            inv *= 254.f;
        }
    }
    // k = 256*blk + 4*j + byte  ->  G = j >> 4, t = j & 15: sub = t >> 3, h = (t >> 2) & 1, c = t & 3
    const int G = j >> 4, t = j & 15;
    // one row: a sub-block's 32 bytes together, for 8-byte reads
    const int off = lb * 256 + G * 64 + (ONE ? (t >> 3) * 32 + (t & 3) * 8 : (t & 3) * 16 + (t >> 3) * 8) + ((t >> 2) & 1) * 4;
#pragma unroll
    for (int l = 0; l < 3; l++)
        if (l < NL) *reinterpret_cast<uint32_t *>(smem + p.off_xq + (size_t)(mrow * NL + l) * p.col_stride + off) = words[l];
    if (ONE) {
        // columns 0 .. 2 and 4 .. 6: the levels for either sub-block (Q4_K's second one enters as q << 4), 3 and 7 unused
        if (j < kMaxCols) {
            const int l = j & 3;
            float a = l < 3 ? alpha : 0.f;
            for (int i = 0; i < l; i++) a *= (1.f / 254.f);
            reinterpret_cast<float *>(smem + p.off_alam)[lb * kMaxCols + j] = FMT == TLB_GGML_Q4_K && j >= 4 ? a * 0.0625f : a;
        }
    } else if (j < kMaxCols) {   // alam[lb][0..7]: this row's levels; other rows' columns are written by their own groups
        const int col = j, l = col - mrow * NL;
        float *alam = reinterpret_cast<float *>(smem + p.off_alam);
        if (l >= 0 && l < NL) {
            float a = alpha;
            for (int i = 0; i < l; i++) a *= (1.f / 254.f);
            alam[lb * kMaxCols + col] = a;
        } else if (col >= M * NL && mrow == 0) {
            alam[lb * kMaxCols + col] = 0.f;   // unused columns
        }
    }
    if (FMT == TLB_GGML_Q4_K) {   // sums of x over sub-blocks of 32 = 8 consecutive k4 = 8 consecutive lanes
        // S: power of two bringing the block maximum into [512, 1024): f16 sums of 32 stay finite
        float S = 1.f;
        if (amax > 0.f && amax < 3.0e38f) {
            const int e = (int)((__float_as_uint(amax) >> 23) & 0xFF);
            const int se = 127 + 9 - (e - 127);
            if (se > 0 && se < 255) S = __uint_as_float((uint32_t)se << 23);
        }
        float t4 = ((v.x + v.y) + (v.z + v.w)) * S;
        t4 += __shfl_xor_sync(0xffffffffu, t4, 1);
        t4 += __shfl_xor_sync(0xffffffffu, t4, 2);
        t4 += __shfl_xor_sync(0xffffffffu, t4, 4);
        __half *xsum = reinterpret_cast<__half *>(smem + p.off_xsum);
        if ((lane & 7) == 0) {
            const __half hi = __float2half_rn(t4);
            const __half lo = __float2half_rn(t4 - __half2float(hi));
            xsum[(size_t)(2 * mrow) * (p.nb_max * 8) + lb * 8 + (j >> 3)] = hi;
            xsum[(size_t)(2 * mrow + 1) * (p.nb_max * 8) + lb * 8 + (j >> 3)] = lo;
        }
        if (j == 0) reinterpret_cast<float *>(smem + p.off_minv)[lb * 4 + mrow] = 1.f / S;
    }
    if (FMT == TLB_GGML_Q6_K) {   // level sums over groups of 16 = 4 consecutive lanes, as f16 (|sum| <= 2032: exact); [lb][col][16]
        __half *sa = reinterpret_cast<__half *>(smem + p.off_sa);
#pragma unroll
        for (int l = 0; l < 3; l++)
            if (l < NL) {
                float s = lsum[l];
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                // one row: columns 0 .. 2 have the sums of the even groups and zeros for the odd ones, 4 .. 6 the other way round
                if (ONE) {
                    const int col = ((j >> 2) & 1) * 4 + l;
                    if ((lane & 3) < 2) sa[((size_t)lb * kMaxCols + ((lane & 3) ? col ^ 4 : col)) * 16 + (j >> 2)] = __float2half_rn((lane & 3) ? 0.f : s);
                } else if ((lane & 3) == 0) {
                    sa[((size_t)lb * kMaxCols + mrow * NL + l) * 16 + (j >> 2)] = __float2half_rn(s);
                }
            }
        if (ONE && (lane & 3) == 2) sa[((size_t)lb * kMaxCols + 3) * 16 + (j >> 2)] = __ushort_as_half(0);
    }
    if (FMT == TLB_GGML_Q4_0) {   // level sums over blocks of 32 = 8 consecutive lanes, int32; [lb*8 + j/8][8 cols]
        int *sa = reinterpret_cast<int *>(smem + p.off_sa);
#pragma unroll
        for (int l = 0; l < 3; l++)
            if (l < NL) {
                float s = lsum[l];
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                s += __shfl_xor_sync(0xffffffffu, s, 4);
                // one row: [lb*4 + j/16][8 cols], -8 times the sums of the even block in columns 0 .. 2, of the odd one in 4 .. 6
                if ((lane & 7) == 0) {
                    if (ONE) sa[(lb * 4 + (j >> 4)) * kMaxCols + ((j >> 3) & 1) * 4 + l] = -8 * __float2int_rn(s);
                    else sa[(size_t)(lb * 8 + (j >> 3)) * kMaxCols + mrow * NL + l] = __float2int_rn(s);
                }
            }
        if (ONE && (lane & 7) == 1) sa[(lb * 4 + (j >> 4)) * kMaxCols + ((j >> 3) & 1) * 4 + 3] = 0;
    }
}

// Fills the shared tables for activation blocks [blk0, blk0 + nb) of every row.  All `nthreads`
// threads of the CTA call it; it ends with a CTA-wide barrier.
//
// Groups of 64 threads take one block each.  Everything a group needs from global memory is
// requested up front - the values of its own blocks (kept in registers), their norm weights, and
// for the fused RMSNorm its share of the REST of the row, which enters only the sum of squares - so
// the prologue costs one round trip to L2, not one per step.
//
// `after_loads(dep)` is called once per thread when the values it requested have arrived (dep is
// computed from them): the caller uses it to start traffic that should not delay those loads.
//
// The norm weights are static, so the caller fetches those of the first pass with
// load_norm_weights() BEFORE it waits for the previous kernel: they are read once per token and
// always miss L2, which would otherwise be the longest latency of the prologue.
constexpr int kKeep = 2;   // blocks per group handled in one pass

__device__ __forceinline__ void load_norm_weights(const MvParams &p, int tid, int nthreads, int blk0, int nb, float4 (&wgt)[kKeep])
{
    const int ngroups = nthreads >> 6, grp = tid >> 6, j = tid & 63;
#pragma unroll
    for (int i = 0; i < kKeep; i++) {
        wgt[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int item = grp + i * ngroups;     // ADD_NORM has one activation row: item == local block
        if (p.prologue == PRO_ADD_NORM && item < nb) wgt[i] = __ldg(reinterpret_cast<const float4 *>(p.norm_w) + (blk0 + item) * 64 + j);
    }
}

// Elements 4j .. 4j+3 of local block lb of an attention output that is still split over the keys (D-element weighted sums, maximum
// and sum of exponentials per split and query head): sum_s exp(m_s - M) v_s / sum_s exp(m_s - M) l_s.  A warp's 128 elements are one
// head of 128 or two of 64, so lane s of a head's W lanes turns split s's pair into a weight and the others take it by shuffle; the
// first rows are under way meanwhile, and more than W splits are taken W at a time.
__device__ __forceinline__ float4 attn_value(const MvParams &p, int nsplit, int e, int lane)
{
    constexpr int kRows = 8;                 // rows asked for at once
    const int W = p.att_dim >> 2, hl = lane & (W - 1);
    const int head = e / p.att_dim, d = e - head * p.att_dim;
    const int kvh = head / p.att_rep, hr = head - kvh * p.att_rep;
    const size_t sstride = (size_t)p.att_rep * (p.att_dim + 4);
    const float *row = p.att_part + ((size_t)kvh * p.att_max_splits * p.att_rep + hr) * (p.att_dim + 4);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float M = -INFINITY, sum = 0.f;
    for (int s0 = 0; s0 < nsplit; s0 += W, row += W * sstride) {
        const int n = min(W, nsplit - s0);
        float2 ml = make_float2(-INFINITY, 0.f);
        if (hl < n) ml = __ldcg(reinterpret_cast<const float2 *>(row + hl * sstride + p.att_dim));
        float4 v[kRows];
        auto load = [&](int sp) {
#pragma unroll
            for (int u = 0; u < kRows; u++)
                if (sp + u < n) v[u] = __ldcg(reinterpret_cast<const float4 *>(row + (sp + u) * sstride + d));
        };
        load(0);
        float mx = ml.x;
        for (int o = W >> 1; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mx = fmaxf(mx, M);
        const float w = hl < n ? expf(ml.x - mx) : 0.f;
        float l = ml.y * w;
        for (int o = W >> 1; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (s0) {
            const float c = expf(M - mx);
            sum *= c; acc.x *= c; acc.y *= c; acc.z *= c; acc.w *= c;
        }
        sum += l;
        M = mx;
        for (int sp = 0;;) {
#pragma unroll
            for (int u = 0; u < kRows; u++)
                if (sp + u < n) {
                    const float ws = __shfl_sync(0xffffffffu, w, sp + u, W);
                    acc.x = fmaf(ws, v[u].x, acc.x); acc.y = fmaf(ws, v[u].y, acc.y); acc.z = fmaf(ws, v[u].z, acc.z); acc.w = fmaf(ws, v[u].w, acc.w);
                }
            sp += kRows;
            if (sp >= n) break;
            load(sp);
        }
    }
    const float inv = 1.f / sum;
    return make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
}

// ONE: one activation row (three levels); its blocks are the items, no division tells them apart.  Only it has fused prologues.
template <int FMT, bool ONE, typename AfterLoads>
__device__ void build_activation(const MvParams &p, MvShared *sh, uint8_t *smem, int tid, int nthreads, int blk0, int nb, int nsplit,
                                 const float4 (&wgt_first)[kKeep], AfterLoads after_loads)
{
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthreads >> 5;
    const int ngroups = nthreads >> 6, grp = tid >> 6, j = tid & 63;
    const int nblk = p.k / 256, n_mine = (ONE ? 1 : p.m) * nb;
    const bool norm = ONE && p.prologue == PRO_ADD_NORM, attn = ONE && p.prologue == PRO_ATTN_MERGE;
    const float *emb = nullptr;
    if (norm && p.token) emb = p.emb_table + (size_t)__ldcg(p.token) * p.k;

    float inv_rms = 0.f;
    for (int first = 0; first < n_mine || (norm && first == 0); first += ngroups * kKeep) {
        float4 keep[kKeep], wgt[kKeep];
#pragma unroll
        for (int i = 0; i < kKeep; i++) {
            const int item = first + grp + i * ngroups;
            if (item < n_mine) {
                const int mrow = ONE ? 0 : item / nb, lb = item - mrow * nb, k4 = (blk0 + lb) * 64 + j;
                keep[i] = attn ? attn_value(p, nsplit, k4 * 4, lane) : prologue_value(p, emb, mrow, k4, 0.f);
                if (norm) wgt[i] = first == 0 ? wgt_first[i] : __ldg(reinterpret_cast<const float4 *>(p.norm_w) + k4);
            }
        }
        float ssq = 0.f;
        if (norm && first == 0 && p.ssq_parts) {
            // The producer of x left partial sums of squares.  Each is read once per CTA and the sums meet at the barrier below:
            // the warps of all CTAs reading all of them met on a handful of L2 lines.  With tiles' slices dealt to all CTAs
            // (qmatvec.cu), a 32-token answer of the TinyLlama shapes 23.4 -> 22.5 ms, 16 of eight Llama-3-8B layers 8.18 -> 8.05.
            for (int i = tid; i < p.n_parts; i += nthreads) ssq += __ldcg(p.ssq_parts + i);
        } else if (norm && first == 0) {
            // the blocks outside [blk0, blk0 + nb): only their squares are needed
            for (int o = grp; o < nblk - nb; o += ngroups) {
                const int k4 = (o < blk0 ? o : o + nb) * 64 + j;
                const float4 v = prologue_value(p, emb, 0, k4, 0.f);
                ssq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                if (p.x_out && blockIdx.x == 0) reinterpret_cast<float4 *>(p.x_out)[k4] = v;
            }
            for (int it = grp; it < n_mine; it += ngroups) {   // own blocks beyond the first pass, if any
                if (it < ngroups * kKeep) continue;
                const int k4 = (blk0 + it) * 64 + j;
                const float4 v = prologue_value(p, emb, 0, k4, 0.f);
                ssq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                if (p.x_out && blockIdx.x == 0) reinterpret_cast<float4 *>(p.x_out)[k4] = v;
            }
#pragma unroll
            for (int i = 0; i < kKeep; i++) {
                const int item = grp + i * ngroups;
                if (item < n_mine) {
                    const float4 v = keep[i];
                    ssq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                    if (p.x_out && blockIdx.x == 0) reinterpret_cast<float4 *>(p.x_out)[(blk0 + item) * 64 + j] = v;
                }
            }
        }
        if (first == 0) {
            float dep = ssq;
#pragma unroll
            for (int i = 0; i < kKeep; i++)
                if (grp + i * ngroups < n_mine) dep += keep[i].x;
            after_loads(dep);
        }
        // step 1 of this pass's blocks: the values, of a norm without their common factor 1 / rms, and each warp's maximum
        float *pair_max = &sh->red_max[grp * 2 * kKeep];
#pragma unroll
        for (int i = 0; i < kKeep; i++) {
            const int item = first + grp + i * ngroups;
            if (item < n_mine) {
                float4 v = keep[i];
                if (norm) { v.x *= wgt[i].x; v.y *= wgt[i].y; v.z *= wgt[i].z; v.w *= wgt[i].w; }
                keep[i] = v;
                const float mx = warp_absmax(v);
                if (lane == 0) pair_max[2 * i + (j >> 5)] = mx;
            }
        }
        if (norm && first == 0) {
            // the squares meet at the barrier that the maxima take anyway
            for (int o = 16; o; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
            if (lane == 0) sh->red_sum[warp] = ssq;
            __syncthreads();
            ssq = 0.f;
            for (int w = 0; w < nwarps; w++) ssq += sh->red_sum[w];
            inv_rms = 1.f / sqrtf(ssq / (float)p.k + p.eps);
        } else if (first + grp < n_mine) {
            named_bar(2 + grp, 64);
        }
        // step 2: the blocks are independent from here on, their instruction streams interleave.  x * weight / rms
        // (crates/tl_cpu/src/ffi.rs:2444-2486), the division as a multiply by 1 / rms; rounding keeps order, so the largest
        // product is the product of the largest
#pragma unroll
        for (int i = 0; i < kKeep; i++) {
            const int item = first + grp + i * ngroups;
            if (item < n_mine) {
                const int mrow = ONE ? 0 : item / nb, lb = item - mrow * nb;
                float4 v = keep[i];
                float mx = fmaxf(pair_max[2 * i], pair_max[2 * i + 1]);
                if (norm) { v.x *= inv_rms; v.y *= inv_rms; v.z *= inv_rms; v.w *= inv_rms; mx *= inv_rms; }
                quantise_block<FMT, ONE>(p, smem, mx, v, mrow, lb, j, lane);
            }
        }
        if (first + grp < n_mine && first + ngroups * kKeep < n_mine) named_bar(2 + grp, 64);   // pair_max is reused by the next pass
    }
    __syncthreads();
}

}  // namespace tlb
