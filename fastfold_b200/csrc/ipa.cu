// Invariant point attention core (AlphaFold Algorithm 22, lines 7-11) as one flash-style kernel.
//
// For every query residue i (four per CTA) the kernel streams the keys j in chunks and keeps, per head h,
// an online softmax over
//     logit[h][j] = w_C * q_i.k_j  +  sqrt(1/3) * (z[i][j] . W_b[h] + b_b[h])
//                   - 0.5 * gamma_h * sum_p |q_pt[i][h][p] - k_pt[j][h][p]|^2  +  inf * (mask_i * mask_j - 1)
// and the three weighted sums   o[h] = sum_j a v_j,   o_pt[h][p] = sum_j a v_pt[j][h][p] (global frame),
// o_pair[h] = sum_j a z[i][j].  The pair row z[i][:] is read ONCE from HBM (bf16) and serves both the bias projection
// and o_pair; the [H, N, N] attention tensor, the [N, N, H, P, 3] point differences and the [N, N, H] bias of the
// composite implementation never exist.  All arithmetic is fp32 (point terms must not lose the cancellation in
// |q - k|^2).  `row0` / `rows` select a block of query rows, so a rank that holds only its row shard of z computes its
// own residues (row-parallel IPA under Dynamic Axial Parallelism).
//
// Replaces the PyTorch composite of the reference (fastfold/model/nn/structure_module.py:383-505), which materialises
// all of the above through cuBLAS and elementwise kernels.
#include "common.cuh"
#include "ipa_api.h"

namespace ffb {

constexpr int IPA_THREADS = 384;   // one warp per head
constexpr int IPA_J = 64;          // keys per chunk
constexpr int IPA_ZP = 8;          // padding (bf16) of a z row in shared memory: consecutive keys fall into different banks

struct IpaArgs {
  const float* q;       // [N][H][C]
  const float* k;       // [N][H][C]
  const float* v;       // [N][H][C]
  const float* q_pts;   // [N][H][Pq][3]
  const float* k_pts;   // [N][H][Pq][3]
  const float* v_pts;   // [N][H][Pv][3]
  const bf16* z;        // [rows][N][CZ]  (row r = query row0 + r)
  const void* wb;       // [H][CZ]
  const void* bb;       // [H]
  const void* gamma;    // [H]  softplus(head_weights) * sqrt(1 / (3 * Pq * 9 / 2))
  const void* mask;     // [N]
  float* o;             // [rows][H][C]
  float* o_pt;          // [rows][H][Pv][3]
  float* o_pair;        // [rows][H][CZ]
  int N, H, C, Pq, Pv, CZ, row0, rows;
  float w_c, w_b, inf;
  int bf;               // which of wb, bb, gamma, mask are bf16 (IPA_BF16_*), the others fp32
};

__device__ __forceinline__ float ipa_load(const void* p, long long i, bool half) {
  return half ? __bfloat162float(reinterpret_cast<const bf16*>(p)[i]) : reinterpret_cast<const float*>(p)[i];
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool in_range) {
  const int bytes = in_range ? 16 : 0;                         // 0: the 16 bytes are filled with zeros, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// R query rows per CTA, 12 warps.
//   logits : warp = head, lane = key (two per chunk); k, k_pts once per key for all R rows, z and w_b from shared memory.
//            The softmax of a (row, head) stays in the warp's registers.
//   sums   : warps 0 .. 2R-1 own (row, two pair channels) for all heads, the others the 480 scalar / point channels for all
//            rows, so that v and v_pts are read once per CTA.
// The z chunk after next is on its way (cp.async) while this one is used; two barriers per chunk.
//
// What bounds it: instruction issue by three warps per scheduler, and, below some 150 CTAs, the number of SMs in use.  So everything
// goes two by two (fma.rn.f32x2): even and odd pair channels in the bias, neighbouring heads in the pair sums, neighbouring rows in the
// value sums, for which the probabilities lie in shared memory in both orders; the sums' order and so the bits are those of single FMAs.
// One row per CTA with one key-value read per row spent its time waiting for L2: every row re-read 3.2 KB of keys, values and points
// per key, a quarter of the warps in flight.
// Four rows at every length: a CTA with two, and two of those per SM, read keys and values twice as often and were slower even
// where four rows leave SMs idle.
//   Measured (B200, the core alone, us, with single FMAs, R = 2 / R = 4): N = 256 90 / 78, 512 192 / 171, 768 592 / 525, 1024 792 / 740,
//   1184 966 / 869, 1536 1796 / 1659, 2048 3207 / 2967; one row per CTA took 349 at 512.  Two by two: 512 165 -> 149, with 16 keys' values
//   on their way instead of 4 130.
template <int R, int H, int C, int PQ, int PV, int CZ>
__global__ void __launch_bounds__(IPA_THREADS, 1) ipa_fwd_kernel(const IpaArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  static_assert(H * 32 == IPA_THREADS && CZ == 128, "one warp per head");
  constexpr int ZROW = CZ + IPA_ZP;
  constexpr int PRS = H * R + 4;                             // + 4: the keys of a warp's 16-byte stores fall into different banks
  static_assert(R == 4 && H % 4 == 0, "four rows in a 16-byte access, pairs of heads");
  constexpr int VC = H * C, VT = H * PV * 3;                 // value channels from v and from v_pts
  constexpr int ZT = R * (CZ / 2);                           // threads on the pair channels
  constexpr int NV_T = IPA_THREADS - ZT;                     // threads on the value channels
  constexpr int NVA = (VC + VT + NV_T - 1) / NV_T;           // value channels per such thread
  extern __shared__ __align__(16) uint8_t ipa_smem[];
  bf16* zs = reinterpret_cast<bf16*>(ipa_smem);                                  // [2][R][J][ZROW]
  float* wbs = reinterpret_cast<float*>(ipa_smem + 2 * R * IPA_J * ZROW * 2);    // [H][CZ]
  float* qs = wbs + H * CZ;                                                      // [R][H][C]
  float* qp = qs + R * H * C;                                                    // [R][H][PQ * 3]
  float* ps = qp + R * H * PQ * 3;                                               // [R][J][H] probabilities of the chunk
  float* pr = ps + R * IPA_J * H;                                                // [J][PRS]: the same as [H][R] per key
  float* alph = pr + IPA_J * PRS;                                                // [R][H] rescale factor of the chunk
  float* lfin = alph + R * H;                                                    // [R][H] row sums at the end
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.x * R;
  const int N = a.N;
  const uint32_t zs_addr = smem_u32(zs);
  auto load_z = [&](int chunk) {
    const int j0 = chunk * IPA_J;
    for (int t = tid; t < R * IPA_J * (CZ / 8); t += IPA_THREADS) {
      const int c8 = t % (CZ / 8), j = t / (CZ / 8) % IPA_J, r = t / (CZ / 8 * IPA_J);
      const bool ok = j0 + j < N && r0 + r < a.rows;
      const bf16* src = ok ? a.z + ((long long)(r0 + r) * N + j0 + j) * CZ + c8 * 8 : a.z;
      cp_async16(zs_addr + (((chunk & 1) * R + r) * IPA_J + j) * ZROW * 2 + c8 * 16, src, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_z(0);
  for (int t = tid; t < H * CZ; t += IPA_THREADS) wbs[t] = ipa_load(a.wb, t, a.bf & IPA_BF16_WB);
  for (int t = tid; t < R * H * C; t += IPA_THREADS) {
    const int r = t / (H * C);
    qs[t] = r0 + r < a.rows ? a.q[(long long)(a.row0 + r0 + r) * H * C + t % (H * C)] : 0.f;
  }
  for (int t = tid; t < R * H * PQ * 3; t += IPA_THREADS) {
    const int r = t / (H * PQ * 3);
    qp[t] = r0 + r < a.rows ? a.q_pts[(long long)(a.row0 + r0 + r) * H * PQ * 3 + t % (H * PQ * 3)] : 0.f;
  }
  float mrun[R], lrun[R], mask_i[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    mrun[r] = -INFINITY;
    lrun[r] = 0.f;
    mask_i[r] = (a.mask && r0 + r < a.rows) ? ipa_load(a.mask, a.row0 + r0 + r, a.bf & IPA_BF16_MASK) : 1.f;
  }
  const float bb_h = ipa_load(a.bb, warp, a.bf & IPA_BF16_BB), ghalf = 0.5f * ipa_load(a.gamma, warp, a.bf & IPA_BF16_GAMMA);
  // accumulators, two by two: pair channels 2 * cp, 2 * cp + 1 of one row for every pair of heads, or NVA value channels for every
  // pair of rows
  const int zr = tid / (CZ / 2), cp = tid % (CZ / 2);
  constexpr int NACC = H > NVA * (R / 2) ? H : NVA * (R / 2);
  uint64_t acc[NACC];
#pragma unroll
  for (int i = 0; i < NACC; ++i) acc[i] = pair2(0.f, 0.f);
  int vhead[NVA], vstep[NVA];
  const float* vbase[NVA];
#pragma unroll
  for (int u = 0; u < NVA; ++u) {
    const int ch = tid - ZT + u * NV_T;
    const bool on = tid >= ZT && ch < VC + VT, pt = ch >= VC;
    vhead[u] = on ? (pt ? (ch - VC) / (PV * 3) : ch / C) : 0;
    vstep[u] = on ? (pt ? VT : VC) : 0;
    vbase[u] = on ? (pt ? a.v_pts + (ch - VC) : a.v + ch) : a.v;
  }
  const int chunks = (N + IPA_J - 1) / IPA_J;
  for (int ck = 0; ck < chunks; ++ck) {
    const int j0 = ck * IPA_J, jn = (N - j0) < IPA_J ? (N - j0) : IPA_J;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                    // chunk landed; everyone is done with the previous chunk's sums
    if (ck + 1 < chunks) load_z(ck + 1);
    const bf16* zc = zs + (ck & 1) * R * IPA_J * ZROW;
    // ---- logits and softmax: warp = head ----
    float lg[R][2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int j = half * 32 + lane;
      const bool on = j < jn;
      const long long jj = on ? j0 + j : 0;
      uint64_t zw[R];                                   // even / odd pair channels
#pragma unroll
      for (int r = 0; r < R; ++r) zw[r] = pair2(bb_h, 0.f);
#pragma unroll 4
      for (int c = 0; c < CZ; c += 8) {
        const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(wbs + warp * CZ + c), w1 = *reinterpret_cast<const ulonglong2*>(wbs + warp * CZ + c + 4);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint4 raw = *reinterpret_cast<const uint4*>(zc + (r * IPA_J + j) * ZROW + c);
          zw[r] = fma2(pair2(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u)), w0.x, zw[r]);
          zw[r] = fma2(pair2(__uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u)), w0.y, zw[r]);
          zw[r] = fma2(pair2(__uint_as_float(raw.z << 16), __uint_as_float(raw.z & 0xffff0000u)), w1.x, zw[r]);
          zw[r] = fma2(pair2(__uint_as_float(raw.w << 16), __uint_as_float(raw.w & 0xffff0000u)), w1.y, zw[r]);
        }
      }
      const float mj = a.mask ? ipa_load(a.mask, jj, a.bf & IPA_BF16_MASK) : 1.f;
      float qk[R], d2[R];
#pragma unroll
      for (int r = 0; r < R; ++r) qk[r] = d2[r] = 0.f;
      const float4* kp = reinterpret_cast<const float4*>(a.k + (jj * H + warp) * C);
#pragma unroll
      for (int c = 0; c < C / 4; ++c) {
        const float4 kv = kp[c];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4 qv = *reinterpret_cast<const float4*>(qs + (r * H + warp) * C + 4 * c);
          qk[r] += qv.x * kv.x + qv.y * kv.y + qv.z * kv.z + qv.w * kv.w;
        }
      }
      const float4* kpt = reinterpret_cast<const float4*>(a.k_pts + (jj * H + warp) * PQ * 3);
#pragma unroll
      for (int c = 0; c < PQ * 3 / 4; ++c) {
        const float4 kv = kpt[c];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4 qv = *reinterpret_cast<const float4*>(qp + (r * H + warp) * PQ * 3 + 4 * c);
          const float dx = qv.x - kv.x, dy = qv.y - kv.y, dz = qv.z - kv.z, dw = qv.w - kv.w;
          d2[r] += dx * dx + dy * dy + dz * dz + dw * dw;
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
        lg[r][half] = on ? a.w_c * qk[r] + a.w_b * (split2(zw[r]).x + split2(zw[r]).y) - ghalf * d2[r] + a.inf * (mask_i[r] * mj - 1.f) : -INFINITY;
    }
    float p0[R], p1[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float mnew = fmaxf(mrun[r], warp_max(fmaxf(lg[r][0], lg[r][1])));
      p0[r] = __expf(lg[r][0] - mnew);                                             // -inf logits (beyond N) give 0
      p1[r] = __expf(lg[r][1] - mnew);
      const float al = __expf(mrun[r] - mnew);                                     // 0 on the first chunk (-inf)
      ps[(r * IPA_J + lane) * H + warp] = p0[r];
      ps[(r * IPA_J + 32 + lane) * H + warp] = p1[r];
      lrun[r] = lrun[r] * al + warp_sum(p0[r] + p1[r]);
      mrun[r] = mnew;
      if (lane == 0) alph[r * H + warp] = al;
    }
    *reinterpret_cast<float4*>(pr + lane * PRS + warp * R) = make_float4(p0[0], p0[1], p0[2], p0[3]);
    *reinterpret_cast<float4*>(pr + (32 + lane) * PRS + warp * R) = make_float4(p1[0], p1[1], p1[2], p1[3]);
    __syncthreads();
    // ---- weighted sums ----
    if (tid < ZT) {
#pragma unroll
      for (int h2 = 0; h2 < H / 2; ++h2) {
        const uint64_t al = *reinterpret_cast<const uint64_t*>(alph + zr * H + 2 * h2);
        acc[h2] = mul2(acc[h2], al);
        acc[H / 2 + h2] = mul2(acc[H / 2 + h2], al);
      }
      const bf16* zp = zc + zr * IPA_J * ZROW + 2 * cp;
      const float* pp = ps + zr * IPA_J * H;
#pragma unroll 4
      for (int j = 0; j < IPA_J; ++j) {                 // rows past N: z = 0 and p = 0
        const uint32_t zz = *reinterpret_cast<const uint32_t*>(zp + j * ZROW);
        const float z0 = __uint_as_float(zz << 16), z1 = __uint_as_float(zz & 0xffff0000u);
        const uint64_t z00 = pair2(z0, z0), z11 = pair2(z1, z1);
#pragma unroll
        for (int h4 = 0; h4 < H / 4; ++h4) {
          const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(pp + j * H + h4 * 4);  // same address in every lane
          acc[h4 * 2] = fma2(p.x, z00, acc[h4 * 2]);
          acc[h4 * 2 + 1] = fma2(p.y, z00, acc[h4 * 2 + 1]);
          acc[H / 2 + h4 * 2] = fma2(p.x, z11, acc[H / 2 + h4 * 2]);
          acc[H / 2 + h4 * 2 + 1] = fma2(p.y, z11, acc[H / 2 + h4 * 2 + 1]);
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < NVA; ++u) {
        acc[u * 2] = mul2(acc[u * 2], pair2(alph[vhead[u]], alph[H + vhead[u]]));
        acc[u * 2 + 1] = mul2(acc[u * 2 + 1], pair2(alph[2 * H + vhead[u]], alph[3 * H + vhead[u]]));
      }
      auto add = [&](int u, int j, float v) {
        const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(pr + j * PRS + vhead[u] * R);
        const uint64_t vv = pair2(v, v);
        acc[u * 2] = fma2(p.x, vv, acc[u * 2]);
        acc[u * 2 + 1] = fma2(p.y, vv, acc[u * 2 + 1]);
      };
      // 16 keys on their way at a time: the four warps that do this read from L2 and have nothing else to fill the wait with (the
      // core at 512 residues: 2 keys 180 us, 4 149, 8 135, 16 130).  Keys past the end have probability 0 and get the value 0: with the last
      // key's, which is loaded in their place, an infinite one would make the sum NaN
#pragma unroll 1
      for (int j = 0; j < jn; j += 16) {
        float v[NVA][16];
#pragma unroll
        for (int u = 0; u < NVA; ++u)
#pragma unroll
          for (int e = 0; e < 16; ++e) v[u][e] = vbase[u][(j0 + min(j + e, jn - 1)) * vstep[u]];
        if (j + 16 > jn) {
#pragma unroll
          for (int e = 1; e < 16; ++e)
#pragma unroll
            for (int u = 0; u < NVA; ++u)
              if (j + e >= jn) v[u][e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < 16; ++e)
#pragma unroll
          for (int u = 0; u < NVA; ++u) add(u, j + e, v[u][e]);
      }
    }
  }
  // ---- normalise and store ----
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (lane == 0) lfin[r * H + warp] = lrun[r];
  __syncthreads();
  if (tid < ZT) {
    if (r0 + zr < a.rows) {
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const float l = lfin[zr * H + h];
        const float2 lo = split2(acc[h / 2]), hi = split2(acc[H / 2 + h / 2]);
        *reinterpret_cast<float2*>(a.o_pair + ((long long)(r0 + zr) * H + h) * CZ + 2 * cp) =
            h & 1 ? make_float2(lo.y / l, hi.y / l) : make_float2(lo.x / l, hi.x / l);
      }
    }
  } else {
#pragma unroll
    for (int u = 0; u < NVA; ++u) {
      const int ch = tid - ZT + u * NV_T;
      if (ch >= VC + VT) continue;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r0 + r >= a.rows) continue;
        const float2 two = split2(acc[u * 2 + r / 2]);
        const float val = (r & 1 ? two.y : two.x) / lfin[r * H + vhead[u]];
        if (ch < VC) a.o[(long long)(r0 + r) * VC + ch] = val;
        else a.o_pt[(long long)(r0 + r) * VT + ch - VC] = val;
      }
    }
  }
}

template <int R>
static int ipa_launch(const IpaArgs& a, cudaStream_t st) {
  constexpr int HH = 12, CC = 16, PQ = 4, PV = 8, CZZ = 128;
  constexpr size_t smem = 2 * R * IPA_J * (CZZ + IPA_ZP) * 2 + sizeof(float) * (HH * CZZ + R * HH * CC + R * HH * PQ * 3 + R * HH * IPA_J + IPA_J * (R * HH + 4) + 2 * R * HH);
  auto kern = ipa_fwd_kernel<R, HH, CC, PQ, PV, CZZ>;
  static SmemLimit limit;
  if (!limit.raise(kern, smem)) return -4;
  launch_light(kern, (a.rows + R - 1) / R, IPA_THREADS, smem, st, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// ---------------------------------------------------------------------------
// What surrounds the core: projections in, concatenated features out, one kernel each.  As PyTorch operations these are some
// 200 launches of a few thousand elements (rotation matrices from quaternions, three-component sums, stacks, conversions),
// which bound the layer: 1.75 ms at N = 512 where the kernels of all of them took 0.45 ms; with the two kernels here and the
// core above 0.26 ms.
// One CTA per residue; a few KB each, so the launch is what they cost.
// ---------------------------------------------------------------------------
struct Frame {
  float r[3][3], t[3];
};

// rot: [N][9] matrices or [N][4] quaternions (w, x, y, z), in fp32
__device__ __forceinline__ Frame load_frame(const float* rot, int is_quat, const float* trans, long long n) {
  Frame f;
  if (is_quat) {
    const float w = rot[n * 4], x = rot[n * 4 + 1], y = rot[n * 4 + 2], z = rot[n * 4 + 3];
    f.r[0][0] = w * w + x * x - y * y - z * z;
    f.r[0][1] = 2.f * (x * y - w * z);
    f.r[0][2] = 2.f * (x * z + w * y);
    f.r[1][0] = 2.f * (x * y + w * z);
    f.r[1][1] = w * w - x * x + y * y - z * z;
    f.r[1][2] = 2.f * (y * z - w * x);
    f.r[2][0] = 2.f * (x * z - w * y);
    f.r[2][1] = 2.f * (y * z + w * x);
    f.r[2][2] = w * w - x * x - y * y + z * z;
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) f.r[i][j] = rot[n * 9 + i * 3 + j];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) f.t[i] = trans[n * 3 + i];
  return f;
}

struct IpaPrepArgs {
  const bf16 *q, *kv, *q_pts, *kv_pts;   // projections [N][H*C], [N][H][2C], [N][3][H*Pq], [N][3][H][Pq+Pv] (x, y, z lie apart)
  const float *rot, *trans;
  int is_quat;
  float *oq, *ok, *ov, *oq_pts, *ok_pts, *ov_pts;   // [N][H][C] x 3, [N][H][P][3] x 3 (global frame)
  int N, H, C, Pq, Pv;
};

__global__ void __launch_bounds__(256) ipa_prep_kernel(const IpaPrepArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const long long n = blockIdx.x;
  const int HC = a.H * a.C;
  for (int i = threadIdx.x; i < HC; i += blockDim.x) {
    const int h = i / a.C, c = i - h * a.C;
    a.oq[n * HC + i] = __bfloat162float(a.q[n * HC + i]);
    a.ok[n * HC + i] = __bfloat162float(a.kv[n * 2 * HC + h * 2 * a.C + c]);
    a.ov[n * HC + i] = __bfloat162float(a.kv[n * 2 * HC + h * 2 * a.C + a.C + c]);
  }
  const Frame f = load_frame(a.rot, a.is_quat, a.trans, n);
  const int nq = a.H * a.Pq, pk = a.Pq + a.Pv, nk = a.H * pk;
  for (int i = threadIdx.x; i < nq + nk; i += blockDim.x) {
    const bool isq = i < nq;
    const int p = isq ? i : i - nq, np = isq ? nq : nk;
    const bf16* src = (isq ? a.q_pts : a.kv_pts) + n * 3 * np + p;
    const float x = __bfloat162float(src[0]), y = __bfloat162float(src[np]), z = __bfloat162float(src[2 * np]);
    float* dst;
    if (isq) {
      dst = a.oq_pts + (n * nq + p) * 3;
    } else {
      const int h = p / pk, r = p - h * pk;
      dst = r < a.Pq ? a.ok_pts + ((n * a.H + h) * a.Pq + r) * 3 : a.ov_pts + ((n * a.H + h) * a.Pv + r - a.Pq) * 3;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) dst[k] = f.r[k][0] * x + f.r[k][1] * y + f.r[k][2] * z + f.t[k];
  }
}

// out [N][H*C | x, y, z of H*Pv local points | their norms | H*CZ] in bf16
__global__ void __launch_bounds__(256) ipa_cat_kernel(const float* __restrict__ o, const float* __restrict__ o_pt, const float* __restrict__ o_pair,
                                                      const float* __restrict__ rot, int is_quat, const float* __restrict__ trans,
                                                      bf16* __restrict__ out, int H, int C, int Pv, int CZ, float eps) {
  pdl_launch_dependents();
  pdl_wait();
  const long long n = blockIdx.x;
  const int HC = H * C, HP = H * Pv, HZ = H * CZ;
  bf16* dst = out + n * (HC + 4 * HP + HZ);
  for (int i = threadIdx.x; i < HC; i += blockDim.x) dst[i] = __float2bfloat16(o[n * HC + i]);
  const Frame f = load_frame(rot, is_quat, trans, n);
  for (int i = threadIdx.x; i < HP; i += blockDim.x) {
    const float* p = o_pt + (n * HP + i) * 3;
    const float x = p[0] - f.t[0], y = p[1] - f.t[1], z = p[2] - f.t[2];
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float v = f.r[0][k] * x + f.r[1][k] * y + f.r[2][k] * z;
      dst[HC + k * HP + i] = __float2bfloat16(v);
      s += v * v;
    }
    dst[HC + 3 * HP + i] = __float2bfloat16(sqrtf(s + eps));
  }
  for (int i = threadIdx.x; i < HZ; i += blockDim.x) dst[HC + 4 * HP + i] = __float2bfloat16(o_pair[n * HZ + i]);
}

}  // namespace ffb

using namespace ffb;

extern "C" {

// Queries, keys, values and points of the core from the layer's bf16 projections and the frames (IpaPrepArgs).
int ffb_ipa_prep(const void* q, const void* kv, const void* q_pts, const void* kv_pts, const float* rot, int is_quat, const float* trans, float* oq,
                 float* ok, float* ov, float* oq_pts, float* ok_pts, float* ov_pts, int N, int H, int C, int Pq, int Pv, void* stream) {
  if (N <= 0 || H <= 0 || C <= 0 || Pq <= 0 || Pv <= 0) return -2;
  IpaPrepArgs a = {(const bf16*)q, (const bf16*)kv, (const bf16*)q_pts, (const bf16*)kv_pts, rot, trans, is_quat, oq, ok, ov, oq_pts, ok_pts, ov_pts,
                   N, H, C, Pq, Pv};
  launch_light(ipa_prep_kernel, N, 256, 0, reinterpret_cast<cudaStream_t>(stream), a);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// The core's outputs in the local frames, with the point norms, as the bf16 input of the output projection.
int ffb_ipa_cat(const float* o, const float* o_pt, const float* o_pair, const float* rot, int is_quat, const float* trans, void* out, int N, int H,
                int C, int Pv, int CZ, float eps, void* stream) {
  if (N <= 0) return -2;
  launch_light(ipa_cat_kernel, N, 256, 0, reinterpret_cast<cudaStream_t>(stream), o, o_pt, o_pair, rot, is_quat, trans, (bf16*)out, H, C, Pv, CZ, eps);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// All pointers are device memory; q / k / v / points / weights / outputs fp32, z bf16 (layouts in IpaArgs).
// Supported configuration: H = 12 heads, C = 16 channels, 4 query / key points, 8 value points, c_z = 128 (AlphaFold's
// structure module); anything else returns -2 and the caller uses its PyTorch composite.
// ..._mixed: wb, bb, gamma and mask in fp32 or, as `bf` says (IpaBf16), in bf16.
int ffb_ipa_fwd_mixed(const float* q, const float* k, const float* v, const float* q_pts, const float* k_pts, const float* v_pts, const void* z,
                      const void* wb, const void* bb, const void* gamma, const void* mask, int bf, float* o, float* o_pt, float* o_pair, int N, int H,
                      int C, int Pq, int Pv, int CZ, int row0, int rows, float w_c, float w_b, float inf, void* stream) {
  if (H != 12 || C != 16 || Pq != 4 || Pv != 8 || CZ != 128) return -2;
  if (rows <= 0) return 0;
  if (N <= 0 || row0 < 0 || row0 + rows > N || (reinterpret_cast<uintptr_t>(z) & 15) || (reinterpret_cast<uintptr_t>(k) & 15) ||
      (reinterpret_cast<uintptr_t>(k_pts) & 15) || (reinterpret_cast<uintptr_t>(o_pair) & 7))
    return -3;
  IpaArgs a;
  a.q = q; a.k = k; a.v = v; a.q_pts = q_pts; a.k_pts = k_pts; a.v_pts = v_pts;
  a.z = reinterpret_cast<const bf16*>(z);
  a.wb = wb; a.bb = bb; a.gamma = gamma; a.mask = mask;
  a.o = o; a.o_pt = o_pt; a.o_pair = o_pair;
  a.N = N; a.H = H; a.C = C; a.Pq = Pq; a.Pv = Pv; a.CZ = CZ; a.row0 = row0; a.rows = rows;
  a.w_c = w_c; a.w_b = w_b; a.inf = inf;
  a.bf = bf;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return ipa_launch<4>(a, st);
}

int ffb_ipa_fwd(const float* q, const float* k, const float* v, const float* q_pts, const float* k_pts, const float* v_pts, const void* z,
                const float* wb, const float* bb, const float* gamma, const float* mask, float* o, float* o_pt, float* o_pair, int N, int H,
                int C, int Pq, int Pv, int CZ, int row0, int rows, float w_c, float w_b, float inf, void* stream) {
  return ffb_ipa_fwd_mixed(q, k, v, q_pts, k_pts, v_pts, z, wb, bb, gamma, mask, 0, o, o_pt, o_pair, N, H, C, Pq, Pv, CZ, row0, rows, w_c, w_b, inf, stream);
}

}  // extern "C"
