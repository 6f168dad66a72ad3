// FP32 products on the tensor cores (included by tc_kernels.cu): every FP32 operand is cut into three
// BF16 parts whose sum is the operand (exactly above 2^-110: below, the last parts fall under BF16's smallest
// numbers; each part the nearest BF16 of what is left), and a product is the six BF16 products of parts whose weights are at least 2^-16 of the first one's:
//   x y = x0 y0 + (x0 y1 + x1 y0) + (x1 y1 + x0 y2 + x2 y0) + terms of either sign below 2^-23 x y
// The tensor cores add in FP32 but do not round to nearest, so no long sum is left to them: an
// accumulator in TMEM holds 64 of K (the five small products first, then the four K16 steps of
// x0 y0), FP32 adds in registers sum the chunks, and what the sums are low by on the mean is put back
// (kSpLow).  Measured against FP64 the factors are as near
// as with the FP32 FMA products this replaces (the tests hold them to the same bounds), at
// 6 / 1900 of a flop's time instead of 1 / 80.
//
// One kernel, five modes, all over 128-row tiles and 64-wide chunks of K:
//   kSpEuclid    slots of  V' W (H-step) or V H' (W-step):  A = the V chunk, cut by sixteen warps on its
//                way from shared memory to TMEM; B = the other factor's chunk (three BF16 copies)
//   kSpKl        slots of  W'(V ./ (WH + eps)): a first product forms S = the chunk of W H in TMEM,
//                and A = V / (S + eps) (- 1 for the additive rule), cut the same way; W H is not stored
//   kSpKlQuality the same H-step, which also sums the quality of the factors it starts from
//   kSpQuality   sum V log10(WH + eps) - WH;  kSpResidual  sum (V - WH)^2 and sum V^2
// V is read as it is (FP32, column-major, both half-steps from the one copy): along K it is
// contiguous for the H-step (rows u) and strided for the W-step (rows i); both arrive by TMA.
// What bounds it: V's 4 bytes an element from HBM (39.5 us at 8192 x 8192) against
// 24 MMAs of 128 x npad x 16 a chunk (21.6 us there at r = 64, 43 us at r = 128).  Measured there:
// kSpEuclid 53 us at r = 64 (the FP32 FMA product: 233), 48 at r = 16; kSpKl 98 at r = 64 and 154 at
// r = 128, bound by one chunk's chain product -> TMEM load -> quotient -> cut -> TMEM store -> product
// (the tensor pipe is busy 43-47%); kSpQuality 86 (was ~370), bound by log10 on the FP32 lanes.

enum SpMode { kSpEuclid = 0, kSpKl = 1, kSpKlQuality = 2, kSpQuality = 3, kSpResidual = 4 };

constexpr int kSpChunk = 64;                       // K per chunk
constexpr int kSpVBytes = kTileM * kSpChunk * 4;   // 32 KB of V a chunk
constexpr int kSpFPart = kSpChunk * 128;           // one part of a 64-column box of the factor chunk: 8 KB
constexpr int kSpFBox = 3 * kSpFPart;
constexpr int kSpWorkers = 16;                     // warps that cut, drain and reduce
constexpr int kSpThreads = 64 + 32 * kSpWorkers + 64;  // + loads, MMA issue, two warps for the Gram / the sums
constexpr int kSpMaxRank = 128;
constexpr int kSpMaxSV = 4, kSpMaxSF = 4;
constexpr int kSpBarBytes = 1024;

struct SpParams {
    int ctas;                    // CTAs that share the chunks; any more of the grid only finish the Gram / the sums
    int tiles, kchunks, kvalid;  // row tiles, 64-wide chunks of K, K itself
    int npad, nbox, max_seg;     // rank rounded up to 16; 64-column boxes of it
    int k_contig;                // V's chunk is contiguous along K (H-step), else along its rows (W-step)
    int sv, sf;                  // ring stages
    float *partials;
    // what the slots' rows are low by (sp_check): [slot][quarter][row], the quarters' sums over a row
    const float *row_sums;       // the other factor's, [K rounded up to 64]
    float2 *checks;
    int *err;
    long long wait_limit;
    // Gram of the other factor from the update kernel's partials, as in tc_gemm_sk_kernel (Euclid)
    const float *gram_partials;
    float *gram_out;
    int gram_count, gram_entries;
    // first product (the other modes): rows of the factor along the tile, [part][row][npad]
    const __nv_bfloat16 *A1;
    long long a1_part;
    int a1_rows;
    float eps;
    int minus_one;
    const float *W, *H;          // the FP32 factors, of n rows and rank r, for plain_wh
    int n, r;
    const float *sum_partials;   // KL: [count][npad] partial sums of the other factor
    float *sum_out;              // [npad]
    int sum_count;
    double *reduce;              // quality: [grid]; residual: [grid][2]
    int *done;                   // CTAs done (the last one sums the others' partials, and resets it)
    float *qout, *qout_host;     // the quality: a device word and the pinned read-back word (or null)
    double *rout;                // the relative residual
};

// packed FP32: two values an operation
__device__ __forceinline__ unsigned long long bits2(float2 a) {
    unsigned long long d;
    asm("mov.b64 %0, {%1,%2};" : "=l"(d) : "f"(a.x), "f"(a.y));
    return d;
}
__device__ __forceinline__ float2 vals2(unsigned long long d) {
    float2 r;
    asm("mov.b64 {%0,%1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
    return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)), "l"(bits2(c)));
    return vals2(d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)));
    return vals2(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)));
    return vals2(d);
}
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return fma2(b, both(-1.f), a); }

// log10 of two positive normal values: x = 2^e (1 + f) with sqrt(1/2) <= 1 + f < sqrt(2), and
// e log10(2) + f Q(f), Q the least-squares polynomial of degree 9 that a reweighted fit (Lawson) takes
// to the smallest largest relative error, 4e-9.  At most 1.9 units in the last place off over
// 2^-3 .. 2^3 (log10f promises 2), for a third of log10f's operations.  `range` collects the largest
// distance of the values' bits from the smallest normal's: below 0x7F000000 all are normal.
__device__ __forceinline__ float2 log10_pair(float2 x, uint32_t &range) {
    auto split = [&](float v, float &m) {
        const int b = __float_as_int(v);
        range = max(range, (uint32_t)b - 0x00800000u);
        const int e = (b - 0x3F3504F3) >> 23;
        m = __int_as_float(b - (e << 23));
        return __int_as_float(0x4B400000 + e);  // 2^23 * 1.5 + e
    };
    float2 m, e;
    e.x = split(x.x, m.x);
    e.y = split(x.y, m.y);
    e = add2(e, both(-12582912.f));
    const float2 f = add2(m, both(-1.f));
    float2 q = both(-3.309807181e-02f);
    q = fma2(q, f, both(5.604422465e-02f));
    q = fma2(q, f, both(-5.751562491e-02f));
    q = fma2(q, f, both(6.159092858e-02f));
    q = fma2(q, f, both(-7.213202864e-02f));
    q = fma2(q, f, both(8.686744422e-02f));
    q = fma2(q, f, both(-1.085805073e-01f));
    q = fma2(q, f, both(1.447647959e-01f));
    q = fma2(q, f, both(-2.171471864e-01f));
    q = fma2(q, f, both(4.342944920e-01f));
    return fma2(e, both(0.30102999566398120f), mul2(q, f));
}

// cut3 of two finite values, the parts packed: 4.5 operations a value.  (An infinity or NaN
// becomes NaN in the later parts; the callers see to those.)
__device__ __forceinline__ void cut_pair(float x0, float x1, uint32_t &w0, uint32_t &w1, uint32_t &w2) {
    auto pack = [](float2 v) {  // the nearest BF16s, the first in the low half
        const __nv_bfloat162 h = __float22bfloat162_rn(v);
        return *reinterpret_cast<const uint32_t *>(&h);
    };
    auto unpack = [](uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u)); };
    const float2 x = make_float2(x0, x1);
    w0 = pack(x);
    const float2 r = sub2(x, unpack(w0));
    w1 = pack(r);
    w2 = pack(sub2(r, unpack(w1)));
}

// 32 lanes x 32 bit, 8 consecutive columns per thread, from registers.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

__device__ __forceinline__ float max_nan(float a, float b) {
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}

// s + c += x with the rounding error of s kept in c (Knuth's TwoSum), two sums at once: as good as sums
// in FP64 at the FP32 pipe's rate (this GPU's FP64 pipe would take longer over V than reading it does)
__device__ __forceinline__ void two_sum(float2 &s, float2 &c, float2 x) {
    const float2 t = add2(s, x), bb = sub2(t, s);
    c = add2(c, add2(sub2(s, sub2(t, bb)), sub2(x, bb)));
    s = t;
}

// A check sum's share of a thread: its sixteen columns of A, read back from TMEM at `ta` (the parts together are
// what they were cut from), by the other factor's row sums z.  (A function of its own, as sp_sums: few chunks
// come here, and inlined they took registers from every chunk: 16384 x 4096, r = 128, with the sample
// 222 us a product, 204 without checks.)
__device__ __noinline__ float sp_check(uint32_t ta, const float *z) {
    float4 zv[4];
#pragma unroll
    for (int c = 0; c < 4; c++) zv[c] = __ldcg(reinterpret_cast<const float4 *>(z) + c);
    __syncwarp();
    float w[3][8];
#pragma unroll
    for (int h = 0; h < 3; h++) tmem_ld8_sync(ta + (uint32_t)(h * 32), w[h]);
    float2 d = both(0.f);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        auto part = [&](int h) {
            const uint32_t u = __float_as_uint(w[h][c]);
            return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
        };
        const float4 q = zv[c / 2];
        d = fma2(add2(part(0), add2(part(1), part(2))), c % 2 ? make_float2(q.z, q.w) : make_float2(q.x, q.y), d);
    }
    return d.x + d.y;
}

// The sum and the sum of the sizes of `cols` columns of the accumulator (or fewer than one: zeros)
__device__ __noinline__ float2 sp_sums(uint32_t ta, int cols) {
    float2 s = both(0.f), size = both(0.f);
    for (int c = 0; c < cols; c += 8) {
        float v[8];
        tmem_ld8_sync(ta + (uint32_t)c, v);
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
            s = add2(s, make_float2(v[k], v[k + 1]));
            size = add2(size, make_float2(fabsf(v[k]), fabsf(v[k + 1])));
        }
    }
    return make_float2(s.x + s.y, size.x + size.y);
}

// An element of W H by FP32 multiply-adds, where the sum of the parts' products is not finite: an infinity's later
// parts are zero, so beside a zero or an infinity it has become NaN
__device__ __noinline__ float plain_wh(const float *W, int n, const float *H, int r, int i, int u) {
    float s = 0.f;
    for (int a = 0; a < r && s == s; a++) s = fmaf(W[(long long)a * n + i], H[(long long)u * r + a], s);
    return s;
}

// What the update kernel needs of the other factor, from the partials its own update left: this CTA's
// share of the Gram's entries (four lanes an entry) or of the column / row sums (a warp an entry),
// by `nt` threads, in a fixed order whatever the number of threads.
template <int MODE>
__device__ __forceinline__ void sp_finish_other(const SpParams &p, int et, int nt) {
    if constexpr (MODE == kSpEuclid) {
        const long long E = p.gram_entries;
        const long long e0 = (long long)blockIdx.x * E / gridDim.x, e1 = (long long)(blockIdx.x + 1) * E / gridDim.x;
        for (long long eb = e0; eb < e1; eb += nt / 4) {
            const long long e = eb + (et >> 2);
            float s = 0.f;
            if (e < e1) {
                int z = et & 3;
                for (; z + 60 < p.gram_count; z += 64) {
                    float v[16];
#pragma unroll
                    for (int q = 0; q < 16; q++) v[q] = p.gram_partials[(size_t)(z + 4 * q) * E + e];
#pragma unroll
                    for (int q = 0; q < 16; q++) s += v[q];
                }
                for (; z < p.gram_count; z += 4) s += p.gram_partials[(size_t)z * E + e];
            }
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (e < e1 && (et & 3) == 0) p.gram_out[e] = s;
        }
    } else if constexpr (MODE == kSpKl) {
        const int E = p.npad, lane = et & 31;
        const int e0 = (int)((long long)blockIdx.x * E / gridDim.x), e1 = (int)((long long)(blockIdx.x + 1) * E / gridDim.x);
        // (in FP64, at most one entry a CTA: a rounded sum moves its whole row of the factor, and the next
        // iteration moves it again the same way)
        for (int ei = e0 + (et >> 5); ei < e1; ei += nt / 32) {
            double s = 0.0;
            int z = lane;
            for (; z + 7 * 32 < p.sum_count; z += 8 * 32) {
                float v[8];
#pragma unroll
                for (int q = 0; q < 8; q++) v[q] = p.sum_partials[(size_t)(z + q * 32) * E + ei];
#pragma unroll
                for (int q = 0; q < 8; q++) s += v[q];
            }
            for (; z < p.sum_count; z += 32) s += p.sum_partials[(size_t)z * E + ei];
            s = warp_sum(s);
            if (lane == 0) p.sum_out[ei] = (float)s;
        }
    }
}

// NPC: rank class (32, 64, 128), at least npad
template <int NPC, int MODE>
__global__ void __launch_bounds__(NPC == 32 && MODE == kSpEuclid ? 768 : kSpThreads, 1)  // (80 registers: an update CTA fits beside)
    sp_kernel(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmF, SpParams p) {
    constexpr bool kFirst = MODE != kSpEuclid;   // has the first product S
    constexpr bool kKl = MODE == kSpKl || MODE == kSpKlQuality, kSum = MODE >= kSpKlQuality;  // ends in a sum
    constexpr bool kReduce = MODE >= kSpQuality;  // ends in a reduction, has no second product
    constexpr int ND1 = kReduce ? 2 : 1;          // S buffers (64 columns)
    constexpr int NR = kKl && NPC == 128 ? 1 : 2;  // A buffers (3 x 32 columns)
    constexpr int ND2 = NR;                       // accumulators (NPC columns)
    const uintptr_t base = (reinterpret_cast<uintptr_t>(tc_dyn_smem) + 1023) & ~uintptr_t(1023);
    const int fBytes = p.nbox * kSpFBox;
    unsigned char *sFr = reinterpret_cast<unsigned char *>(base);
    unsigned char *sVr = sFr + p.sf * fBytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sVr + p.sv * kSpVBytes);
    uint64_t *vfull = bars, *vempty = vfull + kSpMaxSV;
    uint64_t *ffull = vempty + kSpMaxSV, *fempty = ffull + kSpMaxSF;
    uint64_t *rfull = fempty + kSpMaxSF, *rempty = rfull + 2;
    uint64_t *d2full = rempty + 2, *d2empty = d2full + 2;
    uint64_t *d1full = d2empty + 2, *d1empty = d1full + 2;
    uint64_t *a1full = d1empty + 2, *a1empty = a1full + 1, *mdone = a1empty + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mdone + 1);
    double *red = reinterpret_cast<double *>(mdone + 2);  // [2][16]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long T = (long long)p.tiles * p.kchunks;
    if (!kReduce && (int)blockIdx.x >= p.ctas) {
        griddep_wait();
        griddep_launch_dependents();
        sp_finish_other<kKl ? kSpKl : MODE>(p, threadIdx.x, kSpThreads);
        return;
    }
    const long long lo = (long long)blockIdx.x * T / p.ctas;
    const long long hi = (long long)(blockIdx.x + 1) * T / p.ctas;
    const int nblk = (int)(hi - lo);
    const int kc0 = (int)(lo % p.kchunks), t0 = (int)(lo / p.kchunks);

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.sv; s++) {
            mbar_init(&vfull[s], 1);
            mbar_init(&vempty[s], kSpWorkers);
        }
        for (int s = 0; s < p.sf; s++) {
            mbar_init(&ffull[s], 1);
            mbar_init(&fempty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&rfull[b], kSpWorkers);
            mbar_init(&rempty[b], 1);
            mbar_init(&d2full[b], 1);
            mbar_init(&d2empty[b], kSpWorkers);
            mbar_init(&d1full[b], 1);
            mbar_init(&d1empty[b], kSpWorkers);
        }
        mbar_init(a1full, kSpWorkers);
        mbar_init(a1empty, 1);
        mbar_init(mdone, 1);
        fence_mbar_init();
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmF);
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    constexpr uint32_t kA1Cols = kFirst ? 3 * NPC / 2 : 0;
    const uint32_t tA1 = tmem, tD1 = tmem + kA1Cols, tR = tD1 + (kFirst ? ND1 * 64 : 0), tD2 = tR + NR * 96;

    if (warp == 0) {
        if (lane == 0 && nblk > 0) {
            const uint64_t vpol = l2_policy_evict_first();  // V is read once per launch
            int vj = 0, vs = 0, vt = t0, vk = kc0, fj = 0, fs = 0, fk = kc0;
            uint32_t vph = 0, fph = 0, par_v = 0, par_f = 0;
            auto load_v = [&] {
                mbar_arrive_expect_tx(&vfull[vs], (uint32_t)kSpVBytes);
                unsigned char *dst = sVr + vs * kSpVBytes;
                if (p.k_contig) {  // rows u: two 128-byte swizzled boxes of 32 along K
                    tma_load_2d_hint(dst, &tmV, vk * kSpChunk, vt * kTileM, &vfull[vs], vpol);
                    tma_load_2d_hint(dst + kSpVBytes / 2, &tmV, vk * kSpChunk + 32, vt * kTileM, &vfull[vs], vpol);
                } else {           // rows i: one box, 128 rows contiguous at each of the 64 K
                    tma_load_2d_hint(dst, &tmV, vt * kTileM, vk * kSpChunk, &vfull[vs], vpol);
                }
                par_v = (par_v & ~(1u << vs)) | (vph << vs);
                ring_next(vs, vph, p.sv);
                if (++vk == p.kchunks) {
                    vk = 0;
                    vt++;
                }
                vj++;
            };
            // V is no kernel's output: the first stages are requested before the wait
            while (vj < nblk && vj < p.sv) load_v();
            griddep_wait();
            griddep_launch_dependents();
            long long t_start = 0;
            int idle = 0;
            while (vj < nblk || fj < nblk) {
                bool moved = false;
                if (fj < nblk && (fj < p.sf || mbar_test(&fempty[fs], fph ^ 1))) {
                    mbar_arrive_expect_tx(&ffull[fs], (uint32_t)fBytes);
                    for (int q = 0; q < p.nbox; q++)
                        tma_load_3d(sFr + fs * fBytes + q * kSpFBox, &tmF, q * 64, fk * kSpChunk, 0, &ffull[fs]);
                    par_f = (par_f & ~(1u << fs)) | (fph << fs);
                    ring_next(fs, fph, p.sf);
                    if (++fk == p.kchunks) fk = 0;
                    fj++;
                    moved = true;
                }
                if (vj < nblk && mbar_test(&vempty[vs], vph ^ 1)) {
                    load_v();
                    moved = true;
                }
                if (moved) {
                    idle = 0;
                    t_start = 0;
                } else if ((++idle & 63) == 0) {
                    if (*((volatile int *)p.err) != 0) break;
                    const long long now = clock64();
                    if (t_start == 0) {
                        t_start = now;
                    } else if (now - t_start > p.wait_limit) {
                        atomicOr(p.err, kErrWaitEmpty);
                        break;
                    }
                }
            }
            // no copy of this CTA may still be landing when it exits
            for (int s = 0; s < p.sv && s < vj; s++) mbar_wait_quiet(&vfull[s], par_v >> s & 1);
            for (int s = 0; s < p.sf && s < fj; s++) mbar_wait_quiet(&ffull[s], par_f >> s & 1);
        } else {
            griddep_wait();
            griddep_launch_dependents();
        }
    } else if (warp == 1) {
        griddep_wait();
        griddep_launch_dependents();
        // The whole warp runs the loop, one elected lane issues: descriptors and addresses stay
        // uniform, and an MMA costs a few instructions (with one lane in the loop the issue took
        // 120 cycles an MMA, twice what the MMA takes).
        const bool leader = elect_one();
        auto wait = [&](uint64_t *bar, uint32_t parity, int bit) {
            return __all_sync(0xffffffffu, mbar_wait(bar, parity, p.err, bit, p.wait_limit)) != 0;
        };
        const uint32_t id1 = idesc_bf16_f32(kTileM, kSpChunk);
        const uint32_t id2 = idesc_bf16_f32(kTileM, p.npad) | kIdescBMnMajor;
        // descriptors of the factor ring's first stage: K-major for S, MN-major for the second product
        // (its 64-column boxes lie kSpFBox apart); a stage, part or K step moves the start address
        const uint64_t fdk = smem_desc(smem_u32(sFr), 16, 1024, 2), fdm = smem_desc(smem_u32(sFr), kSpFBox, 1024, 2);
        const uint32_t fstep = (uint32_t)fBytes >> 4, a1w = (uint32_t)p.npad / 2;
        const int nk = p.npad / 16;
        // parts in the order of their products' weights, the smallest first
        constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
        int f1 = 0, d1 = 0, seg1 = 0, kk1 = kc0;
        uint32_t f1ph = 0, d1ph = 0;
        bool new1 = true;
        // S of the next chunk; A1 is the tile's rows of the other side's factor
        auto first = [&]() -> bool {
            if (new1 && !wait(a1full, (uint32_t)(seg1 & 1), kErrWaitFull)) return false;
            new1 = false;
            if (!wait(&ffull[f1], f1ph, kErrWaitFull) || !wait(&d1empty[d1], d1ph ^ 1, kErrWaitTmemEmpty)) return false;
            const bool tile_end = ++kk1 == p.kchunks;
            if (leader) {
                tc_fence_after();
                const uint64_t fb = fdk + (uint64_t)(f1 * fstep);
                const uint32_t dd = tD1 + (uint32_t)(d1 * 64);
#pragma unroll
                for (int q = 0; q < 6; q++)
#pragma unroll
                    for (int k = 0; k < NPC / 16; k++)
                        if (k < nk)
                            tc_mma_f16_ts(dd, tA1 + pa[q] * a1w + (uint32_t)(k * 8),
                                          fb + (uint64_t)(((k >> 2) * kSpFBox + pb[q] * kSpFPart + (k & 3) * 32) >> 4), id1,
                                          q + k > 0 ? 1u : 0u);
                tc_commit(&d1full[d1]);
                if constexpr (kReduce) tc_commit(&fempty[f1]);
                if (tile_end) tc_commit(a1empty);  // A1 is free once the tile's last S is done
            }
            __syncwarp();
            ring_next(f1, f1ph, p.sf);
            ring_next(d1, d1ph, ND1);
            if (tile_end) {
                kk1 = 0;
                seg1++;
                new1 = true;
            }
            return true;
        };
        if constexpr (kReduce) {
            for (int j = 0; j < nblk; j++)
                if (!first()) break;
        } else {
            int f2 = 0, rb = 0, db = 0;
            uint32_t f2ph = 0, rph = 0, dph = 0;
            bool ok = true;
            if constexpr (kFirst) ok = nblk == 0 || first();
            for (int j = 0; j < nblk && ok; j++) {
                if constexpr (kFirst) {
                    if (j + 1 < nblk && !first()) break;
                }
                if (!wait(&ffull[f2], f2ph, kErrWaitFull) || !wait(&d2empty[db], dph ^ 1, kErrWaitTmemEmpty) ||
                    !wait(&rfull[rb], rph, kErrWaitTmemFull))
                    break;
                if (leader) {
                    tc_fence_after();
                    const uint64_t fb = fdm + (uint64_t)(f2 * fstep);
                    const uint32_t ra = tR + (uint32_t)(rb * 96), dd = tD2 + (uint32_t)(db * NPC);
#pragma unroll
                    for (int q = 0; q < 6; q++)
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            tc_mma_f16_ts(dd, ra + (uint32_t)(pa[q] * 32 + k * 8),
                                          fb + (uint64_t)((pb[q] * kSpFPart + k * 2048) >> 4), id2, q + k > 0 ? 1u : 0u);
                    tc_commit(&fempty[f2]);
                    tc_commit(&rempty[rb]);
                    tc_commit(&d2full[db]);
                }
                __syncwarp();
                ring_next(f2, f2ph, p.sf);
                ring_next(rb, rph, NR);
                ring_next(db, dph, ND2);
            }
        }
        if (leader) {
            tc_commit(mdone);
            mbar_wait_quiet(mdone, 0);
        }
        __syncwarp();
    } else if (warp < 2 + kSpWorkers) {
        // sixteen workers: a quarter of the rows (their TMEM lanes) by a quarter of the chunk's K for
        // cutting or reducing, by a quarter of the rank for draining.  A chunk is cut while the
        // product of the one before runs, which is drained next.  (V is no kernel's output: without a
        // first product the first chunk is cut before the wait.)  (Two groups of eight that take
        // chunks in turn, for the reductions, measured the same: their arithmetic bounds them.)
        if constexpr (kFirst) {
            griddep_wait();
            griddep_launch_dependents();
        }
        constexpr int NC = NPC / 4;  // columns a thread sums
        const int quarter = warp & 3, part = (warp - 2) >> 2;
        const int row = quarter * 32 + lane, c0 = part * NC;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        int vs = 0, rb = 0, d1 = 0, db = 0, kk = kc0, t = t0, seg = 0, dk = kc0, dseg = 0;
        uint32_t vph = 0, rph = 0, d1ph = 0, dph = 0;
        float2 qs = both(0.f), qc = qs, ws = qs, wc = qs;  // two-term sums
        double far_a = 0.0, far_b = 0.0;  // the residual's sums of what FP32 squares do not hold
        float acc[kReduce ? 1 : NC];
        if constexpr (!kReduce) {
#pragma unroll
            for (int c = 0; c < NC; c++) acc[c] = 0.f;
        }
        // forms those of the columns h .. h + 7 of S again that are not finite, within the first `lim` columns
        auto repair = [&](float (&s)[16], int h, int lim) {
            bool odd = false;
#pragma unroll
            for (int c = 0; c < 8; c++) odd |= !(fabsf(s[h + c]) < kInf) && h + c < lim;
            if (!__any_sync(0xffffffffu, odd)) return;
            float again[8];
#pragma unroll
            for (int c = 0; c < 8; c++) again[c] = s[h + c];
#pragma unroll 1
            for (int c = 0; c < 8; c++) {
                const int k = kk * kSpChunk + part * 16 + h + c, g = t * kTileM + row;
                if (!(fabsf(again[c]) < kInf) && h + c < lim)
                    again[c] = plain_wh(p.W, p.n, p.H, p.r, p.k_contig ? k : g, p.k_contig ? g : k);
            }
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 8; c++) s[h + c] = again[c];
        };
        // the quality's terms of sixteen columns
        auto sample = [&](const float (&v)[16], float (&s)[16], int klim) {
            if constexpr (MODE == kSpQuality || MODE == kSpKlQuality) {
                uint32_t range = 0;
                float2 l[8];
#pragma unroll
                for (int c = 0; c < 8; c++)
                    l[c] = log10_pair(add2(make_float2(s[2 * c], s[2 * c + 1]), both(p.eps)), range);
                if (!__any_sync(0xffffffffu, klim < 16 || range >= 0x7F000000u)) {
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        const float2 s2 = make_float2(s[2 * c], s[2 * c + 1]);
                        two_sum(qs, qc, sub2(mul2(make_float2(v[2 * c], v[2 * c + 1]), l[c]), s2));
                    }
                } else {  // the edge of V, or a sum that is zero, subnormal, infinite or NaN
                    repair(s, 0, klim);
                    repair(s, 8, klim);
#pragma unroll
                    for (int c = 0; c < 16; c++)
                        if (c < klim)
                            two_sum(qs, qc, make_float2(v[c] * log10f(s[c] + p.eps) - s[c], 0.f));
                }
                __syncwarp();
            }
        };
        // Check sums (kSpLow): in the first and every 32nd of this CTA's chunks, sum_k A(row, k) sum_a F(k, a) by FP32
        // multiply-adds, against the sum over a of what the tensor cores make of it.  A thread has a quarter of
        // either.
        float zsum = 0.f, low = 0.f, size = 0.f;
        auto checked = [](int j) { return (j & 31) == 0; };
        // adds the oldest undrained chunk's product; the last chunk of a segment completes a slot
        auto drain = [&](int j, bool last) -> bool {
            if constexpr (!kReduce) {
                if (!mbar_wait(&d2full[db], dph, p.err, kErrWaitTmemFull, p.wait_limit)) return false;
                tc_fence_after();
                constexpr int LD = NC < 16 ? NC : 16;
#pragma unroll
                for (int g = 0; g < NC / LD; g++)
                    if (c0 + g * LD < p.npad) {
                        float v[LD];
                        if constexpr (LD == 8) tmem_ld8_sync(tD2 + lane_off + (uint32_t)(db * NPC + c0 + g * LD), v);
                        else tmem_ld16_sync(tD2 + lane_off + (uint32_t)(db * NPC + c0 + g * LD), v);
#pragma unroll
                        for (int c = 0; c < LD; c++) acc[g * LD + c] += v[c];
                    }
                if (checked(j)) {
                    const float2 sum = sp_sums(tD2 + lane_off + (uint32_t)(db * NPC + c0), min(NC, p.npad - c0));
                    low += zsum - sum.x;
                    size += sum.y;
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&d2empty[db]);
                ring_next(db, dph, ND2);
                if (++dk == p.kchunks || last) {
                    p.checks[((size_t)(blockIdx.x * p.max_seg + dseg) * 4 + part) * kTileM + row] = make_float2(low, size);
                    low = size = 0.f;
                    float *dst = p.partials + ((size_t)(blockIdx.x * p.max_seg + dseg) * kTileM + row) * p.npad + c0;
#pragma unroll
                    for (int g = 0; g < NC / 4; g++)
                        if (c0 + g * 4 < p.npad) {
                            *reinterpret_cast<float4 *>(dst + 4 * g) =
                                make_float4(acc[4 * g], acc[4 * g + 1], acc[4 * g + 2], acc[4 * g + 3]);
                            acc[4 * g] = acc[4 * g + 1] = acc[4 * g + 2] = acc[4 * g + 3] = 0.f;
                        }
                    dk = 0;
                    dseg++;
                }
            }
            return true;
        };
        bool new1 = kFirst;
        for (int j = 0; j < nblk; j++) {
            if constexpr (kFirst) {
                if (new1) {
                    // the tile's factor rows into TMEM, once the previous tile's products are done
                    if (seg > 0 && !mbar_wait(a1empty, (uint32_t)((seg - 1) & 1), p.err, kErrWaitTmemEmpty, p.wait_limit))
                        break;
                    tc_fence_after();
                    const int grow = t * kTileM + row;
                    const int nw = p.npad / 8;  // 4-word groups (8 values) of a row
                    for (int q = 0; q < 3; q++)
                        for (int g = part; g < nw; g += 4) {
                            uint4 w = make_uint4(0, 0, 0, 0);
                            if (grow < p.a1_rows)
                                w = __ldcg(reinterpret_cast<const uint4 *>(p.A1 + q * p.a1_part + (long long)grow * p.npad) + g);
                            __syncwarp();
                            asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(
                                             tA1 + lane_off + (uint32_t)(q * (p.npad / 2) + g * 4)),
                                         "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w)
                                         : "memory");
                        }
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(a1full);
                    new1 = false;
                }
            }
            if (!mbar_wait(&vfull[vs], vph, p.err, kErrWaitFull, p.wait_limit)) break;
            const uint32_t vt = smem_u32(sVr + vs * kSpVBytes);
            // K left from this warp's first column (a reduction counts no row beyond the last either)
            const int klim = kReduce && t * kTileM + row >= p.a1_rows ? 0 : p.kvalid - kk * kSpChunk - part * 16;
            float v[16], s[16];
            if (p.k_contig) {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float4 x = lds128_stage(vt + (part >> 1) * (kSpVBytes / 2) + sw128(row, (part & 1) * 4 + c));
                    v[4 * c] = x.x; v[4 * c + 1] = x.y; v[4 * c + 2] = x.z; v[4 * c + 3] = x.w;
                }
            } else {
#pragma unroll
                for (int c = 0; c < 16; c++) v[c] = lds32_stage(vt + (part * 16 + c) * 512 + row * 4);
            }
            if constexpr (kFirst) {
                if (!mbar_wait(&d1full[d1], d1ph, p.err, kErrWaitTmemFull, p.wait_limit)) break;
                tc_fence_after();
                __syncwarp();
                tmem_ld16_sync(tD1 + lane_off + (uint32_t)(d1 * 64 + part * 16), s);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&d1empty[d1]);
                ring_next(d1, d1ph, ND1);
            }
            uint32_t w0[8], w1[8], w2[8];  // the chunk's three parts, packed in pairs
            if constexpr (MODE == kSpEuclid) {
                // (V is finite, or the update kernel forms the sums again)
#pragma unroll
                for (int c = 0; c < 8; c++) cut_pair(v[2 * c], v[2 * c + 1], w0[c], w1[c], w2[c]);
            } else if constexpr (kKl) {
                // V / (S + eps): the quotient by the approximate reciprocal and one residual step
                // (Markstein), which a division in range rounds like the operator but for rare last
                // bits, without its branch; a warp with any other division takes the operator
                const float less = p.minus_one ? 1.f : 0.f;
#pragma unroll
                for (int h = 0; h < 16; h += 8) {
                    float q[8], dmax = 0.f;
                    bool fine = true;
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        const float d = s[h + c] + p.eps, y = rcp_approx(d), a = v[h + c] * y;
                        q[c] = fmaf(fmaf(-a, d, v[h + c]), y, a);
                        dmax = fmaxf(dmax, fabsf(d));
                        fine = fine && fabsf(q[c]) < 1e38f;
                    }
                    if (__any_sync(0xffffffffu, !fine || dmax > 8e37f || h + 8 > klim)) {
                        const int lim = t * kTileM + row < p.a1_rows ? klim : 0;
                        repair(s, h, lim);
#pragma unroll
                        for (int c = 0; c < 8; c += 2) {  // beyond V: 0 (not 0 / eps)
                            const float x = h + c < lim ? v[h + c] / (s[h + c] + p.eps) - less : 0.f;
                            const float y = h + c + 1 < lim ? v[h + c + 1] / (s[h + c + 1] + p.eps) - less : 0.f;
                            uint32_t a[3], b[3];
                            cut3(x, a[0], a[1], a[2]);
                            cut3(y, b[0], b[1], b[2]);
                            w0[(h + c) / 2] = pack_top(a[0], b[0]);
                            w1[(h + c) / 2] = pack_top(a[1], b[1]);
                            w2[(h + c) / 2] = pack_top(a[2], b[2]);
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < 8; c += 2)
                            cut_pair(q[c] - less, q[c + 1] - less, w0[(h + c) / 2], w1[(h + c) / 2], w2[(h + c) / 2]);
                    }
                    __syncwarp();
                }
            } else if constexpr (MODE == kSpQuality) {
                sample(v, s, klim);
            } else {
                // (v - s)^2 and v^2 with what FP32 drops of them (zeros beyond the last row and K).  Where the
                // squares leave FP32's range (a value above 2^50, an infinity, or all of the sixteen below
                // 2^-40) they are formed in FP64.
                if (klim < 16) {
#pragma unroll
                    for (int c = 0; c < 16; c++)
                        if (c >= klim) v[c] = s[c] = 0.f;
                }
                float most = 0.f;  // (NaN if any is)
#pragma unroll
                for (int c = 0; c < 16; c++) most = max_nan(most, max_nan(fabsf(v[c]), fabsf(s[c])));
                if (__any_sync(0xffffffffu, most != 0.f && !(most >= 0x1p-40f && most <= 0x1p50f))) {
                    repair(s, 0, klim);
                    repair(s, 8, klim);
                    if (!(most >= 0x1p-40f && most <= 0x1p50f)) {
#pragma unroll
                        for (int c = 0; c < 16; c++) {
                            const double d = (double)v[c] - (double)s[c];
                            far_a += d * d;
                            far_b += (double)v[c] * (double)v[c];
                            v[c] = s[c] = 0.f;
                        }
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int c = 0; c < 16; c += 2) {
                    const float2 x = make_float2(v[c], v[c + 1]), y = make_float2(s[c], s[c + 1]);
                    const float2 d = sub2(x, y), bb = sub2(d, x);
                    const float2 e = sub2(sub2(x, sub2(d, bb)), add2(y, bb));
                    const float2 dd = mul2(d, d), vv = mul2(x, x);
                    two_sum(qs, qc, dd);
                    qc = add2(qc, fma2(add2(d, d), e, fma2(d, d, mul2(dd, both(-1.f)))));
                    two_sum(ws, wc, vv);
                    wc = add2(wc, fma2(x, x, mul2(vv, both(-1.f))));
                }
            }
            if constexpr (!kReduce) {
                // a division that takes its slow path leaves lanes apart, and tcgen05.st wants them
                // together: all words are made before the lanes meet, none after
#pragma unroll
                for (int c = 0; c < 8; c++) asm volatile("" : "+r"(w0[c]), "+r"(w1[c]), "+r"(w2[c])::"memory");
                if (!mbar_wait(&rempty[rb], rph ^ 1, p.err, kErrWaitTmemEmpty, p.wait_limit)) break;
                tc_fence_after();
                __syncwarp();
                const uint32_t ra = tR + lane_off + (uint32_t)(rb * 96 + part * 8);
                tmem_st8(ra, w0);
                tmem_st8(ra + 32, w1);
                tmem_st8(ra + 64, w2);
                tmem_st_wait();
                tc_fence_before();
            }
            // The V stage goes back only here, when what was read of it has been used: given back right
            // after the loads it could be refilled before they were done, where a tcgen05.st held
            // them up (seen at the first chunk of a tile).
            if constexpr (kReduce)
                asm volatile("" : "+f"(qs.x), "+f"(qs.y), "+f"(qc.x), "+f"(qc.y), "+f"(ws.x), "+f"(ws.y)::"memory");
            __syncwarp();
            if (lane == 0) {
                if constexpr (!kReduce) mbar_arrive(&rfull[rb]);
                mbar_arrive(&vempty[vs]);
            }
            // (the sample comes behind the chain: the second product has its operand)
            if constexpr (MODE == kSpKlQuality) sample(v, s, t * kTileM + row < p.a1_rows ? klim : 0);
            if (!kFirst && j == 0) {
                griddep_wait();
                griddep_launch_dependents();
            }
            if constexpr (!kReduce)
                if (checked(j))
                    zsum = sp_check(tR + lane_off + (uint32_t)(rb * 96 + part * 8), p.row_sums + kk * kSpChunk + part * 16);
            ring_next(vs, vph, p.sv);
            ring_next(rb, rph, NR);
            if (++kk == p.kchunks) {
                kk = 0;
                t++;
                seg++;
                new1 = kFirst;
            }
            if (j > 0 && !drain(j - 1, false)) break;
            if (j + 1 == nblk) drain(j, true);
        }
        if constexpr (kSum) {
            // (beside an infinite sum its second term is NaN)
            auto total = [](float2 s, float2 c) {
                return (double)s.x + (fabsf(s.x) < kInf ? (double)c.x : 0.0) + ((double)s.y + (fabsf(s.y) < kInf ? (double)c.y : 0.0));
            };
            double a = total(qs, qc), b = total(ws, wc);
            if (MODE == kSpResidual) {
                a += far_a;
                b += far_b;
            }
            a = warp_sum(a);
            if (MODE == kSpResidual) b = warp_sum(b);
            if (lane == 0) {
                red[warp - 2] = a;
                red[16 + warp - 2] = b;
            }
        }
    } else {
        // two more warps finish what the update kernel needs of the other factor
        griddep_wait();
        griddep_launch_dependents();
        sp_finish_other<kKl ? kSpKl : MODE>(p, threadIdx.x - (kSpThreads - 64), 64);
    }
    __syncthreads();
    if constexpr (kSum) {
        if (threadIdx.x == 0) {
            double a = 0.0, b = 0.0;
            for (int w = 0; w < 16; w++) {
                a += red[w];
                b += red[16 + w];
            }
            constexpr int kTerms = MODE == kSpResidual ? 2 : 1;
            p.reduce[kTerms * blockIdx.x] = a;
            if constexpr (kTerms == 2) p.reduce[kTerms * blockIdx.x + 1] = b;
            reinterpret_cast<volatile int *>(red)[0] = atom_acq_rel_add(p.done, 1) == p.ctas - 1;
        }
        __syncthreads();
        if (warp == 0 && reinterpret_cast<volatile int *>(red)[0]) {
            // the last CTA: the partials in CTA order (lane-strided, then a fixed tree)
            constexpr int kTerms = MODE == kSpResidual ? 2 : 1;
            double a = 0.0, b = 0.0;
            for (int c = lane; c < p.ctas; c += 32) {
                a += __ldcg(p.reduce + kTerms * c);
                if constexpr (kTerms == 2) b += __ldcg(p.reduce + kTerms * c + 1);
            }
            a = warp_sum(a);
            if constexpr (kTerms == 2) b = warp_sum(b);
            if (lane == 0) {
                if constexpr (kTerms == 2) {
                    p.rout[0] = relative_residual(a, b);
                } else {
                    p.qout[0] = (float)a;
                    if (p.qout_host) {
                        p.qout_host[0] = (float)a;
                        __threadfence_system();
                    }
                }
                *p.done = 0;
            }
        }
    }
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// Both factors (W n x r, H r x m) as three BF16 parts, row-major: [part][row][npad], zero beyond r
__global__ void sp_cut_factors_kernel(const float *__restrict__ W, int n, const float *__restrict__ H, int m, int r,
                                      __nv_bfloat16 *__restrict__ Ws, __nv_bfloat16 *__restrict__ Hs, int npad) {
    const int is_w = blockIdx.y == 0, rows = is_w ? n : m;
    __nv_bfloat16 *const out = is_w ? Ws : Hs;
    const long long total = (long long)rows * npad;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < total;
         k += (long long)gridDim.x * blockDim.x) {
        const long long c = k / npad, a = k % npad;
        store_cut(out + k, total, a < r ? (is_w ? W[a * rows + c] : H[c * r + a]) : 0.f);
    }
}

// V (n x m) with its columns ld apart
__global__ void sp_pad_columns_kernel(const float *__restrict__ V, int n, int m, float *__restrict__ out, long long ld) {
    for (long long u = blockIdx.y; u < m; u += gridDim.y)
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            out[u * ld + i] = V[u * n + i];
}

// ------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------
struct SpGemm {
    CUtensorMap tmV, tmF;
    SpParams p;
    int grid = 0, smem = 0;
    int *slot_ptr = nullptr, *slot_list = nullptr, *tile_slots = nullptr;
};

}  // namespace gpunmf

// State of a job's FP32 products on the tensor cores; a BF16 job has one for its residual only.
struct SpState {
    int npad = 16, npc = 32, max_ctas = 0;
    __nv_bfloat16 *Ws = nullptr, *Hs = nullptr;  // the factors' three parts, row-major
    float *Vp = nullptr;                         // V with its column stride rounded up to 16 bytes (n % 4 != 0)
    float *P_h = nullptr, *P_w = nullptr;        // partial products (slots)
    float *G_w = nullptr, *G_h = nullptr, *GP_w = nullptr, *GP_h = nullptr;  // Euclid: Grams and their partials
    float *S_w = nullptr, *S_h = nullptr, *SP_w = nullptr, *SP_h = nullptr;  // KL: sums and their partials
    float *Z_w = nullptr, *Z_h = nullptr;        // the factors' row sums
    float2 *C_w = nullptr, *C_h = nullptr;       // the slots' checks
    double *reduce = nullptr;
    int *err = nullptr, *done = nullptr;
    bool sample = false;        // the next KL H-step sums the quality
    char *arena = nullptr;      // all of the above: one allocation
    gpunmf::SpGemm gh, gw, gq;  // H-step, W-step, quality / residual
};

namespace gpunmf {

// The rank class of the kernel.
static int sp_class(int npad) { return npad <= 32 ? 32 : npad <= 64 ? 64 : 128; }

bool sp_supported(int n, int m, int r) { return r <= kSpMaxRank && n > 0 && m > 0; }

// CTAs of a product: stream-K over all SMs, but where that would cut a tile into more pieces than
// the update kernels read at once (few tiles; the KL update's slot table holds kSlotW), a whole number of CTAs
// per tile, at most kSlotW of them.
static int sp_grid(int tiles, int kchunks, int max_ctas) {
    const long long T = (long long)tiles * kchunks;
    if (max_ctas / tiles + 2 > kSlotW)
        return tiles * std::max(1, std::min(std::min(kSlotW, kchunks), max_ctas / tiles));
    return (int)std::min<long long>(max_ctas, T);
}

// The tensor cores cut off, not round: the sum after every step of 16 to 24 bits, and every product two bits
// below the last one of the step's largest (a model of such an adder gives the measured errors).  On positive data a sum
// comes out low, by 0.7 to 1.3 units of 2^-24 where its terms are alike and by up to 3.6 where they span many powers of
// two.  The scale between W(:, a) and H(a, :) is free, so what one half-step's numerators are low by and the
// other's are not adds up from iteration to iteration.  So every CTA measures it, on the data: its first and
// every 32nd chunk have check sums (sp_check, sp_sums), and the update kernels add the fraction found to a row's
// numerators, at the one rounding that they have anyway.  Rows without a checked chunk, batches, and S (whose
// fraction is the same in both half-steps) take what was found on the mean, the table: measured against FP64 over
// uniform, low-rank and count data, which differ by a third either way.
// After 100 iterations of 42 generated jobs (64 .. 2048 rows and columns, ranks 8 .. 64) the factors are 1.0e-6 off (rms;
// largest 1.7e-6), as with FP32 multiply-adds (1.0e-6, 1.6e-6); with every second chunk scaled by 1 + 2^-23, so that sums
// of few chunks got up to twice their share, 2.0e-6 and 4.5e-6.  With W spread over twenty-five powers of two, 0.4e-6
// .. 4.9e-6 (multiply-adds 0.4e-6 .. 2.2e-6; the table alone 9e-6).  The price: 8192 x 8192 a product of 55.2 us
// for 53.5 (r = 64), 75.6 for 74.6 (r = 128); an iteration of 1024 x 512, r = 16, 15.5 us for 14.5; a KL half-step of 361 x 472,
// r = 49, 4.9 us for 4.3.  Checks in a CTA's last chunk and at every tile's start, behind the drain of the chunk before,
// measured the same there and slower at rank 128 (80.5 us a product).
constexpr float kSpLow[9] = {0.f, 0.70f, 0.82f, 0.95f, 1.10f, 1.57f, 1.78f, 2.06f, 2.34f};
static float sp_low(int steps) { return kSpLow[steps] * 0x1p-24f; }
// a numerator's fraction: its chunks of 64 (and a last one of fewer) weighted by their share of K
static float sp_low_sum(int K) {
    const int full = K / kSpChunk * kSpChunk, rest = K - full;
    return (full * sp_low(kSpChunk / 16) + rest * sp_low(ceil_div(rest, 16))) / K;
}

// Hands out the pieces of a job's one allocation (256-byte aligned); without a base it only adds up.
struct SpArena {
    char *base = nullptr;
    size_t used = 0;
    template <class T>
    void get(T **p, size_t count) {
        if (base) *p = reinterpret_cast<T *>(base + used);
        used += (count * sizeof(T) + 255) / 256 * 256;
    }
};

// Slot tables of one product: per tile its slots in K order, as lists and as rows of kSlotW
struct SpTables {
    std::vector<int> ints;  // [tiles + 1] starts, the lists, and where every list is short enough the rows
    int tiles = 0, count = 0, ctas = 0, max_seg = 1;
    bool rows = false;
};

static SpTables sp_tables(int rows, int K, int max_ctas) {
    SpTables t;
    const int kchunks = ceil_div(K, kSpChunk);
    t.tiles = ceil_div(rows, kTileM);
    t.ctas = sp_grid(t.tiles, kchunks, max_ctas);
    std::vector<int> list;
    schedule(t.tiles, kchunks, t.ctas, &t.max_seg, t.ints, list);
    t.count = (int)list.size();
    t.rows = true;
    for (int k = 0; k < t.tiles; k++) t.rows = t.rows && t.ints[k + 1] - t.ints[k] <= kSlotW;
    std::vector<int> table;
    if (t.rows) {
        table.assign((size_t)t.tiles * kSlotW, -1);
        for (int k = 0; k < t.tiles; k++)
            for (int q = t.ints[k]; q < t.ints[k + 1]; q++) table[(size_t)k * kSlotW + (q - t.ints[k])] = list[q];
    }
    while ((t.ints.size() + list.size()) % 4) list.push_back(-1);  // the rows are read 16 bytes at a time
    // (kSlotW is a multiple of 4, so the next product's table starts aligned as well)
    t.ints.insert(t.ints.end(), list.begin(), list.end());
    t.ints.insert(t.ints.end(), table.begin(), table.end());
    return t;
}

static size_t padded_rows(int rows) { return (size_t)ceil_div(rows, kSpChunk) * kSpChunk; }

// Lays a job's pieces out in `a`; th, tw: the products' tables (null for a residual alone).
static void sp_layout(SpState *t, SpArena &a, int rule, int n, int m, int npad, int max_ctas, const SpTables *th,
                      const SpTables *tw, int **ints) {
    const size_t np = npad;
    const long long ldv = (n + 3) / 4 * 4;
    a.get(&t->Ws, 3 * (size_t)n * np);
    a.get(&t->Hs, 3 * (size_t)m * np);
    if (ldv != n) a.get(&t->Vp, (size_t)ldv * m);
    a.get(&t->reduce, 2 * (size_t)max_ctas);
    a.get(&t->err, 2);
    if (!th) return;
    if (rule_is_kl(rule)) {
        a.get(&t->S_w, np);
        a.get(&t->S_h, np);
        a.get(&t->SP_w, np * ceil_div(n, kKlUpdColsW));
        a.get(&t->SP_h, np * ceil_div(m, kKlUpdColsH));
    } else {
        a.get(&t->G_w, np * np);
        a.get(&t->G_h, np * np);
        a.get(&t->GP_w, np * np * ceil_div(n, upd_rows(n, npad)));
        a.get(&t->GP_h, np * np * ceil_div(m, upd_rows(m, npad)));
    }
    a.get(&t->P_h, (size_t)th->ctas * th->max_seg * kTileM * np);
    a.get(&t->P_w, (size_t)tw->ctas * tw->max_seg * kTileM * np);
    a.get(&t->C_h, (size_t)th->ctas * th->max_seg * 4 * kTileM);
    a.get(&t->C_w, (size_t)tw->ctas * tw->max_seg * 4 * kTileM);
    a.get(&t->Z_w, padded_rows(n));
    a.get(&t->Z_h, padded_rows(m));
    a.get(ints, th->ints.size() + tw->ints.size() + 4);
}

size_t sp_footprint(int rule, int n, int m, int r, bool residual_only) {
    SpState t;
    SpArena a;
    int *ints = nullptr;
    if (residual_only) {
        sp_layout(&t, a, rule, n, m, npad_of(r), kNumSMsGB300, nullptr, nullptr, &ints);
    } else {
        const SpTables th = sp_tables(m, n, kNumSMsGB300), tw = sp_tables(n, m, kNumSMsGB300);
        sp_layout(&t, a, rule, n, m, npad_of(r), kNumSMsGB300, &th, &tw, &ints);
    }
    return a.used;
}

// V (n x m FP32, column stride ld): boxes of 32 rows i x 128 columns u, 128-byte swizzled (K along i),
// or of 128 rows x 64 columns (K along u).  L2 sectors promoted to 128 bytes: 256 made batches, whose
// columns start anywhere, read 583 MB for 448 of V (342 us an iteration of 768 uneven ones, 331 so)
static gpunmf_status sp_map_v(CUtensorMap *mp, const float *V, uint64_t n, uint64_t m, uint64_t ld, bool k_contig) {
    auto fn = encode_fn();
    cuuint64_t dims[2] = {n, m};
    cuuint64_t strides[1] = {ld * 4};
    cuuint32_t box[2] = {k_contig ? 32u : (cuuint32_t)kTileM, k_contig ? (cuuint32_t)kTileM : (cuuint32_t)kSpChunk};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn ? fn(mp, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(V), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE,
                         k_contig ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                    : CUDA_ERROR_NOT_SUPPORTED;
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled (FP32 V) failed (%d)", (int)r);
        return GPUNMF_ERR_CUDA;
    }
    return GPUNMF_OK;
}

// A factor's three parts ([part][rows][npad] BF16): boxes of 64 columns x 64 rows x 3 parts
static gpunmf_status sp_map_f(CUtensorMap *mp, const __nv_bfloat16 *F, uint64_t rows, uint64_t npad) {
    auto fn = encode_fn();
    cuuint64_t dims[3] = {npad, rows, 3};
    cuuint64_t strides[2] = {npad * 2, rows * npad * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)kSpChunk, 3};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn ? fn(mp, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16 *>(F), dims, strides, box,
                         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                    : CUDA_ERROR_NOT_SUPPORTED;
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled (factor parts) failed (%d)", (int)r);
        return GPUNMF_ERR_CUDA;
    }
    return GPUNMF_OK;
}

template <int NPC>
static cudaError_t sp_set_smem(int optin) {
    cudaError_t e = cudaFuncSetAttribute(sp_kernel<NPC, kSpEuclid>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sp_kernel<NPC, kSpKl>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sp_kernel<NPC, kSpKlQuality>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sp_kernel<NPC, kSpQuality>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sp_kernel<NPC, kSpResidual>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    return e;
}

static cudaError_t sp_set_smem_once() {
    static OncePerDevice<cudaError_t> once;
    int dev = 0;
    cudaGetDevice(&dev);
    return once.run(dev, [] {
        const int optin = smem_optin();
        cudaError_t result = sp_set_smem<32>(optin);
        if (result == cudaSuccess) result = sp_set_smem<64>(optin);
        if (result == cudaSuccess) result = sp_set_smem<128>(optin);
        return result;
    });
}

template <int MODE>
static cudaError_t sp_launch(const SpState *t, const SpGemm &g, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g.grid);
    cfg.blockDim = dim3(kSpThreads);
    cfg.dynamicSmemBytes = g.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    switch (t->npc) {
        case 32: return cudaLaunchKernelEx(&cfg, sp_kernel<32, MODE>, g.tmV, g.tmF, g.p);
        case 64: return cudaLaunchKernelEx(&cfg, sp_kernel<64, MODE>, g.tmV, g.tmF, g.p);
        default: return cudaLaunchKernelEx(&cfg, sp_kernel<128, MODE>, g.tmV, g.tmF, g.p);
    }
}

// shape, rings and, with `tb` (its tables, on the device at `ints`), the slots of one product (rows x K)
static void sp_setup(gpunmf_job *j, SpGemm &g, int rows, int K, bool k_contig, const SpTables *tb, int *ints,
                     float *slots) {
    SpState *t = j->sp;
    SpParams &p = g.p;
    p = SpParams{};
    p.tiles = ceil_div(rows, kTileM);
    p.kchunks = ceil_div(K, kSpChunk);
    p.kvalid = K;
    p.npad = t->npad;
    p.nbox = (t->npad + 63) / 64;
    p.k_contig = k_contig;
    // a factor stage is held from its load to the end of its second product, a V stage only until it is
    // cut: four stages of the factor and of V where they fit (rank <= 64), else three and two (KL at
    // 16384 x 4096, r = 128: two and four took 181 us a launch, three and two 154)
    p.sf = p.nbox == 1 ? 4 : 3;
    p.sv = p.nbox == 1 ? 4 : 2;
    p.err = t->err;
    p.wait_limit = kWaitLimitCycles;
    p.eps = j->eps;
    p.minus_one = rule_is_additive(j->rule);
    p.W = j->W; p.H = j->H; p.n = j->n; p.r = j->r;
    g.smem = 1024 + p.sf * p.nbox * kSpFBox + p.sv * kSpVBytes + kSpBarBytes;
    p.ctas = g.grid = (int)std::min<long long>(t->max_ctas, (long long)p.tiles * p.kchunks);
    if (!tb) return;
    p.ctas = tb->ctas;
    p.max_seg = tb->max_seg;
    p.partials = slots;
    g.grid = t->max_ctas;  // those without chunks finish the Gram / the sums
    g.slot_ptr = ints;
    g.slot_list = ints + tb->tiles + 1;
    if (tb->rows) g.tile_slots = ints + (tb->ints.size() - (size_t)tb->tiles * kSlotW);
}

gpunmf_status sp_create(gpunmf_job *j, bool residual_only) {
    SpState *t = new (std::nothrow) SpState();
    if (!t) return GPUNMF_ERR_NOMEM;
    j->sp = t;
    const int n = j->n, m = j->m, r = j->r;
    const bool kl = rule_is_kl(j->rule);
    t->npad = npad_of(r);
    t->npc = sp_class(t->npad);
    t->max_ctas = num_sms();
    const size_t np = t->npad;
    const long long ldv = (n + 3) / 4 * 4;
    SpTables th, tw;
    if (!residual_only) {
        th = sp_tables(m, n, t->max_ctas);
        tw = sp_tables(n, m, t->max_ctas);
    }
    SpArena a;
    int *ints = nullptr;
    auto lay = [&] {
        a.used = 0;
        sp_layout(t, a, j->rule, n, m, t->npad, t->max_ctas, residual_only ? nullptr : &th, residual_only ? nullptr : &tw,
                  &ints);
    };
    lay();
    cudaError_t e = job_dev_alloc(j, (void **)&t->arena, a.used);
    if (e == cudaSuccess) {
        a.base = t->arena;
        lay();
        e = cudaMemsetAsync(t->err, 0, 2 * sizeof(int), j->stream);
        t->done = t->err + 1;
    }
    if (e == cudaSuccess && !residual_only)  // (beyond the last row they stay zero)
        e = cudaMemsetAsync(t->Z_w, 0, reinterpret_cast<char *>(t->Z_h + padded_rows(m)) - reinterpret_cast<char *>(t->Z_w), j->stream);
    if (e == cudaSuccess && !residual_only) {
        std::vector<int> both(th.ints);
        both.insert(both.end(), tw.ints.begin(), tw.ints.end());
        e = job_h2d(j, ints, both.data(), both.size() * sizeof(int));
    }
    if (e == cudaSuccess) e = sp_set_smem_once();
    if (e == cudaSuccess && !residual_only && !kl) e = set_update_smem(t->npad);
    if (e != cudaSuccess) {
        set_error("FP32 tensor-core workspace: %s", cudaGetErrorString(e));
        cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? GPUNMF_ERR_NOMEM : GPUNMF_ERR_CUDA;
    }
    if (!residual_only) {
        sp_setup(j, t->gh, m, n, true, &th, ints, t->P_h);
        sp_setup(j, t->gw, n, m, false, &tw, ints + th.ints.size(), t->P_w);
    }
    sp_setup(j, t->gq, m, n, true, nullptr, nullptr, nullptr);
    const float *V = t->Vp ? t->Vp : j->V;
    gpunmf_status st = sp_map_v(&t->gq.tmV, V, n, m, ldv, true);
    if (st == GPUNMF_OK) st = sp_map_f(&t->gq.tmF, t->Ws, n, np);
    t->gq.p.A1 = t->Hs; t->gq.p.a1_part = (long long)m * np; t->gq.p.a1_rows = m;
    t->gq.p.reduce = t->reduce; t->gq.p.done = t->done;
    t->gq.p.qout = j->d_quality;
    void *dp = nullptr;  // the pinned read-back word, where the device can write it
    if (cudaHostGetDevicePointer(&dp, j->h_quality(), 0) == cudaSuccess) t->gq.p.qout_host = static_cast<float *>(dp);
    else cudaGetLastError();
    if (residual_only || st != GPUNMF_OK) return st;
    // H-step: rows u, K = i; W-step: rows i, K = u
    t->gh.tmV = t->gq.tmV;
    t->gh.tmF = t->gq.tmF;
    t->gh.p.A1 = t->Hs; t->gh.p.a1_part = (long long)m * np; t->gh.p.a1_rows = m;
    st = sp_map_v(&t->gw.tmV, V, n, m, ldv, false);
    if (st == GPUNMF_OK) st = sp_map_f(&t->gw.tmF, t->Hs, m, np);
    t->gw.p.A1 = t->Ws; t->gw.p.a1_part = (long long)n * np; t->gw.p.a1_rows = n;
    t->gh.p.row_sums = t->Z_w; t->gh.p.checks = t->C_h;
    t->gw.p.row_sums = t->Z_h; t->gw.p.checks = t->C_w;
    t->gh.p.reduce = t->reduce; t->gh.p.done = t->done;
    t->gh.p.qout = t->gq.p.qout; t->gh.p.qout_host = t->gq.p.qout_host;
    if (kl) {
        t->gh.p.sum_partials = t->SP_w; t->gh.p.sum_out = t->S_w; t->gh.p.sum_count = ceil_div(n, kKlUpdColsW);
        t->gw.p.sum_partials = t->SP_h; t->gw.p.sum_out = t->S_h; t->gw.p.sum_count = ceil_div(m, kKlUpdColsH);
    } else {
        t->gh.p.gram_partials = t->GP_w; t->gh.p.gram_out = t->G_w; t->gh.p.gram_count = ceil_div(n, upd_rows(n, t->npad));
        t->gw.p.gram_partials = t->GP_h; t->gw.p.gram_out = t->G_h; t->gw.p.gram_count = ceil_div(m, upd_rows(m, t->npad));
        t->gh.p.gram_entries = t->gw.p.gram_entries = (int)(np * np);
    }
    return st;
}

static cudaError_t sp_update(gpunmf_job *j, bool is_w, int update) {
    SpState *t = j->sp;
    const SpGemm &g = is_w ? t->gw : t->gh;
    const int rows = is_w ? j->n : j->m;
    if (rule_is_kl(j->rule)) {
        KlUpdParams u{};
        u.X = is_w ? j->W : j->H; u.Xr = is_w ? t->Ws : t->Hs; u.ldr = t->npad; u.part = (long long)rows * t->npad;
        u.ldx = j->n; u.sums = is_w ? t->S_h : t->S_w; u.P = is_w ? t->P_w : t->P_h;
        u.slot_ptr = g.slot_ptr; u.slot_list = g.slot_list; u.tile_slots = g.tile_slots;
        u.sum_partials = is_w ? t->SP_w : t->SP_h;
        u.r = j->r; u.cols = rows; u.npad = t->npad; u.eps = j->eps; u.update = update;
        u.additive = rule_is_additive(j->rule) ? 2 : 0;  // 2: the - 1 is in the numerator already
        u.V = j->V; u.W = j->W; u.H = j->H; u.n = j->n; u.m = j->m;
        u.checks = is_w ? t->C_w : t->C_h; u.row_sums = is_w ? t->Z_w : t->Z_h;
        u.low = sp_low_sum(is_w ? j->m : j->n); u.s_low = sp_low(t->npad / 16);
        return launch_kl_update(u, t->npad, is_w, j->stream);
    }
    UpdParams u{};
    u.X = is_w ? j->W : j->H; u.Xs = is_w ? t->Ws : t->Hs; u.part = (long long)rows * t->npad;
    u.ldx = j->n; u.G = is_w ? t->G_h : t->G_w; u.P = is_w ? t->P_w : t->P_h;
    u.slot_ptr = g.slot_ptr; u.slot_list = g.slot_list; u.is_w = is_w;
    u.gram_partials = is_w ? t->GP_w : t->GP_h;
    u.r = j->r; u.cols = rows; u.npad = t->npad; u.eps = j->eps; u.update = update;
    u.additive = rule_is_additive(j->rule);
    u.V = j->V; u.ldv = j->n; u.F = is_w ? j->H : j->W; u.K = is_w ? j->m : j->n;
    u.checks = is_w ? t->C_w : t->C_h; u.row_sums = is_w ? t->Z_w : t->Z_h;
    u.low = sp_low_sum(u.K);
    return launch_update(u, t->npad, j->stream);
}

static cudaError_t sp_cut_factors(gpunmf_job *j) {
    SpState *t = j->sp;
    const long long most = (long long)std::max(j->n, j->m) * t->npad;
    sp_cut_factors_kernel<<<dim3(std::min(2 * t->max_ctas, ceil_div(most, 256)), 2), 256, 0, j->stream>>>(
        j->W, j->n, j->H, j->m, j->r, t->Ws, t->Hs, t->npad);
    return cudaGetLastError();
}

// What an FP32 job keeps beside its factors, made of them: the parts of both, and the row sums and Gram / sum partials
// of W (of H too for the rule that keeps it).
gpunmf_status sp_refresh(gpunmf_job *j) {
    GPUNMF_CUDA_TRY(sp_cut_factors(j));
    GPUNMF_CUDA_TRY(sp_update(j, true, 0));
    if (j->rule == GPUNMF_ADDITIVE_EUCLIDEAN_FIXED_H) GPUNMF_CUDA_TRY(sp_update(j, false, 0));
    return GPUNMF_OK;
}

gpunmf_status sp_prepare(gpunmf_job *j, bool residual_only) {
    SpState *t = j->sp;
    if (t->Vp) {
        sp_pad_columns_kernel<<<dim3(std::min(ceil_div(j->n, 256), 8), std::min(j->m, 65535)), 256, 0, j->stream>>>(
            j->V, j->n, j->m, t->Vp, (j->n + 3) / 4 * 4);
        GPUNMF_CUDA_TRY(cudaGetLastError());
    }
    return residual_only ? GPUNMF_OK : sp_refresh(j);
}

bool sp_quality_writes_host(const gpunmf_job *j) { return j->sp->gq.p.qout_host != nullptr; }

// KL jobs: the next H-step takes the sample (it records the job's quality event)
bool sp_quality_fold(gpunmf_job *j) {
    j->sp->sample = rule_is_kl(j->rule);
    return j->sp->sample;
}

gpunmf_status sp_iterate(gpunmf_job *j, bool updateW) {
    SpState *t = j->sp;
    const bool kl = rule_is_kl(j->rule);
    gpunmf_status st = job_quality_step(j, true);
    if (st != GPUNMF_OK) return st;
    for (int w = 0; w < 2; w++) {
        if (w ? !updateW : j->rule == GPUNMF_ADDITIVE_EUCLIDEAN_FIXED_H) continue;
        const SpGemm &g = w ? t->gw : t->gh;
        mark_begin(j);
        const bool sample = w == 0 && t->sample;  // a KL H-step
        GPUNMF_CUDA_TRY(!kl      ? sp_launch<kSpEuclid>(t, g, j->stream)
                        : sample ? sp_launch<kSpKlQuality>(t, g, j->stream)
                                 : sp_launch<kSpKl>(t, g, j->stream));
        mark_end(j);
        if (sample) {
            t->sample = false;
            gpunmf_status q = job_quality_sampled(j, sp_quality_writes_host(j));
            if (q != GPUNMF_OK) return q;
        }
        GPUNMF_CUDA_TRY(sp_update(j, w != 0, 1));
        j->launches += 2;
    }
    return GPUNMF_OK;
}

// The quality of the current factors into j->d_quality, and the pinned read-back word.
gpunmf_status sp_quality(gpunmf_job *j) {
    GPUNMF_CUDA_TRY(sp_launch<kSpQuality>(j->sp, j->sp->gq, j->stream));
    j->launches += 1;
    return GPUNMF_OK;
}

// The relative residual of the current factors into *d_out.
gpunmf_status sp_residual(gpunmf_job *j, double *d_out) {
    SpState *t = j->sp;
    if (j->precision == GPUNMF_BF16) GPUNMF_CUDA_TRY(sp_cut_factors(j));  // its iterations keep no parts
    t->gq.p.rout = d_out;
    GPUNMF_CUDA_TRY(sp_launch<kSpResidual>(t, t->gq, j->stream));
    return GPUNMF_OK;
}

void sp_destroy(gpunmf_job *j) {
    SpState *t = j->sp;
    if (!t) return;
    job_dev_free(j, t->arena);
    delete t;
    j->sp = nullptr;
}
