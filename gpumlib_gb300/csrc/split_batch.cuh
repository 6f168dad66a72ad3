// Batches of small Euclidean factorisations by the FP32 products on the tensor cores (included by
// tc_kernels.cu after split_f32.cuh): every half-step of all instances is two launches, the product and
// the update, so its 128-row tiles share the SMs whichever instance they belong to.
//
// The product is kSpEuclid's pipeline over one list of tiles: every CTA takes an equal share of all
// tiles' 64-wide chunks of K (stream-K across instances); a segment's sum is a slot, and the slots are
// numbered in chunk order, so a tile's are consecutive.  Ranks up to 32.  The update takes 64 rows of an
// instance to a CTA; two warps of the product's CTAs sum the Grams from the 64-row partials meanwhile.
// What bounds it: V from HBM at every half-step, once it is larger than L2.
//
// The kernel of batch.cu, which keeps an instance on one CTA, reads V from L2 and needs no launch between
// half-steps: it is the better one for few or very small instances (spb_better).

struct SpbInst {
    int n, m, r, npad;
    long long ldv;                          // column stride of V
    float low_h, low_w;                     // what the numerators are low by (sp_low_sum)
    const float *V;
    float *W, *H;
    __nv_bfloat16 *Ws, *Hs;                 // three parts, [part][row][npad]
    float *GP_w, *GP_h, *G_w, *G_h;         // Gram partials of 64 rows, their sums
};
struct SpbTile {
    int inst, row, kchunks, npad;           // row: the tile's number in its instance
};
struct SpbBlock {
    int inst, row0, slot0, slots;
};
struct SpbParams {
    const SpbInst *insts;
    int count;
    const CUtensorMap *mapV, *mapF;         // per instance
    const SpbTile *tiles;
    const int2 *cta_first;                  // per CTA: its first tile and that tile's first chunk; then a sentinel
    const int *cta_slot;                    // per CTA: its first slot
    long long chunks;
    float *partials;
    int *err;
    long long wait_limit;
};
struct SpbUpdParams {
    const SpbInst *insts;
    const SpbBlock *blocks;
    const float *P;
    float eps;
    int is_w, update;
};

constexpr int kSpbNP = 32;                  // rank class, and a slot's columns
constexpr int kSpbStages = 4;
constexpr int kSpbThreads = 64 + 32 * kSpWorkers + 64;  // loads, MMA issue, workers, two warps for the Grams
constexpr int kSpbSmem = 1024 + kSpbStages * (kSpFBox + kSpVBytes) + kSpBarBytes;
constexpr int kSpbRows = 64, kSpbUpdThreads = 256;  // rows of an update block, its threads

// walks a CTA's tiles chunk by chunk
struct SpbCursor {
    const SpbTile *tiles;
    int t, k;
    SpbTile cur;
    __device__ __forceinline__ SpbCursor(const SpbParams &p, int2 first) : tiles(p.tiles), t(first.x), k(first.y) { load(); }
    __device__ __forceinline__ void load() {
        const int4 v = __ldg(reinterpret_cast<const int4 *>(tiles) + t);
        cur = SpbTile{v.x, v.y, v.z, v.w};
    }
    // to the next chunk; true at a tile's end (the list ends with a tile of its own, never used)
    __device__ __forceinline__ bool next() {
        if (++k < cur.kchunks) return false;
        k = 0;
        t++;
        load();
        return true;
    }
};

template <bool K_CONTIG>
__global__ void __launch_bounds__(kSpbThreads, 1) spb_kernel(SpbParams p) {
    const uintptr_t base = (reinterpret_cast<uintptr_t>(tc_dyn_smem) + 1023) & ~uintptr_t(1023);
    unsigned char *sFr = reinterpret_cast<unsigned char *>(base);
    unsigned char *sVr = sFr + kSpbStages * kSpFBox;
    uint64_t *vfull = reinterpret_cast<uint64_t *>(sVr + kSpbStages * kSpVBytes);
    uint64_t *vempty = vfull + kSpbStages, *ffull = vempty + kSpbStages, *fempty = ffull + kSpbStages;
    uint64_t *rfull = fempty + kSpbStages, *rempty = rfull + 2, *d2full = rempty + 2, *d2empty = d2full + 2;
    uint64_t *mdone = d2empty + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mdone + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nblk = (int)((long long)(blockIdx.x + 1) * p.chunks / gridDim.x - (long long)blockIdx.x * p.chunks / gridDim.x);
    const int2 first = p.cta_first[blockIdx.x];

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSpbStages; s++) {
            mbar_init(&vfull[s], 1);
            mbar_init(&vempty[s], kSpWorkers);
            mbar_init(&ffull[s], 1);
            mbar_init(&fempty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&rfull[b], kSpWorkers);
            mbar_init(&rempty[b], 1);
            mbar_init(&d2full[b], 1);
            mbar_init(&d2empty[b], kSpWorkers);
        }
        mbar_init(mdone, 1);
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, 256);  // two A buffers of 3 x 32 columns, two accumulators of 32
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot, tR = tmem, tD2 = tmem + 192;

    if (warp == 0) {
        if (lane == 0 && nblk > 0) {
            const uint64_t vpol = l2_policy_evict_first();
            SpbCursor cv(p, first), cf(p, first);
            int vj = 0, vs = 0, fj = 0, fs = 0, vinst = -1, finst = -1;
            uint32_t vph = 0, fph = 0, par_v = 0, par_f = 0;
            auto load_v = [&] {
                mbar_arrive_expect_tx(&vfull[vs], (uint32_t)kSpVBytes);
                unsigned char *dst = sVr + vs * kSpVBytes;
                const CUtensorMap *tm = p.mapV + cv.cur.inst;
                if (cv.cur.inst != vinst) {
                    vinst = cv.cur.inst;
                    tma_acquire_desc(tm);
                }
                if (K_CONTIG) {
                    tma_load_2d_hint(dst, tm, cv.k * kSpChunk, cv.cur.row * kTileM, &vfull[vs], vpol);
                    tma_load_2d_hint(dst + kSpVBytes / 2, tm, cv.k * kSpChunk + 32, cv.cur.row * kTileM, &vfull[vs], vpol);
                } else {
                    tma_load_2d_hint(dst, tm, cv.cur.row * kTileM, cv.k * kSpChunk, &vfull[vs], vpol);
                }
                par_v = (par_v & ~(1u << vs)) | (vph << vs);
                ring_next(vs, vph, kSpbStages);
                vj++;
                if (vj < nblk) cv.next();
            };
            while (vj < nblk && vj < kSpbStages) load_v();  // V is no kernel's output
            griddep_wait();
            griddep_launch_dependents();
            long long t_start = 0;
            int idle = 0;
            while (vj < nblk || fj < nblk) {
                bool moved = false;
                if (fj < nblk && (fj < kSpbStages || mbar_test(&fempty[fs], fph ^ 1))) {
                    mbar_arrive_expect_tx(&ffull[fs], (uint32_t)kSpFBox);
                    if (cf.cur.inst != finst) {
                        finst = cf.cur.inst;
                        tma_acquire_desc(p.mapF + finst);
                    }
                    tma_load_3d(sFr + fs * kSpFBox, p.mapF + finst, 0, cf.k * kSpChunk, 0, &ffull[fs]);
                    par_f = (par_f & ~(1u << fs)) | (fph << fs);
                    ring_next(fs, fph, kSpbStages);
                    fj++;
                    if (fj < nblk) cf.next();
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
            for (int s = 0; s < kSpbStages && s < vj; s++) mbar_wait_quiet(&vfull[s], par_v >> s & 1);
            for (int s = 0; s < kSpbStages && s < fj; s++) mbar_wait_quiet(&ffull[s], par_f >> s & 1);
        } else {
            griddep_wait();
            griddep_launch_dependents();
        }
    } else if (warp == 1) {
        griddep_wait();
        griddep_launch_dependents();
        const bool leader = elect_one();
        auto wait = [&](uint64_t *bar, uint32_t parity, int bit) {
            return __all_sync(0xffffffffu, mbar_wait(bar, parity, p.err, bit, p.wait_limit)) != 0;
        };
        const uint64_t fdm = smem_desc(smem_u32(sFr), kSpFBox, 1024, 2);
        constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
        int f2 = 0, rb = 0, db = 0;
        uint32_t f2ph = 0, rph = 0, dph = 0;
        if (nblk > 0) {
            SpbCursor c(p, first);
            for (int j = 0; j < nblk; j++) {
                if (!wait(&ffull[f2], f2ph, kErrWaitFull) || !wait(&d2empty[db], dph ^ 1, kErrWaitTmemEmpty) ||
                    !wait(&rfull[rb], rph, kErrWaitTmemFull))
                    break;
                if (leader) {
                    tc_fence_after();
                    const uint32_t id2 = idesc_bf16_f32(kTileM, c.cur.npad) | kIdescBMnMajor;
                    const uint64_t fb = fdm + (uint64_t)(f2 * (kSpFBox >> 4));
                    const uint32_t ra = tR + (uint32_t)(rb * 96), dd = tD2 + (uint32_t)(db * kSpbNP);
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
                ring_next(f2, f2ph, kSpbStages);
                ring_next(rb, rph, 2);
                ring_next(db, dph, 2);
                if (j + 1 < nblk) c.next();
            }
        }
        if (leader) {
            tc_commit(mdone);
            mbar_wait_quiet(mdone, 0);
        }
        __syncwarp();
    } else if (warp >= 2 + kSpWorkers) {
        // the other factors' Grams, 256 entries of an instance at a time, their partials in order
        griddep_wait();
        griddep_launch_dependents();
        const int et = threadIdx.x - (kSpbThreads - 64);
        constexpr int U = kSpbNP * kSpbNP / 256;
        for (int i = blockIdx.x; i < p.count * U; i += gridDim.x) {
            const SpbInst &d = p.insts[i / U];
            const int E = d.npad * d.npad, e = i % U * 256 + 4 * et;
            if (e >= E) continue;
            const int parts = ((K_CONTIG ? d.n : d.m) + kSpbRows - 1) / kSpbRows;
            const float *in = (K_CONTIG ? d.GP_w : d.GP_h) + e;
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int z = 0; z < parts; z++) {
                const float4 v = __ldcg(reinterpret_cast<const float4 *>(in + (size_t)z * E));
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
            *reinterpret_cast<float4 *>((K_CONTIG ? d.G_w : d.G_h) + e) = s;
        }
    } else if (nblk > 0) {
        constexpr int NC = kSpbNP / 4;
        const int quarter = warp & 3, part = (warp - 2) >> 2;
        const int row = quarter * 32 + lane, c0 = part * NC;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        int vs = 0, rb = 0, db = 0, slot = p.cta_slot[blockIdx.x];
        uint32_t vph = 0, rph = 0, dph = 0;
        float acc[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) acc[c] = 0.f;
        SpbCursor cd(p, first);
        auto drain = [&](bool last) -> bool {
            if (!mbar_wait(&d2full[db], dph, p.err, kErrWaitTmemFull, p.wait_limit)) return false;
            tc_fence_after();
            const int npad = cd.cur.npad;
            if (c0 < npad) {
                float v[NC];
                tmem_ld8_sync(tD2 + lane_off + (uint32_t)(db * kSpbNP + c0), v);
#pragma unroll
                for (int c = 0; c < NC; c++) acc[c] += v[c];
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&d2empty[db]);
            ring_next(db, dph, 2);
            if (cd.k + 1 == cd.cur.kchunks || last) {
                if (c0 < npad) {
                    float4 *dst = reinterpret_cast<float4 *>(p.partials + (size_t)slot * kTileM * kSpbNP + row * npad + c0);
                    dst[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
                    dst[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
                }
#pragma unroll
                for (int c = 0; c < NC; c++) acc[c] = 0.f;
                slot++;
            }
            if (!last) cd.next();
            return true;
        };
        for (int j = 0; j < nblk; j++) {
            if (!mbar_wait(&vfull[vs], vph, p.err, kErrWaitFull, p.wait_limit)) break;
            const uint32_t vt = smem_u32(sVr + vs * kSpVBytes);
            float v[16];
            if (K_CONTIG) {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float4 x = lds128_stage(vt + (part >> 1) * (kSpVBytes / 2) + sw128(row, (part & 1) * 4 + c));
                    v[4 * c] = x.x; v[4 * c + 1] = x.y; v[4 * c + 2] = x.z; v[4 * c + 3] = x.w;
                }
            } else {
#pragma unroll
                for (int c = 0; c < 16; c++) v[c] = lds32_stage(vt + (part * 16 + c) * 512 + row * 4);
            }
            uint32_t w0[8], w1[8], w2[8];
#pragma unroll
            for (int c = 0; c < 8; c++) cut_pair(v[2 * c], v[2 * c + 1], w0[c], w1[c], w2[c]);
            if (!mbar_wait(&rempty[rb], rph ^ 1, p.err, kErrWaitTmemEmpty, p.wait_limit)) break;
            tc_fence_after();
            __syncwarp();
            const uint32_t ra = tR + lane_off + (uint32_t)(rb * 96 + part * 8);
            tmem_st8(ra, w0);
            tmem_st8(ra + 32, w1);
            tmem_st8(ra + 64, w2);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {  // the V stage goes back when what was read of it has been used (sp_kernel)
                mbar_arrive(&rfull[rb]);
                mbar_arrive(&vempty[vs]);
            }
            ring_next(vs, vph, kSpbStages);
            ring_next(rb, rph, 2);
            if (j == 0) {
                griddep_wait();
                griddep_launch_dependents();
            }
            if (j > 0 && !drain(false)) break;
            if (j + 1 == nblk) drain(true);
        }
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 256);
    }
}

// the update of 64 rows of an instance (or, with update 0, only their Gram partial)
__global__ void __launch_bounds__(kSpbUpdThreads, 4) spb_update_kernel(SpbUpdParams p) {
    extern __shared__ __align__(16) float sm[];
    const int4 bv = __ldg(reinterpret_cast<const int4 *>(p.blocks) + blockIdx.x);
    const SpbBlock b{bv.x, bv.y, bv.z, bv.w};
    const SpbInst d = p.insts[b.inst];
    UpdParams u{};
    u.is_w = p.is_w;
    u.X = p.is_w ? d.W : d.H;
    u.cols = p.is_w ? d.n : d.m;
    u.K = p.is_w ? d.m : d.n;
    u.ldx = d.n;
    u.Xs = p.is_w ? d.Ws : d.Hs;
    u.part = (long long)u.cols * d.npad;
    u.gram_partials = p.is_w ? d.GP_w : d.GP_h;
    u.G = p.is_w ? d.G_h : d.G_w;
    u.P = p.P;
    u.npad = kSpbNP;
    u.slot0 = b.slot0;
    u.slots = b.slots;
    u.r = d.r;
    u.eps = p.eps;
    u.update = p.update;
    u.V = d.V;
    u.ldv = d.ldv;
    u.low = p.is_w ? d.low_w : d.low_h;
    u.F = p.is_w ? d.H : d.W;
    if (d.npad == 16) update_rows<16, kSpbRows, kSpbUpdThreads>(u, b.row0, b.row0 / kSpbRows, sm);
    else update_rows<32, kSpbRows, kSpbUpdThreads>(u, b.row0, b.row0 / kSpbRows, sm);
}

// all instances' factors as three parts (grid: blocks per instance x instances x 2)
__global__ void spb_cut_kernel(const SpbInst *__restrict__ insts) {
    const SpbInst d = insts[blockIdx.y];
    const int is_w = blockIdx.z == 0, rows = is_w ? d.n : d.m;
    __nv_bfloat16 *const out = is_w ? d.Ws : d.Hs;
    const float *const X = is_w ? d.W : d.H;
    const long long total = (long long)rows * d.npad;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < total;
         k += (long long)gridDim.x * blockDim.x) {
        const long long c = k / d.npad, a = k % d.npad;
        store_cut(out + k, total, a < d.r ? (is_w ? X[a * rows + c] : X[c * d.r + a]) : 0.f);
    }
}

// ------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------
}  // namespace gpunmf

struct SpBatch {
    int count = 0, grid_h = 0, grid_w = 0, blocks_h = 0, blocks_w = 0;
    float eps = 0.f;
    char *arena = nullptr;
    gpunmf::SpbInst *insts = nullptr;
    gpunmf::SpbBlock *bl_h = nullptr, *bl_w = nullptr;
    gpunmf::SpbParams h, w;
    float *P = nullptr;
    int *err = nullptr;
};

namespace gpunmf {

// one half-step's tiles, CTA shares and update blocks (of rows x K per instance)
struct SpbPlan {
    std::vector<SpbTile> tiles;
    std::vector<SpbBlock> blocks;
    std::vector<int2> first;
    std::vector<int> slot;
    long long chunks = 0;
    int slots = 0, grid = 0;
};

static SpbPlan spb_plan(const std::vector<SpbShape> &shapes, bool w_step, int max_ctas) {
    SpbPlan q;
    std::vector<long long> start;
    for (size_t i = 0; i < shapes.size(); i++) {
        const int rows = w_step ? shapes[i].n : shapes[i].m, K = w_step ? shapes[i].m : shapes[i].n;
        const int kc = ceil_div(K, kSpChunk);
        for (int t = 0; t < ceil_div(rows, kTileM); t++) {
            start.push_back(q.chunks);
            q.tiles.push_back(SpbTile{(int)i, t, kc, npad_of(shapes[i].r)});
            q.chunks += kc;
        }
    }
    start.push_back(q.chunks);
    q.grid = (int)std::min<long long>(max_ctas, q.chunks);
    std::vector<int> tile_slot(q.tiles.size(), -1), tile_slots(q.tiles.size(), 0);
    size_t t = 0;
    for (int c = 0; c < q.grid; c++) {
        const long long lo = c * q.chunks / q.grid, hi = (c + 1) * q.chunks / q.grid;
        while (start[t + 1] <= lo) t++;
        q.first.push_back(make_int2((int)t, (int)(lo - start[t])));
        q.slot.push_back(q.slots);
        for (size_t k = t; k < q.tiles.size() && start[k] < hi; k++) {
            if (tile_slot[k] < 0) tile_slot[k] = q.slots;
            tile_slots[k]++;
            q.slots++;
        }
    }
    for (size_t k = 0; k < q.tiles.size(); k++) {
        const SpbShape &s = shapes[q.tiles[k].inst];
        const int rows = w_step ? s.n : s.m;
        for (int r0 = q.tiles[k].row * kTileM; r0 < std::min(rows, (q.tiles[k].row + 1) * kTileM); r0 += kSpbRows)
            q.blocks.push_back(SpbBlock{q.tiles[k].inst, r0, tile_slot[k], tile_slots[k]});
    }
    q.tiles.push_back(SpbTile{0, 0, 1 << 30, 16});  // what the cursors see past the last tile
    return q;
}

// Whether the launches shared by all instances beat one CTA per instance.  An iteration in us, by what was
// measured: a CTA of the one-CTA kernel takes 9 us and does 27 GFLOP/s, so the largest instance or, of
// more than 456, the average load bounds it; here four launches take 12.5 us, a chunk or a tile 0.6 on
// its SM, and 1216 update blocks 9.  Measured on both sides of the line (one CTA / shared launches): one
// 64 x 64, r = 4: 10.3 / 12.2; one 300 x 200, r = 8: 62 / 13.6; 400 of 128 x 100, r = 8: 27.9 / 37.6;
// 100 of them 27.7 / 23.1; 2000 of 100 x 100, r = 8: 118 / 147; 10 of the benchmark's uneven ones 492 / 29,
// 768 of them 1996 / 368, 4096 of them 3226 / 1846.
bool spb_better(const std::vector<SpbShape> &shapes) {
    double most = 0, all = 0, work = 0, blocks = 0;
    for (const SpbShape &s : shapes) {
        const double us = 9.0 + 4.0 * s.n * s.m * (s.r <= 4 ? 4 : s.r <= 8 ? 8 : s.r <= 16 ? 16 : 32) / 27e3;
        most = std::max(most, us);
        all += us;
        const double tn = ceil_div(s.n, kTileM), tm = ceil_div(s.m, kTileM);
        work += tn * (1 + ceil_div(s.m, kSpChunk)) + tm * (1 + ceil_div(s.n, kSpChunk));
        blocks += ceil_div(s.n, kSpbRows) + ceil_div(s.m, kSpbRows);
    }
    const double one = std::max(most, all / (3.0 * kNumSMsGB300));
    const double shared = 12.5 + 0.6 * work / kNumSMsGB300 + 9.0 * blocks / (8.0 * kNumSMsGB300);
    return 1.15 * shared < one;
}

// V of instance i at shapes[i].V (device, columns ldv = n rounded up to 4 apart), W and H its factors.
// Work is enqueued on s; the factors may be filled after this and before spb_reset.
gpunmf_status spb_create(const std::vector<SpbShape> &shapes, float eps, cudaStream_t s, SpBatch **out) {
    *out = nullptr;
    SpBatch *b = new (std::nothrow) SpBatch();
    if (!b) return GPUNMF_ERR_NOMEM;
    const size_t count = shapes.size();
    b->count = (int)count;
    b->eps = eps;
    const SpbPlan ph = spb_plan(shapes, false, num_sms()), pw = spb_plan(shapes, true, num_sms());
    std::vector<SpbInst> insts(count);
    std::vector<CUtensorMap> maps(4 * count);  // V and W's parts (H-step), V and H's parts (W-step)
    CUtensorMap *d_maps = nullptr;
    SpbTile *t_h = nullptr, *t_w = nullptr;
    int2 *f_h = nullptr, *f_w = nullptr;
    int *sl_h = nullptr, *sl_w = nullptr;
    SpArena a;
    auto lay = [&] {
        a.used = 0;
        a.get(&d_maps, maps.size());
        a.get(&b->insts, count);
        a.get(&t_h, ph.tiles.size());
        a.get(&t_w, pw.tiles.size());
        a.get(&f_h, ph.first.size());
        a.get(&f_w, pw.first.size());
        a.get(&sl_h, ph.slot.size());
        a.get(&sl_w, pw.slot.size());
        a.get(&b->bl_h, ph.blocks.size());
        a.get(&b->bl_w, pw.blocks.size());
        a.get(&b->err, 1);
        a.get(&b->P, (size_t)std::max(ph.slots, pw.slots) * kTileM * kSpbNP);
        for (size_t i = 0; i < count; i++) {
            const SpbShape &q = shapes[i];
            SpbInst &d = insts[i];
            const size_t np = npad_of(q.r);
            d.n = q.n; d.m = q.m; d.r = q.r; d.npad = (int)np; d.ldv = (q.n + 3) / 4 * 4;
            d.low_h = sp_low_sum(q.n); d.low_w = sp_low_sum(q.m);
            d.V = q.V; d.W = q.W; d.H = q.H;
            a.get(&d.Ws, 3 * (size_t)q.n * np);
            a.get(&d.Hs, 3 * (size_t)q.m * np);
            a.get(&d.GP_w, np * np * ceil_div(q.n, kSpbRows));
            a.get(&d.GP_h, np * np * ceil_div(q.m, kSpbRows));
            a.get(&d.G_w, np * np);
            a.get(&d.G_h, np * np);
        }
    };
    lay();
    cudaError_t e = cudaMalloc((void **)&b->arena, a.used);
    if (e != cudaSuccess) {
        set_error("batch workspace of %zu bytes: %s", a.used, cudaGetErrorString(e));
        cudaGetLastError();
        delete b;
        return GPUNMF_ERR_NOMEM;
    }
    a.base = b->arena;
    lay();
    gpunmf_status st = GPUNMF_OK;
    for (size_t i = 0; i < count && st == GPUNMF_OK; i++) {
        const SpbInst &d = insts[i];
        st = sp_map_v(&maps[i], d.V, d.n, d.m, d.ldv, true);
        if (st == GPUNMF_OK) st = sp_map_f(&maps[count + i], d.Ws, d.n, d.npad);
        if (st == GPUNMF_OK) st = sp_map_v(&maps[2 * count + i], d.V, d.n, d.m, d.ldv, false);
        if (st == GPUNMF_OK) st = sp_map_f(&maps[3 * count + i], d.Hs, d.m, d.npad);
    }
    auto put = [&](void *dst, const void *src, size_t bytes) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
    };
    put(d_maps, maps.data(), maps.size() * sizeof(CUtensorMap));
    put(b->insts, insts.data(), count * sizeof(SpbInst));
    auto plan = [&](const SpbPlan &q, SpbTile *t, int2 *f, int *sl, SpbBlock *bl, SpbParams &p, const CUtensorMap *mv,
                    const CUtensorMap *mf) {
        put(t, q.tiles.data(), q.tiles.size() * sizeof(SpbTile));
        put(f, q.first.data(), q.first.size() * sizeof(int2));
        put(sl, q.slot.data(), q.slot.size() * sizeof(int));
        put(bl, q.blocks.data(), q.blocks.size() * sizeof(SpbBlock));
        p = SpbParams{b->insts, (int)count, mv, mf, t, f, sl, q.chunks, b->P, b->err, kWaitLimitCycles};
    };
    plan(ph, t_h, f_h, sl_h, b->bl_h, b->h, d_maps, d_maps + count);
    plan(pw, t_w, f_w, sl_w, b->bl_w, b->w, d_maps + 2 * count, d_maps + 3 * count);
    b->grid_h = ph.grid; b->grid_w = pw.grid;
    b->blocks_h = (int)ph.blocks.size(); b->blocks_w = (int)pw.blocks.size();
    if (e == cudaSuccess) e = cudaMemsetAsync(b->err, 0, sizeof(int), s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // the host vectors end here
    if (e == cudaSuccess) e = cudaFuncSetAttribute(spb_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSpbSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(spb_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSpbSmem);
    if (e != cudaSuccess) {
        set_error("batch set-up failed: %s", cudaGetErrorString(e));
        st = GPUNMF_ERR_CUDA;
    }
    if (st != GPUNMF_OK) {
        cudaFree(b->arena);
        delete b;
        return st;
    }
    *out = b;
    return GPUNMF_OK;
}

template <class K, class P>
static cudaError_t spb_launch(K kernel, int grid, int threads, int smem, cudaStream_t s, const P &p) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

static cudaError_t spb_update(SpBatch *b, bool is_w, int update, cudaStream_t s) {
    const SpbUpdParams u{b->insts, is_w ? b->bl_w : b->bl_h, b->P, b->eps, is_w, update};
    return spb_launch(spb_update_kernel, is_w ? b->blocks_w : b->blocks_h, kSpbUpdThreads, update_smem_bytes(kSpbNP, kSpbRows), s, u);
}

// After the factors have been written: their parts and the Gram partials of W.  (An error goes with the old ones.)
gpunmf_status spb_reset(SpBatch *b, cudaStream_t s) {
    GPUNMF_CUDA_TRY(cudaMemsetAsync(b->err, 0, sizeof(int), s));
    for (int i0 = 0; i0 < b->count; i0 += 65535) {
        spb_cut_kernel<<<dim3(4, std::min(65535, b->count - i0), 2), 256, 0, s>>>(b->insts + i0);
        GPUNMF_CUDA_TRY(cudaGetLastError());
    }
    GPUNMF_CUDA_TRY(spb_update(b, true, 0, s));
    return GPUNMF_OK;
}

gpunmf_status spb_run(SpBatch *b, int iters, cudaStream_t s) {
    for (int it = 0; it < iters; it++) {
        GPUNMF_CUDA_TRY(spb_launch(spb_kernel<true>, b->grid_h, kSpbThreads, kSpbSmem, s, b->h));
        GPUNMF_CUDA_TRY(spb_update(b, false, 1, s));
        GPUNMF_CUDA_TRY(spb_launch(spb_kernel<false>, b->grid_w, kSpbThreads, kSpbSmem, s, b->w));
        GPUNMF_CUDA_TRY(spb_update(b, true, 1, s));
    }
    return GPUNMF_OK;
}

int *spb_error_word(SpBatch *b) { return b->err; }

void spb_destroy(SpBatch *b) {
    if (!b) return;
    cudaFree(b->arena);
    delete b;
}
