// Host side of the batched pipeline: builds per-kernel job tables for a batch
// of operations (uneven levels, mixed modes) and launches the seven phase
// kernels on a stream. A built plan only launches kernels, so it can be
// captured in a CUDA graph and replayed.
#include "pipeline.hpp"

#include "devonce.hpp"

#include <algorithm>
#include <cstring>
#include <map>
#include <set>
#include <stdexcept>

namespace pl {

namespace {

int sm_count() { return gfx::current_sm_count(); }



// PATH 0 / 1: the integer / FP64 job segment of a phase; PATH 2: the mixed
// segment (both kinds interleaved, one launch).
template <int LOGN, int PATH>
struct Variant {
    template <int W>
    static void col_attrs() {
        constexpr int SMEM = ntt::Geo<LOGN, W>::COL_SMEM;
        cudaFuncSetAttribute(p2_inv_col<LOGN, PATH, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        cudaFuncSetAttribute(p3_modup_fwd_col<LOGN, PATH, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        cudaFuncSetAttribute(p7a_moddown_inv_col<LOGN, PATH, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        cudaFuncSetAttribute(p7b_moddown_inv_col<LOGN, PATH, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        cudaFuncSetAttribute(p8_moddown_fwd_col<LOGN, PATH, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    }
    static void attrs() {
        using G = ntt::Geo<LOGN>;
        col_attrs<ntt::COL_WIDE>();
        col_attrs<ntt::COL_NARROW>();
        cudaFuncSetAttribute(p1_inv_row<LOGN, PATH>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::ROW_SMEM);
        cudaFuncSetAttribute(p4_modup_fwd_row<LOGN, PATH>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::ROW_SMEM);
        cudaFuncSetAttribute(p6_moddown_inv_row<LOGN, PATH>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::ROW_SMEM);
        cudaFuncSetAttribute(p9_final_fwd_row<LOGN, PATH>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::ROW_SMEM);
    }
    // Phase k of the jobs in segment PATH (P5 and P7 have one integer kernel
    // and are launched by the caller).
    static void phase(int k, const Plan& p, cudaStream_t s, bool& after) {
        using G = ntt::Geo<LOGN>;
        const uint32_t cnt = p.job_cnt[k][PATH];
        if (!cnt) return;
        const DevCtx& D = p.dc;
        const PairDesc* pd = p.d_pairs;
        const uint2* J = p.d_jobs + p.job_off[k][PATH];
        auto run = [&](auto* kernel, unsigned grid, unsigned block, size_t smem) {
            if (gfx::chain_launch(kernel, after, grid, block, smem, s, D, pd, J) == cudaSuccess) after = true;
        };
        // a column kernel on wide tiles, or on narrow ones where those leave SMs idle
        const bool narrow = ntt::narrow_tiles<LOGN>(cnt, sm_count());
        auto run_col = [&](auto* wide, auto* slim) {
            using N = ntt::Geo<LOGN, ntt::COL_NARROW>;
            if (narrow) run(slim, cnt * N::COL_TILES, N::COL_THREADS, N::COL_SMEM);
            else run(wide, cnt * G::COL_TILES, G::COL_THREADS, G::COL_SMEM);
        };
        switch (k) {
            case 0: run(p1_inv_row<LOGN, PATH>, cnt * G::ROW_TILES, G::ROW_THREADS, G::ROW_SMEM); break;
            case 1: run_col(p2_inv_col<LOGN, PATH, ntt::COL_WIDE>, p2_inv_col<LOGN, PATH, ntt::COL_NARROW>); break;
            case 2: run_col(p3_modup_fwd_col<LOGN, PATH, ntt::COL_WIDE>, p3_modup_fwd_col<LOGN, PATH, ntt::COL_NARROW>); break;
            case 3: run(p4_modup_fwd_row<LOGN, PATH>, cnt * G::ROW_TILES, G::ROW_THREADS, G::ROW_SMEM); break;
            case 5: run(p6_moddown_inv_row<LOGN, PATH>, cnt * G::ROW_TILES, G::ROW_THREADS, G::ROW_SMEM); break;
            case 6: run_col(p7a_moddown_inv_col<LOGN, PATH, ntt::COL_WIDE>, p7a_moddown_inv_col<LOGN, PATH, ntt::COL_NARROW>); break;
            case NPHASE: run_col(p7b_moddown_inv_col<LOGN, PATH, ntt::COL_WIDE>, p7b_moddown_inv_col<LOGN, PATH, ntt::COL_NARROW>); break;
            case 7: run_col(p8_moddown_fwd_col<LOGN, PATH, ntt::COL_WIDE>, p8_moddown_fwd_col<LOGN, PATH, ntt::COL_NARROW>); break;
            case 8: run(p9_final_fwd_row<LOGN, PATH>, cnt * G::ROW_TILES, G::ROW_THREADS, G::ROW_SMEM); break;
            default: break;
        }
    }
};

template <int LOGN>
struct Launcher {
    // Kernel attributes, once per ring size and device (and thread-safe). The
    // P5 forms' dynamic shared memory grows with dnum, so their limits are set
    // to the largest size any context can ask for (a limit set for the first
    // context's dnum would be too low for a later context with a different
    // one).
    static void attrs(uint32_t) {
        static gfx::DeviceOnce once;
        once(set_attrs);
    }
    static void set_attrs() {
        Variant<LOGN, 0>::attrs();
        Variant<LOGN, 1>::attrs();
        Variant<LOGN, 2>::attrs();
        p3ws_attrs<0>();
        p3ws_attrs<1>();
        p3ws_attrs<2>();
        cudaFuncSetAttribute(p5_mac<LOGN, MAC_NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, mac_smem(MAC_MAX_DNUM));
        cudaFuncSetAttribute(p5_mac<LOGN, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, mac_smem(MAC_MAX_DNUM));
        cudaFuncSetAttribute(p5_mac_async<LOGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAC_ASYNC_SMEM_MAX);
        cudaFuncSetAttribute(p5_mac_tma<LOGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAC_TMA_SMEM_MAX);
        cudaFuncSetAttribute(p5_mac_fp<LOGN, 4, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, mac_smem(MAC_MAX_DNUM));
        cudaFuncSetAttribute(p5_mac_fp<LOGN, 2, 5>, cudaFuncAttributeMaxDynamicSharedMemorySize, mac_smem(MAC_MAX_DNUM));
        cudaFuncSetAttribute(p5_mac_fp_tma<LOGN, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAC_TMA_SMEM_MAX);
        cudaFuncSetAttribute(p5_mac_fp_tma<LOGN, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAC_TMA_SMEM_MAX);
    }
    // persistent warp-specialised P3 over job segment PATH: form 1 = 128
    // conversion threads, two CTAs per SM; form 2 = 256, one CTA per SM
    template <int PATH>
    static void p3ws_attrs() {
        cudaFuncSetAttribute(p3ws_modup_fwd_col<LOGN, PATH, 128, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             P3WS<LOGN, 128>::SMEM);
        cudaFuncSetAttribute(p3ws_modup_fwd_col<LOGN, PATH, 256, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             P3WS<LOGN, 256>::SMEM);
    }
    template <int PATH>
    static void p3ws(const Plan& p, cudaStream_t s, bool& after) {
        using G = ntt::Geo<LOGN>;
        const uint32_t cnt = p.job_cnt[2][PATH];
        if (!cnt) return;
        const u32 ntiles = cnt * G::COL_TILES;
        const uint2* J = p.d_jobs + p.job_off[2][PATH];
        if (p.p3_form == 1) {
            const unsigned grid = std::min<unsigned>(ntiles, 2u * (unsigned)sm_count());
            if (gfx::chain_launch(p3ws_modup_fwd_col<LOGN, PATH, 128, 2>, after, grid, P3WS<LOGN, 128>::NT,
                                  P3WS<LOGN, 128>::SMEM, s, p.dc, p.d_pairs, J, ntiles) == cudaSuccess)
                after = true;
        } else {
            const unsigned grid = std::min<unsigned>(ntiles, (unsigned)sm_count());
            if (gfx::chain_launch(p3ws_modup_fwd_col<LOGN, PATH, 256, 1>, after, grid, P3WS<LOGN, 256>::NT,
                                  P3WS<LOGN, 256>::SMEM, s, p.dc, p.d_pairs, J, ntiles) == cudaSuccess)
                after = true;
        }
    }
    // The integer forms of P5 over the first nint key-row jobs.
    static void launch_p5_int(const Plan& p, cudaStream_t s, uint32_t nint, bool& after) {
        constexpr int MAC_TILES = (1 << LOGN) / MAC_TILE;
        const DevCtx& D = p.dc;
        const unsigned grid = nint * MAC_TILES;
        auto run = [&](auto* kernel, unsigned g, unsigned block, size_t smem) {
            if (gfx::chain_launch(kernel, after, g, block, smem, s, D, p.d_pairs, p.d_mac_jobs, p.d_plist) ==
                cudaSuccess)
                after = true;
        };
        if (p.p5_form == P5_TMA && mac_tma_ok(D.dnum))
            run(p5_mac_tma<LOGN>, nint * ((1u << LOGN) / P5T_TILE), P5T_NT, p5t_smem((int)D.dnum));
        else if (p.p5_form == P5_ASYNC && mac_async_ok(D.dnum))
            run(p5_mac_async<LOGN>, grid, MACA_NT, maca_smem((int)D.dnum));
        else if (p.p5_form == P5_REG256)
            run(p5_mac<LOGN, 256>, grid, 256, mac_smem(D.dnum));
        else
            run(p5_mac<LOGN, MAC_NT>, grid, MAC_NT, mac_smem(D.dnum));
    }
    static void launch(const Plan& p, cudaStream_t s, unsigned mask) {
        using G = ntt::Geo<LOGN>;
        constexpr int MAC_TILES = (1 << LOGN) / MAC_TILE;
        attrs(p.dc.dnum);
        const DevCtx& D = p.dc;
        bool after = false;   // a kernel of this call directly before on `s`
        for (int k = 0; k < NPHASE; ++k) {
            if (!(mask >> k & 1)) continue;
            if (k == 4) {
                // key rows: [integer rows | 50-bit Q rows]; the second segment goes to
                // the FP64 kernel when p5_fp, else both to the integer form
                const uint32_t nfp = p.p5_fp ? p.job_cnt[4][1] : 0u;
                const uint32_t nint = p.job_cnt[4][0] + p.job_cnt[4][1] - nfp;
                // with p5_split the FP64 rows run on a second stream beside the integer
                // rows (different pipes, disjoint outputs), joined before P6
                cudaStream_t sf = s;
                const bool split = p.p5_split && nfp && nint && ensure_side(p);
                if (split) {
                    cudaEventRecord(p.ev_fork, s);
                    cudaStreamWaitEvent(p.side, p.ev_fork, 0);
                    sf = p.side;
                    after = false;
                }
                const uint4* fj = p.d_mac_jobs + p.job_off[4][1];
                auto run = [&](auto* kernel, unsigned g, unsigned block, size_t smem) {
                    if (gfx::chain_launch(kernel, after, g, block, smem, sf, D, p.d_pairs, fj, p.d_plist) ==
                            cudaSuccess && !split)
                        after = true;
                };
                if (nfp && p.p5_fp_form == 2 && mac_tma_ok(D.dnum))
                    run(p5_mac_fp_tma<LOGN, 3>, nfp * ((1u << LOGN) / P5T_TILE), P5T_NT, p5t_smem((int)D.dnum, 3));
                else if (nfp && p.p5_fp_form == 3 && mac_tma_ok(D.dnum))
                    run(p5_mac_fp_tma<LOGN, 2>, nfp * ((1u << LOGN) / P5T_TILE), P5T_NT, p5t_smem((int)D.dnum, 2, true));
                else if (nfp && p.p5_fp_form == 1)
                    run(p5_mac_fp<LOGN, 2, 5>, nfp * MAC_TILES, MACF_NT, mac_smem(D.dnum));
                else if (nfp)
                    run(p5_mac_fp<LOGN, 4, 4>, nfp * MAC_TILES, MACF_NT, mac_smem(D.dnum));
                if (split) {
                    launch_p5_int(p, s, nint, after);
                    cudaEventRecord(p.ev_join, p.side);
                    cudaStreamWaitEvent(s, p.ev_join, 0);
                    after = false;
                    continue;
                }
                if (!nint) continue;
                launch_p5_int(p, s, nint, after);
            } else if (k == 6) {   // P7a then P7b (U and r_l need the P towers)
                for (int kk : {6, (int)NPHASE}) {
                    if ((p.mix >> 6 & 1) && p.job_cnt[kk][0] && p.job_cnt[kk][1]) {
                        Variant<LOGN, 2>::phase(kk, p, s, after);
                    } else {
                        Variant<LOGN, 0>::phase(kk, p, s, after);
                        Variant<LOGN, 1>::phase(kk, p, s, after);
                    }
                }
            } else if (k == 2 && p.p3_form) {
                if ((p.mix >> 2 & 1) && p.job_cnt[2][0] && p.job_cnt[2][1]) p3ws<2>(p, s, after);
                else { p3ws<0>(p, s, after); p3ws<1>(p, s, after); }
            } else if ((p.mix >> k & 1) && p.job_cnt[k][0] && p.job_cnt[k][1]) {
                Variant<LOGN, 2>::phase(k, p, s, after);
            } else {
                Variant<LOGN, 0>::phase(k, p, s, after);
                Variant<LOGN, 1>::phase(k, p, s, after);
            }
        }
    }
};

}  // namespace

bool supported_logn(int logn) { return logn >= 10 && logn <= 16; }

int input_count(uint32_t mode) { return mode == EMR ? 4 : (mode == ROT || mode == HROT) ? 2 : 1; }
uint32_t output_towers(const Op& op) { return (op.mode == EMR || op.mode == RESCALE) ? op.L - 1 : op.L; }  // ROT, HROT, KS: L

size_t op_workspace_words(const gfx::Context& c, uint32_t L) {
    return (size_t)ws_layout(L, c.K(), c.alpha()).total * c.n();
}

void validate(const gfx::Context& c, const Op& op) {
    if (op.L < 1 || op.L > c.fullQ()) throw std::invalid_argument("level out of range");
    if ((op.mode == EMR || op.mode == RESCALE) && op.L < 2) throw std::invalid_argument("rescale needs L >= 2");
    if (c.alpha() > (uint32_t)MAXA) throw std::invalid_argument("digit width above the fused limit");
    if (c.dnum() > (uint32_t)MAC_MAX_DNUM) throw std::invalid_argument("too many digits for the key-stationary MAC");
    if (op.mode > HROT) throw std::invalid_argument("unknown mode");
    const int nin = input_count(op.mode);
    for (int k = 0; k < nin; ++k) if (!op.in[k]) throw std::invalid_argument("null input");
    if (!op.out[0] || (op.mode != RESCALE && !op.out[1])) throw std::invalid_argument("null output");
    if ((op.mode == ROT || op.mode == HROT) && (op.galois % 2 == 0 || op.galois >= 2ull * c.n()))
        throw std::invalid_argument("bad Galois element");
    auto misaligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    for (int k = 0; k < nin; ++k)
        if (misaligned(op.in[k])) throw std::invalid_argument("input buffers must be 16-byte aligned");
    if (misaligned(op.out[0]) || (op.mode != RESCALE && misaligned(op.out[1])))
        throw std::invalid_argument("output buffers must be 16-byte aligned");
}

// Host tables of a batch: pair descriptors, per-phase jobs and P5 groups.
struct HostTables {
    std::vector<PairDesc> pairs;
    std::vector<uint2> jobs;       // all phases, concatenated
    std::vector<uint4> mac_jobs;
    std::vector<uint32_t> plist;
    size_t job_off[NPHASE + 1][3] = {};     // [phase (+ the second P7 launch)][integer, FP64, mixed]
    uint32_t job_cnt[NPHASE + 1][3] = {};
};

static void fill_tables(const gfx::Context& c, const std::vector<Op>& ops, const std::vector<u64*>& ws_ptrs,
                        HostTables& T) {
    const uint32_t K = c.K();
    T.pairs.assign(ops.size(), PairDesc{});
    std::vector<uint2> jobs[NPHASE + 1];   // index NPHASE: the second P7 launch (U and r_l)
    std::map<std::pair<uint64_t, uint32_t>, std::vector<uint32_t>> rows;
    std::map<std::pair<const u64*, uint32_t>, uint32_t> hoist_lead;   // (c1, level) -> first HROT op
    for (size_t pi = 0; pi < ops.size(); ++pi) {
        const Op& op = ops[pi];
        PairDesc& P = T.pairs[pi];
        std::memset(&P, 0, sizeof(P));
        P.L = op.L;
        P.mode = op.mode;
        P.galois = op.galois;
        for (int k = 0; k < 4; ++k) P.in[k] = op.in[k];
        P.out[0] = op.out[0];
        P.out[1] = op.out[1];
        P.ws = ws_ptrs[pi];
        P.ysrc = P.ws;
        bool modup = true;   // this op computes its own ModUp (P1-P4)
        if (op.mode == HROT) {
            auto ins = hoist_lead.emplace(std::make_pair(op.in[1], op.L), (uint32_t)pi);
            if (!ins.second) {
                P.ysrc = T.pairs[ins.first->second].ws;
                modup = false;
            }
        }
        if (op.mode != RESCALE) {
            const gfx::Key* key = c.key(op.key_id);
            if (!key) throw std::invalid_argument("missing eval key");
            if (!key->av) throw std::logic_error("eval key not resident (not pinned by the plan)");
            P.kav = key->av;
            P.kbv = key->bv;
        }
        const uint32_t L = op.L, QlP = L + K, pu = (uint32_t)pi;
        const uint32_t nparts = (L + c.alpha() - 1) / c.alpha();
        if (op.mode == RESCALE) {
            jobs[0].push_back({pu, L - 1});
            jobs[1].push_back({pu, L - 1});
            for (uint32_t i = 0; i + 1 < L; ++i) { jobs[7].push_back({pu, i}); jobs[8].push_back({pu, i}); }
            continue;
        }
        if (modup) {
            for (uint32_t i = 0; i < L; ++i) { jobs[0].push_back({pu, i}); jobs[1].push_back({pu, i}); }
            for (uint32_t p = 0; p < nparts; ++p) {
                const uint32_t st = c.alpha() * p, sp = std::min(c.alpha(), L - st);
                for (uint32_t i = 0; i < QlP; ++i)
                    if (i < st || i >= st + sp) {
                        jobs[2].push_back({pu, p * QlP + i});
                        jobs[3].push_back({pu, p * QlP + i});
                    }
            }
        }
        for (uint32_t i = 0; i < QlP; ++i) rows[{op.key_id, qp_of(i, L, c.fullQ())}].push_back(pu);
        const bool emr = op.mode == EMR;
        for (uint32_t cc = 0; cc < 2; ++cc) {
            for (uint32_t t = emr ? 0 : 1; t <= K; ++t) jobs[5].push_back({pu, cc * (K + 1) + t});
            for (uint32_t t = 1; t <= K; ++t) jobs[6].push_back({pu, cc * (K + 1) + t});
            if (emr) jobs[NPHASE].push_back({pu, cc * (K + 1)});   // P7b: U of component cc
        }
        const uint32_t outL = emr ? L - 1 : L;
        for (uint32_t cc = 0; cc < 2; ++cc)
            for (uint32_t i = 0; i < outL; ++i) { jobs[7].push_back({pu, cc * L + i}); jobs[8].push_back({pu, cc * L + i}); }
    }
    T.mac_jobs.clear();
    T.plist.clear();
    // P5 jobs in two segments: key rows the integer forms must take (P rows,
    // Q rows with q >= 2^50), then Q rows with q < 2^50, which the FP64 form
    // may take instead
    std::vector<uint4> mac_fp;
    for (auto& kv : rows) {
        const auto& v = kv.second;
        const uint32_t r = kv.first.second;
        const bool fp = r < c.fullQ() && fp_tower(c.Q()[r]);
        for (size_t g = 0; g < v.size(); g += MAC_GROUP) {
            const uint32_t cnt = (uint32_t)std::min<size_t>(MAC_GROUP, v.size() - g);
            (fp ? mac_fp : T.mac_jobs).push_back({r, (uint32_t)T.plist.size(), cnt, 0});
            T.plist.insert(T.plist.end(), v.begin() + g, v.begin() + g + cnt);
        }
    }
    const uint32_t n_int_rows = (uint32_t)T.mac_jobs.size();
    T.mac_jobs.insert(T.mac_jobs.end(), mac_fp.begin(), mac_fp.end());
    // Route the transform jobs of each NTT phase to the integer or the FP64
    // kernel by the modulus of the tower they transform (P7 stays integer:
    // one CTA there mixes P towers and tower L-1).
    const std::vector<u64>& Qv = c.Q();
    const std::vector<u64>& Pv = c.P();
    auto qp_mod = [&](u32 qp) { return qp < c.fullQ() ? Qv[qp] : Pv[qp - c.fullQ()]; };
    auto tower = [&](int k, const uint2& j) -> u32 {
        const PairDesc& P = T.pairs[j.x];
        switch (k) {
            case 0: case 1: return j.y;
            case 2: case 3: return qp_of(j.y % (P.L + K), P.L, c.fullQ());
            case 5: case 6: case NPHASE: { const u32 t = j.y % (K + 1); return t == 0 ? P.L - 1 : c.fullQ() + t - 1; }
            default: return j.y % P.L;   // 7, 8
        }
    };
    T.jobs.clear();
    for (int k = 0; k <= NPHASE; ++k) {
        const bool split = k != 4;
        for (int v = 0; v < 2; ++v) {
            T.job_off[k][v] = T.jobs.size();
            for (const uint2& j : jobs[k]) {
                const bool fp = split && fp_tower(qp_mod(tower(k, j)));
                if ((int)fp == v) T.jobs.push_back(j);
            }
            T.job_cnt[k][v] = (uint32_t)(T.jobs.size() - T.job_off[k][v]);
        }
        // mixed segment: the two lists interleaved in proportion, FP64 jobs
        // tagged with JOB_FP, so neighbouring CTAs load different pipes
        T.job_off[k][2] = T.jobs.size();
        const uint32_t na = T.job_cnt[k][0], nb = T.job_cnt[k][1];
        if (split && na && nb) {
            const size_t oa = T.job_off[k][0], ob = T.job_off[k][1];
            uint32_t ia = 0, ib = 0;
            while (ia < na || ib < nb) {
                const bool take_b = ia == na || (ib < nb && (uint64_t)ib * na <= (uint64_t)ia * nb);
                if (take_b) { uint2 j = T.jobs[ob + ib++]; j.y |= JOB_FP; T.jobs.push_back(j); }
                else { const uint2 j = T.jobs[oa + ia++]; T.jobs.push_back(j); }
            }
        }
        T.job_cnt[k][2] = (uint32_t)(T.jobs.size() - T.job_off[k][2]);
    }
    T.job_cnt[4][0] = n_int_rows;
    T.job_off[4][1] = n_int_rows;                         // offset of the FP64 segment in mac_jobs
    T.job_cnt[4][1] = (uint32_t)T.mac_jobs.size() - n_int_rows;
    T.job_cnt[4][2] = 0;
}

// The plan's second stream and fork / join events (made on the current device
// at first use); false if they cannot be made, and P5 then runs on one stream.
bool ensure_side(const Plan& p) {
    if (p.side) return true;
    cudaStream_t st = nullptr;
    cudaEvent_t a = nullptr, b = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return false;
    if (cudaEventCreateWithFlags(&a, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&b, cudaEventDisableTiming) != cudaSuccess) {
        if (a) cudaEventDestroy(a);
        cudaStreamDestroy(st);
        return false;
    }
    p.side = st;
    p.ev_fork = a;
    p.ev_join = b;
    return true;
}

Plan::Plan() : staging(std::make_unique<HostTables>()) {}

Plan::~Plan() {
    if (ctx) {
        for (uint64_t id : key_pins) ctx->release(id);
        gfx::Context::drop(ctx);                 // may delete a retired context: touch it no more
    }
    if (d_blob) cudaFree(d_blob);
    if (h_blob) cudaFreeHost(h_blob);
    for (void* h : old_h_blobs) cudaFreeHost(h);
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_join) cudaEventDestroy(ev_join);
    if (side) cudaStreamDestroy(side);
    if (own_ws && ws) cudaFree(ws);
}

// All tables of a plan live in one device blob (pairs, jobs, P5 groups, pair
// lists at 256-byte aligned offsets), uploaded by one copy from a pinned host
// mirror, so an asynchronous rebuild does not wait for the stream.
static void commit(Plan& p, const HostTables& T, const std::vector<Op>& ops, cudaStream_t s, bool async) {
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t b_pairs = al(T.pairs.size() * sizeof(PairDesc));
    const size_t b_jobs = al(T.jobs.size() * sizeof(uint2));
    const size_t b_mac = al(T.mac_jobs.size() * sizeof(uint4));
    const size_t b_plist = al(T.plist.size() * sizeof(uint32_t));
    const size_t total = std::max<size_t>(b_pairs + b_jobs + b_mac + b_plist, 256);
    if (total > p.blob_cap) {
        // Grow by doubling without stalling the device: an asynchronous rebuild
        // frees the old device blob in stream order (its last reader is earlier
        // work on s) and keeps the old pinned mirror until the plan is
        // destroyed; cudaFree / cudaFreeHost here would wait for every running
        // kernel, which stalled the serving loop's host whenever its batches
        // reached a new size.
        const size_t cap = std::max<size_t>(2 * total, (size_t)1 << 16);
        void* nd = nullptr;
        void* nh = nullptr;
        const cudaError_t ed = async ? cudaMallocAsync(&nd, cap, s) : cudaMalloc(&nd, cap);
        if (ed != cudaSuccess) throw std::runtime_error("plan allocation failed");
        if (cudaMallocHost(&nh, cap) != cudaSuccess) {
            if (async) cudaFreeAsync(nd, s); else cudaFree(nd);
            throw std::runtime_error("plan host allocation failed");
        }
        if (p.d_blob) {
            if (async) cudaFreeAsync(p.d_blob, s); else cudaFree(p.d_blob);
        }
        if (p.h_blob) {
            if (async) p.old_h_blobs.push_back(p.h_blob); else cudaFreeHost(p.h_blob);
        }
        p.d_blob = nd;
        p.h_blob = nh;
        p.blob_cap = cap;
    }
    char* h = static_cast<char*>(p.h_blob);
    char* d = static_cast<char*>(p.d_blob);
    std::memcpy(h, T.pairs.data(), T.pairs.size() * sizeof(PairDesc));
    std::memcpy(h + b_pairs, T.jobs.data(), T.jobs.size() * sizeof(uint2));
    std::memcpy(h + b_pairs + b_jobs, T.mac_jobs.data(), T.mac_jobs.size() * sizeof(uint4));
    std::memcpy(h + b_pairs + b_jobs + b_mac, T.plist.data(), T.plist.size() * sizeof(uint32_t));
    const size_t used = b_pairs + b_jobs + b_mac + b_plist;
    if (used) {
        cudaError_t e = async ? cudaMemcpyAsync(d, h, used, cudaMemcpyHostToDevice, s)
                              : cudaMemcpy(d, h, used, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) throw std::runtime_error(std::string("plan upload: ") + cudaGetErrorString(e));
    }
    p.d_pairs = reinterpret_cast<PairDesc*>(d);
    p.d_jobs = reinterpret_cast<uint2*>(d + b_pairs);
    p.d_mac_jobs = reinterpret_cast<uint4*>(d + b_pairs + b_jobs);
    p.d_plist = reinterpret_cast<uint32_t*>(d + b_pairs + b_jobs + b_mac);
    for (int k = 0; k <= NPHASE; ++k)
        for (int v = 0; v < 3; ++v) { p.job_off[k][v] = T.job_off[k][v]; p.job_cnt[k][v] = T.job_cnt[k][v]; }
    p.nops = (uint32_t)ops.size();
    p.ops = ops;
    p.overwrites = -1;
    p.pairs_host = T.pairs;
}

// Makes every key the batch uses resident and pinned for the plan's lifetime
// (releasing the keys of the plan's previous batch).
static void pin_keys(Plan& p, const gfx::Context& c, const std::vector<Op>& ops) {
    std::set<uint64_t> ids;
    for (const Op& op : ops)
        if (op.mode != RESCALE) ids.insert(op.key_id);
    const gfx::Context* old = p.ctx;
    if (old)
        for (uint64_t id : p.key_pins) old->release(id);
    p.key_pins.clear();
    if (old != &c) {
        c.hold();
        p.ctx = &c;
        if (old) gfx::Context::drop(old);
    }
    try {
        for (uint64_t id : ids) {
            if (!c.acquire(id)) throw std::invalid_argument("missing eval key");
            p.key_pins.push_back(id);
        }
    } catch (...) {
        for (uint64_t id : p.key_pins) c.release(id);
        p.key_pins.clear();
        throw;
    }
}

std::unique_ptr<Plan> build_plan(const gfx::Context& c, const std::vector<Op>& ops, u64* ws, size_t ws_words) {
    if (!supported_logn((int)c.logn())) throw std::invalid_argument("pipeline supports n = 2^10 .. 2^16");
    auto plan = std::make_unique<Plan>();
    plan->dc = c.dev();                          // plan->ctx (and its hold) is set by pin_keys
    plan->logn = c.logn();
    size_t need = 0;
    for (const Op& op : ops) { validate(c, op); need += op_workspace_words(c, op.L); }
    if (!ws) {
        if (cudaMalloc(&plan->ws, std::max<size_t>(need, 1) * 8) != cudaSuccess)
            throw std::runtime_error("workspace allocation failed");
        plan->own_ws = true;
        ws = plan->ws;
    } else if (ws_words < need) {
        throw std::length_error("workspace too small");
    } else if (reinterpret_cast<uintptr_t>(ws) & 15) {
        throw std::invalid_argument("workspace must be 16-byte aligned");
    }
    plan->ws_words = need;
    pin_keys(*plan, c, ops);
    std::vector<u64*> wsp(ops.size());
    size_t off = 0;
    for (size_t i = 0; i < ops.size(); ++i) { wsp[i] = ws + off; off += op_workspace_words(c, ops[i].L); }
    HostTables T;
    fill_tables(c, ops, wsp, T);
    commit(*plan, T, ops, 0, false);
    return plan;
}

void build_plan_into(Plan& p, const gfx::Context& c, const std::vector<Op>& ops, const std::vector<u64*>& ws_ptrs,
                     cudaStream_t s) {
    if (!supported_logn((int)c.logn())) throw std::invalid_argument("pipeline supports n = 2^10 .. 2^16");
    if (ws_ptrs.size() != ops.size()) throw std::invalid_argument("one workspace per operation");
    for (u64* w : ws_ptrs)
        if (!w || (reinterpret_cast<uintptr_t>(w) & 15)) throw std::invalid_argument("workspace must be 16-byte aligned");
    for (const Op& op : ops) validate(c, op);
    pin_keys(p, c, ops);
    p.dc = c.dev();
    p.logn = c.logn();
    p.tuned = false;
    HostTables& T = *p.staging;
    fill_tables(c, ops, ws_ptrs, T);
    commit(p, T, ops, s, true);
}

namespace {
__global__ void k_set_pair(PairDesc* dst, PairDesc v) { *dst = v; }
}  // namespace

void rebind(Plan& p, uint32_t idx, const Op& op, const gfx::Context& c, cudaStream_t s) {
    if (idx >= p.pairs_host.size()) throw std::invalid_argument("rebind: index");
    validate(c, op);
    const Op& old = p.ops[idx];
    if (old.mode == HROT || op.mode == HROT) throw std::invalid_argument("rebind: hoisted rotations cannot be rebound");
    const bool same_shape = old.L == op.L && (old.mode == op.mode ||
                            ((old.mode == KS || old.mode == ROT) && (op.mode == KS || op.mode == ROT)));
    if (!same_shape) throw std::invalid_argument("rebind: level or job shape differs");
    if (op.key_id != old.key_id && p.ops.size() > 1)
        throw std::invalid_argument("rebind: changing the key of one operation of a shared batch");
    if (op.mode != RESCALE && op.key_id != old.key_id) {   // single-op plan: move the pin
        if (!c.acquire(op.key_id)) throw std::invalid_argument("missing eval key");
        for (auto& id : p.key_pins)
            if (id == old.key_id) { c.release(id); id = op.key_id; break; }
    }
    PairDesc P = p.pairs_host[idx];
    P.mode = op.mode;
    P.galois = op.galois;
    for (int k = 0; k < 4; ++k) P.in[k] = op.in[k];
    P.out[0] = op.out[0];
    P.out[1] = op.out[1];
    if (op.mode != RESCALE) {
        const gfx::Key* key = c.key(op.key_id);
        if (!key) throw std::invalid_argument("missing eval key");
        P.kav = key->av;
        P.kbv = key->bv;
    }
    p.pairs_host[idx] = P;
    p.ops[idx] = op;
    p.overwrites = -1;
    k_set_pair<<<1, 1, 0, s>>>(p.d_pairs + idx, P);
}

namespace {
// A schedule's place in the context's cache: the batch-size class, floor(log2) of
// the number of operations with a key product (rescales have none, so they do
// not set the key product's forms), beside what changes which forms win: rings
// shared with other streams, hoisted rotations, rotations without products (the
// P5 ring forms read their source blocks whole, the register forms gather them
// word by word), and rescales, whose jobs take part in the choice of separate or
// interleaved launches. So the order in which a program first launches its
// batches does not matter: each kind is timed on its own kind.
struct TuneKey {
    uint64_t own;        // this batch's entry
    uint64_t products;   // the entry of a batch of products of the same size
};
TuneKey tune_key(const Plan& p) {
    uint32_t keyed = 0, cls = 0;
    bool hoisted = false, plain = false, product = false;
    for (const Op& op : p.ops) {
        keyed += op.mode != RESCALE;
        hoisted = hoisted || op.mode == HROT;
        plain = plain || op.mode == ROT;
        product = product || op.mode == EMR || op.mode == KS;
    }
    while ((2u << cls) <= (keyed ? keyed : p.nops)) ++cls;
    const uint64_t base = (p.concurrent ? 1ull << 48 : 0ull) | ((uint64_t)p.logn << 40) |
                          ((uint64_t)p.dc.dnum << 32) | (hoisted ? 1ull << 16 : 0ull) | cls;
    return {base | (plain && !product ? 1ull << 17 : 0ull) | (keyed < p.nops ? 1ull << 18 : 0ull), base};
}
// choice: bits 0-1 = P5 form, bits 3-4 = P3 form (0 plain, 1 and 2
// warp-specialised), bit 6 = P5 key rows of 50-bit Q towers on the FP64
// pipe, bit 7 = its occupancy form (0: 4 digits in flight, 4 CTAs per SM;
// 1: 2 digits, 5 CTAs), bits 8-16 = phases launched over their interleaved
// integer / FP64 job list (else as two launches), bit 17 = P5's FP64 and
// integer rows on two streams at once, bit 18 = the FP64 rows in the TMA
// form (p5_mac_fp_tma, three stages; with bit 7, two)
void apply_choice(Plan& p, int choice) {
    p.p5_form = choice & 3;
    p.p5_fp = (choice >> 6) & 1;
    p.p5_fp_form = ((choice >> 18) & 1 ? 2 : 0) + ((choice >> 7) & 1);
    if (p.p5_fp_form >= 2 && !mac_tma_ok(p.dc.dnum)) p.p5_fp_form = 0;
    p.p5_split = (choice >> 17) & 1;
    if (p.p5_split) ensure_side(p);   // outside any graph capture where possible
    if (p.p5_form == P5_ASYNC && !mac_async_ok(p.dc.dnum)) p.p5_form = P5_REG128;
    if (p.p5_form == P5_TMA && !mac_tma_ok(p.dc.dnum)) p.p5_form = P5_REG128;
    p.mix = ((unsigned)choice >> 8) & 0x1ffu;
    p.p3_form = (choice >> 3) & 3;
    if (p.p3_form > 2) p.p3_form = 0;
}
// Whether any output of the batch overlaps an input of it, the operation's own or
// another's. Found once per set of buffers (a batch that is never timed asks at
// every launch): inputs in order of their start, each with the furthest end up to
// it, against the inputs that start before an output ends.
bool overwrites_inputs(Plan& p) {
    if (p.overwrites >= 0) return p.overwrites != 0;
    const uintptr_t tower = sizeof(u64) << p.logn;
    std::vector<std::pair<uintptr_t, uintptr_t>> in;
    for (const Op& op : p.ops)
        for (int k = 0; k < input_count(op.mode); ++k) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(op.in[k]);
            in.push_back({a, a + op.L * tower});
        }
    std::sort(in.begin(), in.end());
    for (size_t i = 1; i < in.size(); ++i) in[i].second = std::max(in[i].second, in[i - 1].second);
    bool hit = false;
    for (const Op& op : p.ops)
        for (int k = 0; k < (op.mode == RESCALE ? 1 : 2); ++k) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(op.out[k]), b = a + output_towers(op) * tower;
            const auto it = std::lower_bound(in.begin(), in.end(), std::make_pair(b, (uintptr_t)0));
            hit = hit || (it != in.begin() && std::prev(it)->second > a);
        }
    p.overwrites = hit ? 1 : 0;
    return hit;
}
}  // namespace

void tune(Plan& p, cudaStream_t s, bool measure) {
    if (p.tuned || !p.nops || !p.ctx) return;
    const gfx::Context& c = *p.ctx;
    const TuneKey key = tune_key(p);
    int choice = 0;
    if (c.tuned_choice(key.own, choice)) {
        apply_choice(p, choice);
        p.tuned = true;
        return;
    }
    // 4-word register P5 with FP64 Q rows, plain P3, interleaved paths
    constexpr int DEFAULT = P5_REG128 | 64 | (0x1ff << 8);
    // until the batch is timed: the products' entry, else the default
    apply_choice(p, c.tuned_choice(key.products, choice) ? choice : DEFAULT);
    if (!measure) return;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return;
    // Timing re-runs the batch, so none of its operations may write over an input.
    // A batch with out-of-place rescales is timed like any other: without, 13 mixed
    // operations at N = 2^14 kept the default key-product form (97 us where the
    // tuned forms take 68; the whole step 402 -> 385 us). Rescales alone have no key
    // product to choose a form for.
    bool keyed = false;
    for (const Op& op : p.ops) keyed = keyed || op.mode != RESCALE;
    if (!keyed || overwrites_inputs(p)) return;
    cudaEvent_t a, b;
    if (cudaEventCreate(&a) != cudaSuccess) return;
    if (cudaEventCreate(&b) != cudaSuccess) { cudaEventDestroy(a); return; }
    launch(p, s);                                // every workspace slot holds data of this batch
    bool ok = true;
    // One decision per dimension, each timed on the phases it changes: two
    // interleaved passes, best of three launches per candidate and pass; a
    // candidate replaces the current value only if it is 1.5% faster.
    auto pick = [&](unsigned mask, int field_mask, const std::vector<int>& values, int cur) {
        std::vector<float> best(values.size(), 1e30f);
        for (int pass = 0; pass < 2 && ok; ++pass)
            for (size_t ci = 0; ci < values.size() && ok; ++ci) {
                apply_choice(p, (cur & ~field_mask) | values[ci]);
                launch(p, s, mask);
                for (int r = 0; r < 3; ++r) {
                    cudaEventRecord(a, s);
                    launch(p, s, mask);
                    cudaEventRecord(b, s);
                    if (cudaEventSynchronize(b) != cudaSuccess) { ok = false; break; }
                    float ms = 0;
                    cudaEventElapsedTime(&ms, a, b);
                    best[ci] = std::min(best[ci], ms);
                }
            }
        size_t win = 0;                          // values[0] is the current setting
        for (size_t ci = 1; ci < values.size(); ++ci)
            if (best[ci] < best[win]) win = ci;
        if (!ok || best[win] > 0.985f * best[0]) win = 0;
        return (cur & ~field_mask) | values[win];
    };
    int cur = DEFAULT;
    for (int k : {0, 1, 2, 3, 5, 6, 7, 8}) {                       // interleaved or separate, per phase
        const bool both = (p.job_cnt[k][0] && p.job_cnt[k][1]) ||
                          (k == 6 && p.job_cnt[NPHASE][0] && p.job_cnt[NPHASE][1]);
        if (!both) continue;
        const int bit = 1 << (8 + k);
        cur = pick(1u << k, bit, {bit, 0}, cur);
    }
    cur = pick(1u << 2, 24, {0, 8, 16}, cur);                      // P3 form
    if (p.job_cnt[4][1]) {
        // P5 FP64 rows (register form 0, then the TMA form where its ring fits,
        // else register form 1) or integer; the TMA form wins the large
        // batches, form 0 the small ones (its ring's set-up is not amortised)
        const std::vector<int> fpv = mac_tma_ok(p.dc.dnum) && !p.concurrent
                                         ? std::vector<int>{64, 64 | 128, 64 | 1 << 18, 64 | 128 | 1 << 18, 0}
                                         : std::vector<int>{64, 64 | 128, 0};
        cur = pick(1u << 4, 64 | 128 | 1 << 18, fpv, cur);
        if (cur & 64) cur = pick(1u << 4, 1 << 17, {0, 1 << 17}, cur);   // FP64 and integer rows concurrent
    }
    std::vector<int> p5v = {P5_REG128, P5_REG256};
    if (mac_async_ok(p.dc.dnum)) p5v.push_back(P5_ASYNC);
    if (mac_tma_ok(p.dc.dnum)) p5v.push_back(P5_TMA);
    cur = pick(1u << 4, 3, p5v, cur);                              // P5 form
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    apply_choice(p, cur);
    c.set_tuned_choice(key.own, cur);
    p.tuned = true;
}

cudaError_t launch(const Plan& p, cudaStream_t s, unsigned mask) {
    switch (p.logn) {
        case 10: Launcher<10>::launch(p, s, mask); break;
        case 11: Launcher<11>::launch(p, s, mask); break;
        case 12: Launcher<12>::launch(p, s, mask); break;
        case 13: Launcher<13>::launch(p, s, mask); break;
        case 14: Launcher<14>::launch(p, s, mask); break;
        case 15: Launcher<15>::launch(p, s, mask); break;
        case 16: Launcher<16>::launch(p, s, mask); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace pl
