/*
 * swehr_launch.cuh -- launch geometry and enqueueing of the two step kernels
 * of one form (included once per form, by swehr_step_f64.cu and
 * swehr_step_f32.cu, which are compiled with different contraction flags).
 */
#pragma once
#include <cuda_runtime.h>

#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "swehr_kernels.h"
#include "swehr_tile.cuh"

namespace swehr {

typedef CUresult (*TensorMapEncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                      const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                      CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

/* cuTensorMapEncodeTiled through the runtime's driver entry point (no link
 * against libcuda); null when the driver does not offer it */
static inline TensorMapEncodeFn tensor_map_encoder()
{
    static TensorMapEncodeFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (TensorMapEncodeFn)p;
    }
    return fn;
}

/* A 3-D tensor (ny, nx, planes) of T planes at base with the domain's pitch
 * and plane stride, copied in boxes of box_x x box_y x 1.  The driver checks
 * the base (16-byte aligned), the strides (multiples of 16 bytes) and the
 * box's inner extent (a multiple of 16 bytes). */
template <class T>
static inline bool encode_planes(TensorMapEncodeFn enc, CUtensorMap *m, const void *base, const DevParams &P,
                                 int planes, unsigned box_x, unsigned box_y)
{
    const cuuint64_t dims[3] = {(cuuint64_t)P.ny, (cuuint64_t)P.nx, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)P.pitch * sizeof(T), (cuuint64_t)P.plane * sizeof(T)};
    const cuuint32_t box[3] = {box_x, box_y, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUtensorMapDataType dt = sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    return enc(m, dt, 3, const_cast<void *>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}

/* A kernel's dynamic shared memory limit belongs to the process (on one
 * device), not to the simulation or pool that sets it: one that needs less,
 * made later, must leave the others' launches possible, so it is only raised.
 * (The limit set is remembered: asking for a kernel's attributes costs a new
 * simulation 0.4 ms a kernel.) */
static inline cudaError_t raise_smem_limit(const void *fn, size_t bytes)
{
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, size_t> limits;
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t &limit = limits[{dev, fn}];
    if (limit < bytes) limit = bytes;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
}

inline namespace SWEHR_TILE_NS {

/* Tiles per SM up to which a domain is stepped by k_run_tile.  Measured (B200,
 * 7 classes, ponded flow, us a step, two kernels and many steps a launch):
 *   tiles      1     64    175    384    750    969   1280   1536   2816
 *   FP64    35.1   32.0   33.2   48.8   71.6   99.5  121.8  138.2  219.7
 *           32.3   27.4   29.4   48.1   70.1   97.7  124.4  143.7  221.2
 *   mixed   22.3   22.0   23.3   25.5   35.0   42.6   48.7   60.1   94.8
 *           19.2   18.4   20.7   23.2   33.5   46.2   45.7   60.5   98.7
 * What a launch saves is the same at any size, but the wave pass runs at the
 * update's occupancy and a block's tiles wait for the slowest block at every
 * barrier; from about 970 tiles (6.5 per SM) it depends on how full the last
 * wave of tiles is which is faster.  With interior solid cells (the wave pass takes one cell
 * a thread: 517 x 389, 10 classes 134 and 150 us) and with budgets (block 0
 * folds the sums between two barriers: 200 x 50 mixed 40 and 47 us) two kernels
 * stay. */
#define RUN_TILES_PER_SM 4

template <class PP, class RS>
struct FormLauncher {
    typedef typename PP::R R;

    static size_t update_smem(int S, int stage_m = 1) { return StagedLayout::make(S, sizeof(R), stage_m).total; }

    /* The update kernel and shared memory for S classes: M_k staged unless
     * leaving it in global memory fits more blocks per SM (measured: staging
     * is 2-5 % faster at equal occupancy; at 10 FP64 classes dropping it
     * doubles the resident blocks and the update runs ~27 % faster).  Sets
     * both kernels' shared-memory limits. */
    static cudaError_t pick_staging(void *f_with, void *f_without, int S, size_t &smem, int &occ, int &stage_m,
                                    void *&fn, size_t extra = 0)
    {
        const size_t with = update_smem(S, 1) + extra, without = update_smem(S, 0) + extra;
        int ow = 0, oo = 0;
        cudaError_t e = raise_smem_limit(f_with, with);
        if (e != cudaSuccess) return e;
        e = raise_smem_limit(f_without, without);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ow, f_with, TILE_THREADS, with);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&oo, f_without, TILE_THREADS, without);
        if (e != cudaSuccess) return e;
        stage_m = ow >= oo;
        smem = stage_m ? with : without;
        occ = stage_m ? ow : oo;
        fn = stage_m ? f_with : f_without;
        if (occ < 1) occ = 1;
        return cudaSuccess;
    }
    static size_t wave_smem() { return 0; }   /* the wave pass stages nothing */

    static int init_gz(const DevParams &P, const BufsT<RS> &B, int64_t n, cudaStream_t s)
    {
        k_init_gz<PP, RS><<<4 * 148, TILE_THREADS, 0, s>>>(P, B, n);
        return (int)cudaGetLastError();
    }

    /* Tensor maps for the update kernel's tile loads (planes of one domain):
     * each state set's planes of the storage type with the halo box and the
     * cell box, its FP64 planes with the cell box, the three topography
     * planes with the z_prev and z window boxes, and the Ks plane.  Returns 0
     * when every map was encoded. */
    static int encode_tma(const DevParams &P, const BufsT<RS> &B, TmaMaps &tm)
    {
        TensorMapEncodeFn enc = tensor_map_encoder();
        if (!enc) return 1;
        memset(&tm, 0, sizeof tm);
        const bool mixed = !std::is_same<RS, double>::value;
        const int planes = mixed ? 9 + P.S : P_FIXED + 2 * P.S;     /* the storage-type block of a set */
        bool ok = true;
        for (int s = 0; s < 2; s++) {
            ok = ok && encode_planes<RS>(enc, &tm.m[TM_HALO0 + s], B.set[s].h, P, planes, Cols<RS>::rj, HALO_ROWS);
            ok = ok && encode_planes<RS>(enc, &tm.m[TM_CELL0 + s], B.set[s].h, P, planes, T_J, T_I);
            if (mixed)
                ok = ok && encode_planes<double>(enc, &tm.m[TM_CELLD0 + s], B.set[s].vinf, P, 1 + P.S, T_J, T_I);
            else
                ok = ok && encode_planes<double>(enc, &tm.m[TM_CELLD0 + s], B.set[s].h, P, planes, T_J, T_I);
        }
        ok = ok && encode_planes<double>(enc, &tm.m[TM_ZP], B.z[0], P, 3, R_J, ZP_ROWS);
        ok = ok && encode_planes<double>(enc, &tm.m[TM_ZC], B.z[0], P, 3, R_J, ZC_ROWS);
        if (B.ks) ok = ok && encode_planes<RS>(enc, &tm.m[TM_KS], B.ks, P, 1, T_J, T_I);
        return ok ? 0 : 2;
    }

    template <int MAXS, bool BUDGET, bool SM, bool TMA, int NS = 0>
    static void *update_fn() { return (void *)k_update_tile<PP, RS, MAXS, BUDGET, SM, TMA, NS>; }

    /* Kernels built for one class count (1..10): their class loops have no exit
     * tests, so the compiler interleaves the classes' independent quotient
     * chains, and their staging layout is constant (mixed form, 7 classes: -7 %
     * and -3.5 % against the kernels for up to 8).  Whether M_k is staged
     * follows from the count too: where it costs no resident blocks. */
    template <int NS>
    static constexpr bool exact_staged()
    {
        auto blocks = [](size_t bytes) {
            const size_t fit = 233472 / (bytes + 1024 + 256);     /* an SM's shared memory; 1 KB a block is the system's */
            return fit < (size_t)PP::kMinBlocks ? fit : (size_t)PP::kMinBlocks;
        };
        return blocks(StagedLayout::make(NS, sizeof(R), 1).total + 128) >= blocks(StagedLayout::make(NS, sizeof(R), 0).total + 128);
    }
    struct Exact {
        void *update = nullptr, *run = nullptr;
        int stage_m = 1;
    };
    template <int NS>
    static Exact exact_of()
    {
        constexpr bool sm = exact_staged<NS>();
        return Exact{update_fn<NS, false, sm, true, NS>(), (void *)k_run_tile<PP, RS, NS, sm, NS>, sm};
    }
    static Exact exact(int S)
    {
        switch (S) {
        case 1: return exact_of<1>();
        case 2: return exact_of<2>();
        case 3: return exact_of<3>();
        case 4: return exact_of<4>();
        case 5: return exact_of<5>();
        case 6: return exact_of<6>();
        case 7: return exact_of<7>();
        case 8: return exact_of<8>();
        case 9: return exact_of<9>();
        case 10: return exact_of<10>();
        default: return Exact();
        }
    }

    /* with budgets (tensor maps) */
    template <bool SM>
    static void *pick_budget(int S)
    {
        if (S == 7) return update_fn<8, true, SM, true, 7>();
        if (S == 10) return update_fn<16, true, SM, true, 10>();
        if (S <= 4) return update_fn<4, true, SM, true>();
        if (S <= 8) return update_fn<8, true, SM, true>();
        return update_fn<16, true, SM, true>();
    }
    /* without tensor maps (a driver that cannot encode them) */
    template <bool BUDGET, bool SM>
    static void *pick_copies(int S)
    {
        if (S <= 4) return update_fn<4, BUDGET, SM, false>();
        if (S <= 8) return update_fn<8, BUDGET, SM, false>();
        return update_fn<16, BUDGET, SM, false>();
    }
    template <bool SM>
    static void *pick_update(int S, bool budget, bool tma)
    {
        if (!tma) return budget ? pick_copies<true, SM>(S) : pick_copies<false, SM>(S);
        return budget ? pick_budget<SM>(S) : update_fn<16, false, SM, true>();
    }

    /* Policy::Wide's kernels (one instantiation, in a translation unit of its
     * own); M_k stays in global memory */
    static WideKernels wide_kernels()
    {
        typedef typename PP::Wide W;
        return WideKernels{(void *)k_wave_cells<W, RS>,
                           {{(void *)k_update_tile<W, RS, 16, false, false, false, 0>,
                             (void *)k_update_tile<W, RS, 16, true, false, false, 0>},
                            {(void *)k_update_tile<W, RS, 16, false, false, true, 0>,
                             (void *)k_update_tile<W, RS, 16, true, false, true, 0>}},
                           (void *)k_wave_batch<W, RS>,
                           {(void *)k_update_batch<W, RS, 16, false, false, 0, false>,
                            (void *)k_update_batch<W, RS, 16, true, false, 0, false>}};
    }

    static int configure(const DevParams &P, int num_sms, StepConfig &cfg, const WideKernels &wide)
    {
        const int64_t ntiles = (int64_t)((P.nx + T_I - 1) / T_I) * ((P.ny + T_J - 1) / T_J);
        void *fu = nullptr;
        void *fw = (void *)k_wave_cells<PP, RS>;
        size_t su = 0;
        const size_t sw = wave_smem();
        int occ_u = 0, occ_w = 0, stage_m = 1;
        const bool ordinary = PP::ordinary(P);
        const bool tma = cfg.tma != 0;
        cfg.tma = tma ? 1 : 0;
        const Exact x = ordinary && tma && !P.budget ? exact(P.S) : Exact();
        void *fr = nullptr;                    /* the many-step kernel of fu's layout */
        cudaError_t e;
        if (!ordinary) {
            fu = wide.update[tma][P.budget != 0];
            fw = wide.wave;
            stage_m = 0;
            su = update_smem(P.S, 0) + (tma ? 128 : 0);
            e = raise_smem_limit(fu, su);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_u, fu, TILE_THREADS, su);
        } else if (x.update) {
            fu = x.update;
            fr = x.run;
            stage_m = x.stage_m;
            su = update_smem(P.S, stage_m) + 128;
            e = raise_smem_limit(fu, su);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_u, fu, TILE_THREADS, su);
        } else {
            e = pick_staging(pick_update<true>(P.S, P.budget != 0, tma), pick_update<false>(P.S, P.budget != 0, tma), P.S, su,
                             occ_u, stage_m, fu, tma ? 128 : 0);
            if (tma && !P.budget)
                fr = stage_m ? (void *)k_run_tile<PP, RS, 16, true, 0> : (void *)k_run_tile<PP, RS, 16, false, 0>;
        }
        if (e != cudaSuccess) return (int)e;
        e = raise_smem_limit(fw, sw);
        if (e != cudaSuccess) return (int)e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_w, fw, TILE_THREADS, sw);
        if (e != cudaSuccess) return (int)e;
        if (occ_u < 1) occ_u = 1;
        if (occ_w < 1) occ_w = 1;
        cfg.grid_update = (int)(ntiles < (int64_t)num_sms * occ_u ? ntiles : (int64_t)num_sms * occ_u);
        cfg.grid_wave = (int)(ntiles < (int64_t)num_sms * occ_w ? ntiles : (int64_t)num_sms * occ_w);
        cfg.smem_update = su;
        cfg.smem_wave = sw;
        cfg.fn_update = fu;
        cfg.fn_wave = fw;
        cfg.stage_m = stage_m;
        cfg.fn_run = nullptr;
        if (fr && !P.has_solid && ntiles <= (int64_t)RUN_TILES_PER_SM * num_sms) {
            int occ = 0, coop = 0, dev = 0;
            e = raise_smem_limit(fr, su);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fr, TILE_THREADS, su);
            if (e == cudaSuccess) e = cudaGetDevice(&dev);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
            if (e != cudaSuccess) return (int)e;
            /* every block resident at once */
            if (coop && (int64_t)num_sms * occ >= cfg.grid_update) {
                cfg.fn_run = fr;
                cfg.smem_run = su;
            }
        }
        return 0;
    }

    template <int MAXS, bool BUDGET, bool SM, int NS, bool COMMON>
    static void *ubatch_fn() { return (void *)k_update_batch<PP, RS, MAXS, BUDGET, SM, NS, COMMON>; }

    /* batched kernel for exactly NS classes (every running scenario has NS):
     * M_k staged where that leaves the resident blocks the kernel is
     * register-budgeted for */
    template <int MAXS, int NS, bool COMMON>
    static cudaError_t exact_batch(bool budget, BatchConfig::Update &u)
    {
        constexpr int blocks = COMMON ? PP::kCommonMinBlocks : PP::kBatchMinBlocks;      /* as in k_update_batch */
        constexpr bool sm = NS == 7 || (NS == 10 && sizeof(RS) == 4 && blocks == 2);
        void *f = ubatch_fn<MAXS, false, sm, NS, COMMON>();
        if constexpr (!COMMON)
            if (budget) f = ubatch_fn<MAXS, true, sm, NS, COMMON>();
        u.smem_x[NS] = update_smem(NS, sm);
        cudaError_t e = raise_smem_limit(f, u.smem_x[NS]);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&u.occ_x[NS], f, TILE_THREADS, u.smem_x[NS]);
        if (u.occ_x[NS] < 1) u.occ_x[NS] = 1;
        u.fn_x[NS] = f;
        return e;
    }

    template <bool SM, bool COMMON>
    static void *pick_ub(int max_classes, bool budget)
    {
        if constexpr (!COMMON)
            if (budget) {
                if (max_classes <= 4) return ubatch_fn<4, true, SM, 0, false>();
                if (max_classes <= 8) return ubatch_fn<8, true, SM, 0, false>();
                return ubatch_fn<16, true, SM, 0, false>();
            }
        if (max_classes <= 4) return ubatch_fn<4, false, SM, 0, COMMON>();
        if (max_classes <= 8) return ubatch_fn<8, false, SM, 0, COMMON>();
        return ubatch_fn<16, false, SM, 0, COMMON>();
    }

    template <bool COMMON>
    static cudaError_t configure_updates(int max_classes, bool budget, BatchConfig::Update &u)
    {
        void *with = pick_ub<true, COMMON>(max_classes, budget), *without = pick_ub<false, COMMON>(max_classes, budget);
        cudaError_t e = cudaSuccess;
        for (int S = 0; S <= 16 && e == cudaSuccess; S++) {
            const int Sc = S < 1 ? 1 : (S > max_classes ? max_classes : S);
            int stage_m = 1;
            e = pick_staging(with, without, Sc, u.smem_s[S], u.occ_s[S], stage_m, u.fn_s[S]);
        }
        if (e == cudaSuccess && max_classes >= 7) e = exact_batch<8, 7, COMMON>(budget, u);
        if (e == cudaSuccess && max_classes >= 10) e = exact_batch<16, 10, COMMON>(budget, u);
        /* limits for the largest shape either kernel is launched with */
        if (e == cudaSuccess)
            e = raise_smem_limit(with, update_smem(max_classes));
        if (e == cudaSuccess)
            e = raise_smem_limit(without, update_smem(max_classes, 0));
        return e;
    }

    /* the wide kernels of a pool, once it has a scenario that needs them (to load
     * them costs 50 ms) */
    static int configure_batch_wide(int max_classes, bool budget, BatchConfig &cfg, const WideKernels &wide)
    {
        void *f = wide.update_batch[budget];
        cudaError_t e = raise_smem_limit(f, update_smem(max_classes, 0));
        for (int S = 0; S <= 16 && e == cudaSuccess; S++) {
            BatchConfig::Update &u = cfg.wide;
            u.fn_s[S] = f;
            u.smem_s[S] = update_smem(S < 1 ? 1 : (S > max_classes ? max_classes : S), 0);
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&u.occ_s[S], f, TILE_THREADS, u.smem_s[S]);
            if (u.occ_s[S] < 1) u.occ_s[S] = 1;
        }
        cfg.fn_wave_wide = wide.wave_batch;
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cfg.occ_wave_wide, wide.wave_batch, TILE_THREADS, wave_smem());
        if (cfg.occ_wave_wide < 1) cfg.occ_wave_wide = 1;
        return (int)e;
    }

    static int configure_batch(int max_classes, bool budget, BatchConfig &cfg)
    {
        void *fw = (void *)k_wave_batch<PP, RS>;
        const size_t sw = wave_smem();
        cudaError_t e = raise_smem_limit(fw, sw);
        if (e != cudaSuccess) return (int)e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cfg.occ_wave, fw, TILE_THREADS, sw);
        if (e != cudaSuccess) return (int)e;
        if (cfg.occ_wave < 1) cfg.occ_wave = 1;
        e = configure_updates<false>(max_classes, budget, cfg.own);
        if (e == cudaSuccess && !budget) e = configure_updates<true>(max_classes, budget, cfg.common);
        if (e != cudaSuccess) return (int)e;
        cfg.fn_wave = fw;
        cfg.smem_wave = sw;
        cfg.threads = TILE_THREADS;
        cfg.tile_i = T_I;
        cfg.tile_j = T_J;
        return 0;
    }

    static int launch(const DevParams &P, const BufsT<RS> &B, Ctl *ctl, const double *rain, double *partials,
                      double *stage, double *saveflow, const TmaMaps &tm, const StepConfig &cfg, cudaStream_t s,
                      cudaEvent_t ev0, cudaEvent_t ev1)
    {
        void *wargs[] = {(void *)&P, (void *)&B, (void *)&ctl};
        cudaLaunchKernel(cfg.fn_wave, dim3(cfg.grid_wave), dim3(TILE_THREADS), wargs, cfg.smem_wave, s);
        if (ev0) cudaEventRecord(ev0, s);
        void *args[] = {(void *)&P, (void *)&B, (void *)&ctl, (void *)&rain, (void *)&partials, (void *)&stage,
                        (void *)&saveflow, (void *)&tm};
        cudaLaunchKernel(cfg.fn_update, dim3(cfg.grid_update), dim3(TILE_THREADS), args, cfg.smem_update, s);
        if (ev1) cudaEventRecord(ev1, s);
        return (int)cudaGetLastError();
    }

    static int launch_run(const DevParams &P, const BufsT<RS> &B, Ctl *ctl, const double *rain, double *stage, double *saveflow, const TmaMaps &tm, const StepConfig &cfg, int steps,
                          cudaStream_t s)
    {
        void *args[] = {(void *)&P, (void *)&B, (void *)&ctl, (void *)&rain, (void *)&stage,
                        (void *)&saveflow, (void *)&tm, (void *)&steps};
        return (int)cudaLaunchCooperativeKernel(cfg.fn_run, dim3(cfg.grid_update), dim3(TILE_THREADS), args, cfg.smem_run, s);
    }

    /* the two passes of a step one at a time (a slab of a split domain takes
     * the largest wave speed over every slab between them) */
    static int launch_wave(const DevParams &P, const BufsT<RS> &B, Ctl *ctl, const StepConfig &cfg, cudaStream_t s)
    {
        void *wargs[] = {(void *)&P, (void *)&B, (void *)&ctl};
        cudaLaunchKernel(cfg.fn_wave, dim3(cfg.grid_wave), dim3(TILE_THREADS), wargs, cfg.smem_wave, s);
        return (int)cudaGetLastError();
    }

    static int launch_update(const DevParams &P, const BufsT<RS> &B, Ctl *ctl, const double *rain, double *partials,
                             double *stage, double *saveflow, const TmaMaps &tm, const StepConfig &cfg, cudaStream_t s)
    {
        void *args[] = {(void *)&P, (void *)&B, (void *)&ctl, (void *)&rain, (void *)&partials, (void *)&stage,
                        (void *)&saveflow, (void *)&tm};
        cudaLaunchKernel(cfg.fn_update, dim3(cfg.grid_update), dim3(TILE_THREADS), args, cfg.smem_update, s);
        return (int)cudaGetLastError();
    }
};

}  // inline namespace SWEHR_TILE_NS
}  // namespace swehr
