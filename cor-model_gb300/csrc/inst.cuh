// inst.cuh -- instantiates the kernels of one model set and its ModelOps.
#pragma once

#include <cstddef>

#include "model_ops.h"

#define COR_MODEL_INSTANCE(NAME, I, E, C)                                                                  \
    namespace cor {                                                                                        \
    using MS_##NAME = ModelSet<I, E, C>;                                                                   \
    static cudaError_t occ_##NAME(int* n) {                                                                \
        cudaError_t e = cudaFuncSetAttribute(trace_kernel<MS_##NAME, kTraceThreads>,                       \
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRegroupSmem); \
        if (e != cudaSuccess) return e;                                                                    \
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, trace_kernel<MS_##NAME, kTraceThreads>,    \
                                                             kTraceThreads, kRegroupSmem);                 \
    }                                                                                                      \
    static cudaError_t gen_##NAME(const TraceArgs& a, unsigned blocks, cudaStream_t s) {                   \
        cudaError_t e = cudaFuncSetAttribute(trace_kernel<MS_##NAME, kTraceThreads>,                       \
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRegroupSmem); \
        if (e != cudaSuccess) return e;                                                                    \
        trace_kernel<MS_##NAME, kTraceThreads><<<blocks, kTraceThreads, kRegroupSmem, s>>>(a);             \
        return cudaGetLastError();                                                                         \
    }                                                                                                      \
    static cudaError_t socc_##NAME(int* n) {                                                               \
        cudaError_t e = cudaFuncSetAttribute(stream_kernel<MS_##NAME>,                                     \
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRegroupSmem); \
        if (e != cudaSuccess) return e;                                                                    \
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, stream_kernel<MS_##NAME>, kTraceThreads,   \
                                                             kRegroupSmem);                              \
    }                                                                                                      \
    static cudaError_t stream_##NAME(const StreamArgs& a, unsigned blocks, cudaStream_t s) {               \
        cudaError_t e = cudaFuncSetAttribute(stream_kernel<MS_##NAME>,                                     \
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRegroupSmem); \
        if (e != cudaSuccess) return e;                                                                    \
        stream_kernel<MS_##NAME><<<blocks, kTraceThreads, kRegroupSmem, s>>>(a);                         \
        return cudaGetLastError();                                                                         \
    }                                                                                                      \
    static cudaError_t field_##NAME(const DevParams* p, int np, const int32_t* idx, const double* pos,     \
                                    int64_t n, double* out, CrustalTables crust, cudaStream_t s) {         \
        int dev = 0, sms = 1, per_sm = 1;                                                                  \
        cudaError_t e = cudaGetDevice(&dev);                                                               \
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);       \
        if (e == cudaSuccess)                                                                              \
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, field_kernel<MS_##NAME>, kFieldThreads, 0); \
        if (e != cudaSuccess) return e;                                                                    \
        const int64_t resident = (int64_t)sms * (per_sm > 0 ? per_sm : 1);                                 \
        const int64_t per_warp = (n + 4 * resident - 1) / (4 * resident);                                  \
        const int per_thread =                                                                             \
            E == 0 && n >= (int64_t)sms * 2 * kFieldThreads * kFieldPerThread ? kFieldPerThread : 1;       \
        const int64_t per_block = C != 0 ? 4 * per_warp : (int64_t)kFieldThreads * per_thread;             \
        const unsigned blocks = (unsigned)((n + per_block - 1) / per_block);                               \
        field_kernel<MS_##NAME><<<blocks, kFieldThreads, 0, s>>>(p, np, idx, pos, n, out, crust, per_warp, \
                                                                 per_thread);                              \
        return cudaGetLastError();                                                                         \
    }                                                                                                      \
    static cudaError_t tables_##NAME(const T96Tables* t96, const TS05Tables* ts05) {                       \
        /* only what the set's kernels read: a copy takes about 8 us of cor_ctx_create */                  \
        cudaError_t e = cudaSuccess;                                                                       \
        if (E != COR_EXTERNAL_NONE && E != COR_EXTERNAL_TS05) {                                            \
            e = cudaMemcpyToSymbol(c_t96, t96, sizeof(T96Tables));                                         \
            if (e == cudaSuccess && C == 0) e = cudaMemcpyToSymbol(g_t96, t96, sizeof(T96Tables));         \
        }                                                                                                  \
        if (e == cudaSuccess && E != COR_EXTERNAL_NONE && E != COR_EXTERNAL_T96) {                         \
            e = cudaMemcpyToSymbol(c_ts05, ts05, sizeof(TS05Tables));                                      \
            if (e == cudaSuccess && C == 0) e = cudaMemcpyToSymbol(g_ts05, ts05, sizeof(TS05Tables));      \
        }                                                                                                  \
        return e;                                                                                          \
    }                                                                                                      \
    template <class MS, bool TEAM = MS::crustal == 0>                                                      \
    struct Team_##NAME {                                                                                   \
        /* the functions' limit is the device's, not the context's: every call of every thread sets the  */\
        /* same one, that of the most slots, whatever its own launch needs                               */\
        static constexpr size_t kLimit = kTeamSlotsOf<MS> * sizeof(TeamSlot<MS>);                          \
        template <class F>                                                                                 \
        static cudaError_t limit(F* kernel) {                                                              \
            return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLimit); \
        }                                                                                                  \
        static cudaError_t occ(int* n_slots, int* n) {                                                     \
            *n_slots = kTeamSlotsOf<MS>;                                                                   \
            const cudaError_t e = limit(team_trace_kernel<MS>);                                            \
            if (e != cudaSuccess) return e;                                                                \
            return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, team_trace_kernel<MS>, kTeamThreads, kLimit);\
        }                                                                                                  \
        static cudaError_t run(const TraceArgs& a, int n_slots, unsigned blocks, cudaStream_t s) {         \
            const size_t smem = (size_t)n_slots * sizeof(TeamSlot<MS>);                                    \
            const cudaError_t e = limit(team_trace_kernel<MS>);                                            \
            if (e != cudaSuccess) return e;                                                                \
            team_trace_kernel<MS><<<blocks, team_threads(n_slots), smem, s>>>(a, n_slots);                 \
            return cudaGetLastError();                                                                     \
        }                                                                                                  \
        static cudaError_t field(const DevParams* p, int np, const int32_t* idx, const double* pos, int64_t n,\
                                 double* out, int n_slots, unsigned blocks, cudaStream_t s) {              \
            const size_t smem = (size_t)n_slots * sizeof(TeamSlot<MS>);                                    \
            const cudaError_t e = limit(team_field_kernel<MS>);                                            \
            if (e != cudaSuccess) return e;                                                                \
            team_field_kernel<MS><<<blocks, team_threads(n_slots), smem, s>>>(p, np, idx, pos, n, out, n_slots);\
            return cudaGetLastError();                                                                     \
        }                                                                                                  \
        static cudaError_t load() {                                                                        \
            const cudaError_t e = limit(team_trace_kernel<MS>);                                            \
            return e != cudaSuccess ? e : limit(team_field_kernel<MS>);                                    \
        }                                                                                                  \
        static constexpr auto occ_ptr = &occ;                                                              \
        static constexpr auto field_ptr = &field;                                                          \
        static constexpr auto run_ptr = &run;                                                              \
    };                                                                                                     \
    template <class MS>                                                                                    \
    struct Team_##NAME<MS, false> {                                                                        \
        static cudaError_t load() { return cudaSuccess; }                                                  \
        static constexpr std::nullptr_t occ_ptr = nullptr;                                                 \
        static constexpr std::nullptr_t run_ptr = nullptr;                                                 \
        static constexpr std::nullptr_t field_ptr = nullptr;                                               \
    };                                                                                                     \
    template <class MS, bool HALVES = kPlain<MS>>                                                          \
    struct Halves_##NAME {                                                                                 \
        static cudaError_t run(const TraceArgs& a, unsigned blocks, cudaStream_t s) {                      \
            constexpr int T = kTraceThreads / 2;                                                           \
            constexpr size_t smem = sizeof(RegroupScratchOf<T>);                                           \
            cudaError_t e = cudaFuncSetAttribute(trace_kernel<MS, T>,                                      \
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
            if (e != cudaSuccess) return e;                                                                \
            trace_kernel<MS, T><<<blocks, T, smem, s>>>(a);                                                \
            return cudaGetLastError();                                                                     \
        }                                                                                                  \
        static cudaError_t load() {                                                                        \
            cudaFuncAttributes at;                                                                         \
            return cudaFuncGetAttributes(&at, trace_kernel<MS, kTraceThreads / 2>);                        \
        }                                                                                                  \
        static constexpr auto ptr = &run;                                                                  \
    };                                                                                                     \
    template <class MS>                                                                                    \
    struct Halves_##NAME<MS, false> {                                                                      \
        static cudaError_t load() { return cudaSuccess; }                                                  \
        static constexpr std::nullptr_t ptr = nullptr;                                                     \
    };                                                                                                     \
    static cudaError_t load_##NAME() {                                                                     \
        cudaFuncAttributes at;                                                                             \
        int n = 0;                                                                                         \
        cudaError_t e = occ_##NAME(&n);                                                                    \
        if (e == cudaSuccess) e = socc_##NAME(&n);                                                         \
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, field_kernel<MS_##NAME>);                     \
        if (e == cudaSuccess) e = Team_##NAME<MS_##NAME>::load();                                          \
        if (e == cudaSuccess) e = Halves_##NAME<MS_##NAME>::load();                                        \
        return e;                                                                                          \
    }                                                                                                      \
    const ModelOps ops_##NAME = {I * 100 + E * 10 + C, occ_##NAME, gen_##NAME, field_##NAME, tables_##NAME, \
                                 socc_##NAME, stream_##NAME, Team_##NAME<MS_##NAME>::occ_ptr,               \
                                 Team_##NAME<MS_##NAME>::run_ptr, Team_##NAME<MS_##NAME>::field_ptr,         \
                                 Halves_##NAME<MS_##NAME>::ptr, load_##NAME};                              \
    }
