// Launch helpers of pk_kernel: one instantiation per (value type, model, derivatives, operation count, coset size,
// sign group); the translation units dsf_pk_*.cu hold the instantiations.
#pragma once
#include "dsf_pk_kernel.cuh"

namespace dsf {

// the symmetry form of a launch: n_sym operations in cosets of cs that form the sign group pat (cs = 4: kPatD2,
// kPatC2hB; cs = 2: the mask of the axes that the second operation flips); inv: the second half of the operations
// are the images of the first half under an inversion at the origin; cen: the engine takes an inversion at the origin
// beside them (HC; the common groups: -1, 2/m, mmm -- others run the general kernels, which are right for them too)
struct PkForm {
    int n_sym = 0, cs = 0, pat = 0;
    bool inv = false, cen = false;
};

struct PkArgs {
    const DevStructure *S = nullptr;
    const CallBuffers *C = nullptr;
    const PkLaunch *L = nullptr;
    const PkBatch *B = nullptr;  // a batched launch of `blocks` blocks instead of one structure's
    PkForm form;
    bool split_kinds = false;    // one launch per ADP kind
    int n_tiles = 0, n_chunks = 0, blocks = 0;
    size_t smem = 0;
    cudaStream_t st = nullptr;
};

constexpr int kPat2Y = 5, kPat2Z = 3, kPatInv = 7;  // cs = 2: a two-fold axis along b, along c, an inversion

// runs f with the compile-time form that equals `f0`, one of the compiled ones of the model; false when none does.
//   HC (operations without the inversion): P1 and P-1; P2_1, P2_1/c, C2/c; P4_1; 222; 422
//   other models (all operations modulo centring): 1; 2; -1; 222; 2/m; mmm; any eight.  Eight in no compiled coset
//   form (P4_3 2_1 2 as listed, 4/m) against sf_grad_body, independent atoms: FP32, 2,000 atoms, 50,021 reflections
//   1,448 -> 1,130 us (isotropic 867 -> 770); FP64, 500 atoms, 10,001 reflections 7,762 -> 2,798 us; tabulated in FP64,
//   150 atoms, 20,021 reflections 5,484 -> 2,790 us
template <int N_, int CS_, int PAT_, bool INV_ = false, bool CEN_ = false>
struct PkC {
    static constexpr int N = N_, CS = CS_, PAT = PAT_;
    static constexpr bool INV = INV_, CEN = CEN_;
};
template <typename C>
inline bool pk_is(const PkForm &f)
{
    return f.n_sym == C::N && f.cs == C::CS && (C::CS == 1 || f.pat == C::PAT) && f.inv == C::INV && f.cen == C::CEN;
}
template <bool CEN, typename F>
inline bool pk_hc_form_of(const PkForm &f, F &&go)
{
    if (pk_is<PkC<1, 1, 0, false, CEN> >(f)) return go(PkC<1, 1, 0, false, CEN>{}), true;
    if (pk_is<PkC<2, 2, kPat2Y, false, CEN> >(f)) return go(PkC<2, 2, kPat2Y, false, CEN>{}), true;
    if (pk_is<PkC<4, 4, kPatD2, false, CEN> >(f)) return go(PkC<4, 4, kPatD2, false, CEN>{}), true;
    if constexpr (!CEN) {
        if (pk_is<PkC<4, 2, kPat2Z> >(f)) return go(PkC<4, 2, kPat2Z>{}), true;
        if (pk_is<PkC<8, 4, kPatD2> >(f)) return go(PkC<8, 4, kPatD2>{}), true;
    }
    return false;
}
template <typename F>
inline bool pk_hc_form(const PkForm &f, F &&go)
{
    return f.cen ? pk_hc_form_of<true>(f, go) : pk_hc_form_of<false>(f, go);
}
template <typename F>
inline bool pk_generic_form(const PkForm &f, F &&go)
{
    if (pk_is<PkC<1, 1, 0> >(f)) return go(PkC<1, 1, 0>{}), true;
    if (pk_is<PkC<2, 2, kPat2Y> >(f)) return go(PkC<2, 2, kPat2Y>{}), true;
    if (pk_is<PkC<2, 2, kPatInv, true> >(f)) return go(PkC<2, 2, kPatInv, true>{}), true;
    if (pk_is<PkC<4, 4, kPatD2> >(f)) return go(PkC<4, 4, kPatD2>{}), true;
    if (pk_is<PkC<4, 4, kPatC2hB, true> >(f)) return go(PkC<4, 4, kPatC2hB, true>{}), true;
    if (pk_is<PkC<8, 4, kPatD2, true> >(f)) return go(PkC<8, 4, kPatD2, true>{}), true;
    if (pk_is<PkC<8, 1, 0> >(f)) return go(PkC<8, 1, 0>{}), true;
    return false;
}

template <typename K>
cudaError_t launch_pk_tiles(K k, int threads, int n_tiles, const PkArgs &A)
{
    if (n_tiles <= 0) return cudaSuccess;
    cudaError_t e = allow_dynamic_smem(k, A.smem);
    if (e != cudaSuccess) return e;
    k<<<A.n_chunks * n_tiles, threads, A.smem, A.st>>>(*A.S, *A.C, *A.L);
    return cudaGetLastError();
}

template <typename V, int MODEL, bool MP, bool GRAD, typename C>
cudaError_t launch_pk(const PkArgs &A)
{
    constexpr int TH = pk_threads<V>();
    if constexpr (sizeof(V) != sizeof(double) || VTraits<V>::NA == 2) {
        if (A.split_kinds) {
            const cudaError_t e = launch_pk_tiles(pk_kernel<V, MODEL, MP, C::N, C::CS, GRAD, C::INV, C::PAT, C::CEN, 0>, TH,
                                                  A.L->T.n_plain, A);
            if (e != cudaSuccess) return e;
            return launch_pk_tiles(pk_kernel<V, MODEL, MP, C::N, C::CS, GRAD, C::INV, C::PAT, C::CEN, 1>, TH,
                                   A.n_tiles - A.L->T.n_plain, A);
        }
    }
    return launch_pk_tiles(pk_kernel<V, MODEL, MP, C::N, C::CS, GRAD, C::INV, C::PAT, C::CEN, 2>, TH, A.n_tiles, A);
}

template <typename V, int MODEL, typename C>
cudaError_t launch_pk_batch(const PkArgs &A)
{
    auto k = pk_batch_kernel<V, MODEL, C::N, C::CS, C::INV, C::PAT, C::CEN>;
    cudaError_t e = allow_dynamic_smem(k, A.smem);
    if (e != cudaSuccess) return e;
    k<<<A.blocks, pk_threads<V>(), A.smem, A.st>>>(*A.B);
    return cudaGetLastError();
}

// a form's launch, cudaErrorInvalidValue where the form is not compiled (the engine asks pk_compiled first)
template <typename V, int MODEL, bool MP, bool GRAD>
cudaError_t dispatch_pk(const PkArgs &A)
{
    cudaError_t e = cudaErrorInvalidValue;
    auto go = [&](auto c) { e = launch_pk<V, MODEL, MP, GRAD, decltype(c)>(A); };
    if constexpr (MODEL == MODEL_HC) pk_hc_form(A.form, go);
    else pk_generic_form(A.form, go);
    return e;
}

template <typename V, int MODEL>
cudaError_t dispatch_pk_batch(const PkArgs &A)
{
    cudaError_t e = cudaErrorInvalidValue;
    auto go = [&](auto c) { e = launch_pk_batch<V, MODEL, decltype(c)>(A); };
    if constexpr (MODEL == MODEL_HC) pk_hc_form(A.form, go);
    else pk_generic_form(A.form, go);
    return e;
}

// per-translation-unit entries
cudaError_t launch_pk_f64_hc(const PkArgs &A);
cudaError_t launch_pk_f64_hc_mp(const PkArgs &A);
cudaError_t launch_pk_f64_hc_f(const PkArgs &A);
cudaError_t launch_pk_f64_iam(const PkArgs &A);
cudaError_t launch_pk_f64_table(const PkArgs &A);
cudaError_t launch_pk_f32_hc(const PkArgs &A);
cudaError_t launch_pk_f32_hc_f(const PkArgs &A);
cudaError_t launch_pk_f32_iam(const PkArgs &A);
cudaError_t launch_pk_f32_iam_f(const PkArgs &A);
cudaError_t launch_pk_f32_hc_mp(const PkArgs &A);
cudaError_t launch_pk_f32_hc_batch(const PkArgs &A);
cudaError_t launch_pk_f32_hc1(const PkArgs &A);
cudaError_t launch_pk_f32_hc1_f(const PkArgs &A);
cudaError_t launch_pk_f32_hc1_batch(const PkArgs &A);
cudaError_t launch_pk_f32_iam_batch(const PkArgs &A);

// record tables (dsf_prep_kernels.cu): kind 0: F2 slots (duplicated floats), 1: float slots, 2: double slots
cudaError_t launch_pk_prep(const DevStructure &S, int n_hkl_pad, int cs, int kind, void *out, cudaStream_t st);

}  // namespace dsf
