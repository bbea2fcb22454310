// lbm_ops_impl.cuh — the storage-typed work of a single domain (initial
// state, the pull and AA step loops, import and export), written once as
// templates and instantiated for one storage format per translation unit
// (lbm_ops_f32.cu, lbm_ops_f16.cu, lbm_ops_bf16.cu, lbm_ops_f64.cu), so that
// the kernels of the four formats compile in parallel.
#pragma once
#include "lbm_domain.cuh"
#include "lbm_quad.cuh"

namespace lbm {

template <class S>
int ops_tensor_maps(lbm_domain* d, int sm_count) {
  return domain_tensor_maps<S>(d, sm_count);
}

// k_init: pull form: arF_0 in lat[1], its collision in lat[0]; AA: arF_0 in
// the natural layout of lat[0], collided by the first step
template <class S>
int ops_launch_init(lbm_domain* d, cudaStream_t st) {
  const InitParams ip = init_params(d);
  return with_model<S>(d, [&](auto coll, auto les) -> int {
    // pull: arF_0 in lat[1], its collision in lat[0]; AA: arF_0 in the
    // natural layout of lat[0], collided by the first step
    const bool aa = d->opt.stream_mode == LBM_STREAM_AA;
    StepArgs<S> a = make_args<S>(d, nullptr, d->lat[aa ? 0 : 1], 0);
    a.den_out = d->den[0];
    a.ux_out = d->ux;
    a.uy_out = d->uy;
    a.uz_out = d->uz;
    const dim3 b = block_of(d->g.nx), gr = grid_of(d->g, b);
    k_init<S, decltype(coll)::value, decltype(les)::value>
        <<<gr, b, 0, st>>>(a, aa ? nullptr : (S*)d->lat[0], ip);
    CK(cudaGetLastError());
    return LBM_OK;
  });
}

template <class S>
int ops_run_pull(lbm_domain* d, int nsteps) {
  return with_model<S>(d, [&](auto coll, auto les) -> int {
    return issue_run(
        d, nsteps,
        // the last two steps write rho, the last one u
        [&](cudaStream_t st, int cur, long long k, int left) {
          StepArgs<S> a = make_args<S>(d, d->lat[cur], d->lat[cur ^ 1], k);
          if (left < 2) a.den_out = d->den[k & 1];
          if (left == 0) {
            a.ux_out = d->ux;
            a.uy_out = d->uy;
            a.uz_out = d->uz;
          }
          return launch_step<S, decltype(coll)::value, decltype(les)::value>(d, a, st);
        },
        [](cudaStream_t, int, long long) { return cudaSuccess; });
  });
}

// rho and u of the AA state after step `step` (layout cur) into den[step & 1]
// and u; the face buffers are those of AA step s (k = s + 1)
template <class S>
cudaError_t aa_macro_on(lbm_domain* d, cudaStream_t st, int cur, long long step, int entry) {
  StepArgs<S> m = aa_args<S>(d, step + 1, false, cur);
  m.den_out = d->den[step & 1];
  m.ux_out = d->ux;
  m.uy_out = d->uy;
  m.uz_out = d->uz;
  const dim3 gf = flat_grid(d->g), bf(kFlat);
  if constexpr (kDev<S>) {
    if (d->g.rows == kRowsQuad)
      return cur ? launch_chained(k_aa_words<S, COLL_SRT, false, false, 1, true>,
                                  aa_neighbor_grid(d->g), bf, st, m, entry)
                 : launch_chained(k_aa_words<S, COLL_SRT, false, false, 0, true>, gf, bf, st, m,
                                  entry);
  }
  return cur ? launch_chained(k_aa_macro<S, 1>, gf, bf, st, m, entry)
             : launch_chained(k_aa_macro<S, 0>, gf, bf, st, m, entry);
}

template <class S>
int ops_aa_macro(lbm_domain* d) {
  return launch_status(
      aa_macro_on<S>(d, d->stream, d->cur, d->step, d->post_direct ? kAAComplete : kAAPending),
      "rho and u");
}

template <class S>
int ops_run_aa(lbm_domain* d, int nsteps) {
  return with_model<S>(d, [&](auto coll, auto les) -> int {
    constexpr int C = decltype(coll)::value;
    constexpr bool L = decltype(les)::value;
    auto args = [&](long long k, bool den, int neighbor) {
      return aa_args<S>(d, k, den, neighbor);
    };
    // quad rows (16-bit): k_aa_words, one word of four nodes per thread,
    // except the first step after the initial state (a local step, whose
    // slots are all at the node: the per-node step over quad rows)
    [[maybe_unused]] bool words = false;
    const dim3 bf(kFlat);
    const dim3 ga((unsigned)(((long long)d->g.px * d->g.nz + kFlat - 1) / kFlat), d->g.ny, 1);
    [[maybe_unused]] dim3 gw(1, 1, 1), gn(1, 1, 1);
    if constexpr (kDev<S>) {
      if (d->g.rows != kRowsPlain) {
        if (!aa_words_apply(d->g))
          return set_error(LBM_ERR_INVALID, "AA domain rows without the word step");
        words = true;
        gw = flat_grid(d->g);
        gn = aa_neighbor_grid(d->g);
      }
    }
    auto launch = [&](cudaStream_t st, const StepArgs<S>& a, int nb, int entry) -> cudaError_t {
      if constexpr (kDev<S>) {
        if (words && entry != kAAFromInit) {
          if (a.sr)
            return nb ? launch_chained(k_aa_words<S, C, L, true, 1>, gn, bf, st, a, entry)
                      : launch_chained(k_aa_words<S, C, L, true, 0>, gw, bf, st, a, entry);
          return nb ? launch_chained(k_aa_words<S, C, L, false, 1>, gn, bf, st, a, entry)
                    : launch_chained(k_aa_words<S, C, L, false, 0>, gw, bf, st, a, entry);
        }
        if (words) {
          StepArgs<S> an = a;  // one node per item
          an.ri = d->g.px;
          an.mrow = ~0ull / (unsigned long long)an.ri + 1;
          return launch_chained(k_aa_step<S, C, L, 0>, ga, bf, st, an, entry);
        }
      }
      return nb ? launch_chained(k_aa_step<S, C, L, 1>, ga, bf, st, a, entry)
                : launch_chained(k_aa_step<S, C, L, 0>, ga, bf, st, a, entry);
    };
    // the first step from a complete natural layout (initial state, import)
    // has its own entry mode: never inside a graph
    int left = nsteps;
    if (d->aa_first || d->post_direct) {
      const int rc = launch_status(launch(d->stream, args(d->step + 1, left <= 2, 0), 0,
                                          d->aa_first ? kAAFromInit : kAAComplete),
                                   "a step");
      if (rc) return rc;
      d->aa_first = false;
      d->post_direct = false;
      d->cur = 1;
      ++d->step;
      if (--left == 0) return ops_aa_macro<S>(d);
    }
    return issue_run(
        d, left,
        // the last two steps write the rho of their input arF (the previous-step
        // density of the residual); rho and u of the final arF follow
        [&](cudaStream_t st, int cur, long long k, int todo) {
          return launch(st, args(k, todo < 2, cur), cur, kAAPending);
        },
        [&](cudaStream_t st, int cur, long long k) {
          return aa_macro_on<S>(d, st, cur, k, kAAPending);
        });
  });
}

// k_import from d->staging (the AoS arF already on the device)
template <class S>
int ops_import(lbm_domain* d, int padded) {
  return with_model<S>(d, [&](auto coll, auto les) -> int {
    const bool aa = d->opt.stream_mode == LBM_STREAM_AA;
    StepArgs<S> a = make_args<S>(d, nullptr, d->lat[aa ? 0 : 1], 0);
    a.den_out = d->den[0];
    a.ux_out = d->ux;
    a.uy_out = d->uy;
    a.uz_out = d->uz;
    const dim3 b = block_of(d->g.nx), gr = grid_of(d->g, b);
    k_import<S, decltype(coll)::value, decltype(les)::value>
        <<<gr, b, 0, d->stream>>>(a, d->staging, padded, aa ? nullptr : (S*)d->lat[0]);
    CK(cudaGetLastError());
    return LBM_OK;
  });
}

// k_export into d->staging
template <class S>
int ops_export(lbm_domain* d, int padded) {
  const bool aa = d->opt.stream_mode == LBM_STREAM_AA;
  // AA: the face buffers of AA step s are those of make_args with k = s + 1
  StepArgs<S> a = make_args<S>(d, d->lat[aa ? 0 : d->cur ^ 1], nullptr, d->step + (aa ? 1 : 0));
  const int mode = aa ? (d->cur ? kExportAASwapped
                                : (d->post_direct ? kExportDirect : kExportAANaturalPending))
                      : (d->post_direct ? kExportDirect : kExportPull);
  const dim3 b = block_of(d->g.nx), gr = grid_of(d->g, b);
  k_export<S><<<gr, b, 0, d->stream>>>(a, d->staging, padded, mode);
  CK(cudaGetLastError());
  return LBM_OK;
}

template <class S>
StorageOps make_ops() {
  StorageOps o;
  o.tensor_maps = &ops_tensor_maps<S>;
  o.launch_init = &ops_launch_init<S>;
  o.run_pull = &ops_run_pull<S>;
  o.run_aa = &ops_run_aa<S>;
  o.import_staging = &ops_import<S>;
  o.export_staging = &ops_export<S>;
  o.aa_macro = &ops_aa_macro<S>;
  return o;
}

}  // namespace lbm
