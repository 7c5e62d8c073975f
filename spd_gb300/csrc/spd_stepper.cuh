// Launch sequence of one SD-ADER step for dimension D and degree P
// (src/sdader_simulator.py:361-378); instantiated in spd_step.cu.
#pragma once
#include "spd_ctx.cuh"

namespace spd_host {

template <int D, int P>
int adjoint_vjp(spd_ctx* C);

template <int D, int P>
struct CmaxOnly {
static __device__ __forceinline__ void run(Blk B, const Geo& g, const double* __restrict__ W_cv,
                                           unsigned long long* __restrict__ cmax_bits, int* __restrict__ nan_flag) {
  constexpr int P_ = D + 1;
  const long long q = B.id * (long long)blockDim.x + threadIdx.x;
  double cval = 0.0;
  bool isnan_c = false;
  if (q < g.Nq) {
    double c = sound_speed(W_cv[(long long)P_ * g.Nq + q], W_cv[q], g.gamma, g.min_c2) * (double)D;
#pragma unroll
    for (int v = 1; v <= D; ++v) c = c + abs_bits(W_cv[(long long)v * g.Nq + q]);
    if (nan_w(c)) isnan_c = true;
    else cval = c;
  }
  // the warp's maximum (comparisons on the integer keys)
  for (int off = 16; off > 0; off >>= 1) {
    const double o = __shfl_down_sync(0xffffffffu, cval, off);
    cval = fgt(o, cval) ? o : cval;
  }
  const unsigned nb = __ballot_sync(0xffffffffu, isnan_c);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(cmax_bits, (unsigned long long)__double_as_longlong(cval));
    if (nb) atomicOr(nan_flag, 1);
  }
}
};
template <int D, int P>
__global__ void k_cmax_only(Geo g, const double* __restrict__ W_cv, unsigned long long* __restrict__ cmax_bits,
                            int* __restrict__ nan_flag) {
  CmaxOnly<D, P>::run(hw_blk(), g, W_cv, cmax_bits, nan_flag);
}

template <int D>
struct PrimOnly {
  static __device__ __forceinline__ void run(Blk B, const Geo& g, const double* __restrict__ U_cv,
                                             double* __restrict__ W_cv) {
    constexpr int V = D + 2;
    const long long q = B.id * (long long)blockDim.x + threadIdx.x;
    if (q >= g.Nq) return;
    double u[V], W[V];
#pragma unroll
    for (int v = 0; v < V; ++v) u[v] = U_cv[(long long)v * g.Nq + q];
    prims<D>(u, W, g.gamma, g.iso != 0);
#pragma unroll
    for (int v = 0; v < V; ++v) W_cv[(long long)v * g.Nq + q] = W[v];
  }
};
template <int D>
__global__ void k_prim_only(Geo g, const double* __restrict__ U_cv, double* __restrict__ W_cv) {
  PrimOnly<D>::run(hw_blk(), g, U_cv, W_cv);
}


template <int D, int P>
struct Stepper : StepperBase {
  using k = K<D, P>;

  // Block shape of the interior kernel: ``cells`` x rows, up to
  // INTERIOR_THREADS threads.  Its shared memory per cell is the tile of
  // (variable, point, node) values (mode 2 has none) and the flux points of a
  // chunk of its (node, line) pairs.
  static constexpr size_t SMEM_MAX = 227 * 1024, SMEM_SM = 228 * 1024, SMEM_BLOCK = 1024;
  static size_t tile_bytes(int nodes) { return (size_t)k::V * k::NS * nodes * sizeof(double); }
  static constexpr size_t line_bytes() { return (size_t)k::V * (k::nf - 2) * sizeof(double); }
  struct Shape {
    int cells = 0, rows = 0, chunk = 0, blocks = 0;  // chunk 0: does not fit
  };
  static size_t interior_smem(const Shape& s, int nodes) { return (tile_bytes(nodes) + line_bytes() * s.chunk) * s.cells; }
  // the largest chunk, in equal parts of all lines, that leaves room for
  // INTERIOR_BLOCKS blocks per SM, or for as many as fit with the smallest
  static Shape interior_shape(int cells, int T) {
    Shape best;
    const int lines = T * k::NJ;
    for (int parts = 1; parts <= lines; ++parts) {
      Shape s;
      s.cells = cells;
      s.chunk = (lines + parts - 1) / parts;
      const size_t b = interior_smem(s, T);
      if (b > SMEM_MAX) continue;
      s.blocks = std::min<int>(INTERIOR_BLOCKS, (int)(SMEM_SM / (b + SMEM_BLOCK)));
      s.rows = std::max(1, std::min(INTERIOR_THREADS / cells, s.chunk * k::V));
      if (s.blocks > best.blocks) best = s;
      if (best.blocks == INTERIOR_BLOCKS) break;
    }
    return best;
  }

  int configure(spd_ctx* C) override {
    max_cpb = 64;
    while (max_cpb > 1 && interior_shape(max_cpb, C->T).chunk == 0) max_cpb /= 2;
    if (interior_shape(max_cpb, C->T).chunk == 0)
      return fail(C, SPD_ERR_ARG, "the step's tile exceeds the shared memory");
    // the widest block that keeps the most threads resident, 16 cells (128
    // bytes of a row) at most
    int best = -1;
    cpb = 1;
    for (int cells = std::min(16, max_cpb); cells >= std::min(4, max_cpb); cells /= 2) {
      const Shape s = interior_shape(cells, C->T);
      if (s.blocks * s.rows * cells > best) {
        best = s.blocks * s.rows * cells;
        cpb = cells;
      }
    }
    CK(cudaFuncSetAttribute(k_interior<D, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX));
    CK(cudaFuncSetAttribute(k_interior_ext<D, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX));
    return 0;
  }

  // cells per block of the interior kernel: the context's own number, or,
  // while none was set and the step is not recorded for a batched launch
  // (which needs one block shape for all instances), fewer where the grid
  // would not give every SM two blocks
  int interior_cells(const spd_ctx* C) const {
    int cells = cpb;
    if (auto_cpb && !C->brec)
      while (cells > 4 && (C->geo.Nc + cells - 1) / cells < 2 * SMS) cells /= 2;
    return cells;
  }
  // the Riemann problems of one Picard iteration; EQ: the form with the well-balanced mode's equilibrium edge
  // values and the isothermal system
  template <bool EQ, int SV>
  void riemann_all(spd_ctx* C, int Teff) {
    const Geo& g = C->geo;
    RiemannDirs r{};
    unsigned nb = 0;
    for (int d = 0; d < D; ++d) {
      r.trace[d] = C->trace[d];
      r.bcfix[d] = C->bcfix[d];
      r.Fi[d] = C->Fi[d];
      r.meq[d] = C->Meq_fp[d];
      r.blocks[d] = blocks_for((long long)Teff * k::NJ * n_iface(g, d), 128);
      nb += r.blocks[d];
    }
    launch<RiemannAll<D, P, EQ, SV>>(C, "k_riemann_sd", k_riemann_all<D, P, EQ, SV>, nb, 128, 0, g, Teff,
                                     C->cfg.riemann_solver_sd, r);
  }

  // the Riemann problems of one Picard iteration with every branch taped
  // (BM 1) or replayed (BM 2), one instantiation per direction as in the
  // plain form.  The runtime-direction instantiation is not used: on
  // sm_103a its LLF branch returned NaN for every flux in 2D (HLLC, 1D and
  // the same device function called from a plain kernel were exact).
  template <int BM>
  void riemann_taped(spd_ctx* C, int d, unsigned nb, int Teff, int solver, unsigned* tp) {
    const Geo& g = C->geo;
    constexpr int D1 = (D > 1 ? 1 : 0), D2 = (D > 2 ? 2 : 0);
    if (d == 0)
      k_riemann_sd<D, P, BM, 0><<<nb, 128, 0, C->stream>>>(g, d, Teff, solver, C->trace[d], C->bcfix[d], C->Fi[d],
                                                          tp, nullptr);
    else if (d == 1)
      k_riemann_sd<D, P, BM, D1><<<nb, 128, 0, C->stream>>>(g, d, Teff, solver, C->trace[d], C->bcfix[d], C->Fi[d],
                                                           tp, nullptr);
    else
      k_riemann_sd<D, P, BM, D2><<<nb, 128, 0, C->stream>>>(g, d, Teff, solver, C->trace[d], C->bcfix[d], C->Fi[d],
                                                           tp, nullptr);
  }

  int predictor(spd_ctx* C, int final_mode) {
    const Geo& g = C->geo;
    if (C->recording)
      CK(cudaMemcpyAsync(C->hist_usp, C->U_sp, sizeof(double) * k::V * k::NS * g.Nc, cudaMemcpyDeviceToDevice,
                         C->stream));
    {
      ProfScope ps_(C, "k_traces_sp");
      launch<TracesSp<D, P>>(C, "k_traces_sp", k_traces_sp<D, P>, blocks_for(g.Nc * (D * k::NJ * k::V), 128), 128, 0, C->ops, g, C->U_sp,
                             C->trace[0], C->trace[1], C->trace[2]);
    }
    CKL();
    const int m = C->T - 1;
    for (int it = 0; it <= m; ++it) {
      const int Teff = (it == 0) ? 1 : C->T;
      const int solver = C->cfg.riemann_solver_sd;
      if (C->tape_mode == 0) {
        ProfScope ps_(C, "k_riemann_sd");
        if (C->Meq_fp[0] || C->cfg.isothermal) riemann_all<true, -1>(C, Teff);
        else if (C->brec && !C->brec->one_sd) riemann_all<false, -1>(C, Teff);
        else if (solver == RS_LLF) riemann_all<false, RS_LLF>(C, Teff);
        else riemann_all<false, RS_HLLC>(C, Teff);
        CKL();
      }
      for (int d = 0; d < D && C->tape_mode != 0; ++d) {
        const unsigned nb = blocks_for((long long)Teff * k::NJ * n_iface(g, d), 128);
        unsigned* tp = C->tape_rs[d] + ((size_t)C->tape_step * C->T + it) * C->T * k::NJ * n_iface(g, d);
        ProfScope ps_(C, "k_riemann_sd");
        if (C->tape_mode == 1) riemann_taped<1>(C, d, nb, Teff, solver, tp);
        else riemann_taped<2>(C, d, nb, Teff, solver, tp);
        CKL();
      }
      const int mode = (it < m) ? 0 : final_mode;
      const double* Uin = (it == 0) ? C->U_sp : C->U_ader;
      const int Tu = (it == 0) ? 1 : C->T;
      const bool visc = C->cfg.viscosity != 0;
      if (visc) {
        // viscous fluxes of this iteration (src/sdader_simulator.py:239-268)
        {
          ProfScope ps_(C, "k_visc_grad");
          launch<ViscGrad<D, P>>(C, "k_visc_grad", k_visc_grad<D, P>,
                                 blocks_for(g.Nc * (D * k::NJ) * Teff, VISC_THREADS), VISC_THREADS, 0, C->ops,
                                 g, Teff, Uin, Tu, C->trace[0], C->trace[1], C->trace[2], C->bcfix[0], C->bcfix[1],
                                 C->bcfix[2], C->Wfp[0], C->Wfp[1], C->Wfp[2], C->dWsp, (const double*)C->Meq_fp[0],
                                 (const double*)C->Meq_fp[1], (const double*)C->Meq_fp[2]);
        }
        CKL();
        {
          ProfScope ps_(C, "k_visc_flux");
          launch<ViscFlux<D, P>>(C, "k_visc_flux", k_visc_flux<D, P>,
                                 blocks_for(g.Nc * (D * k::NJ) * Teff, VISC_THREADS), VISC_THREADS, 0, C->ops,
                                 g, Teff, C->dWsp, C->Wfp[0], C->Wfp[1], C->Wfp[2], C->bcfix[0], C->bcfix[1],
                                 C->bcfix[2], C->cfg.nu, C->cfg.beta, C->Gv[0], C->Gv[1], C->Gv[2]);
        }
        CKL();
      }
      const int cells = interior_cells(C);
      const Shape shape = interior_shape(cells, C->T);
      const dim3 block(cells, shape.rows);
      const size_t sm = interior_smem(shape, mode == 2 ? 0 : (mode == 0 ? C->T : Teff));
      if (visc || C->gphi_sp || C->Ueq_sp || C->cfg.isothermal) {
        ProfScope ps_(C, "k_interior");
        launch<InteriorExt<D, P>>(C, "k_interior", k_interior_ext<D, P>, blocks_for(g.Nc, cells), block, sm, C->ops,
                                  g, mode, Teff, shape.chunk, Uin, Tu, C->dt, C->U_sp, C->U_ader, C->Fi[0], C->Fi[1], C->Fi[2],
                                  C->trace[0], C->trace[1], C->trace[2], C->Ffp[0], C->Ffp[1], C->Ffp[2],
                                  visc ? C->Gv[0] : nullptr, C->Gv[1], C->Gv[2], (const double*)C->gphi_sp,
                                  (const double*)C->Meq_fp[0], (const double*)C->Meq_fp[1],
                                  (const double*)C->Meq_fp[2], (const double*)C->Feq_fp[0],
                                  (const double*)C->Feq_fp[1], (const double*)C->Feq_fp[2]);
      } else {
        ProfScope ps_(C, "k_interior");
        launch<Interior<D, P>>(C, "k_interior", k_interior<D, P>, blocks_for(g.Nc, cells), block, sm, C->ops, g, mode,
                               Teff, shape.chunk, Uin, Tu, C->dt, C->U_sp, C->U_ader, C->Fi[0], C->Fi[1], C->Fi[2], C->trace[0],
                               C->trace[1], C->trace[2], C->Ffp[0], C->Ffp[1], C->Ffp[2]);
      }
      CKL();
      if (C->recording && mode == 0) {
        const size_t n = (size_t)k::V * C->T * k::NS * g.Nc;
        CK(cudaMemcpyAsync(C->hist_ader + (size_t)it * n, C->U_ader, n * sizeof(double), cudaMemcpyDeviceToDevice,
                           C->stream));
      }
    }
    return 0;
  }

  int sp_to_cv(spd_ctx* C) override {
    const Geo& g = C->geo;
    {
      ProfScope ps_(C, "k_sp_to_cv");
      launch<SpToCv<D, P>>(C, "k_sp_to_cv", k_sp_to_cv<D, P>,
                           blocks_for(g.Nc * (k::V * Full<D, P>::tiles), 128), 128, 0, g,
                           (const Coef*)C->Kt_sp_to_cv, C->K_soft, C->U_sp, C->U_cv);
    }
    CKL();
    return 0;
  }

  int wcv(spd_ctx* C) override {
    const Geo& g = C->geo;
    {
      ProfScope ps_(C, "k_prim_only");
      launch<PrimOnly<D>>(C, "k_prim_only", k_prim_only<D>, blocks_for(g.Nq, BS), BS, 0, g, C->U_cv, C->W_cv);
    }
    CKL();
    return 0;
  }

  int cmax(spd_ctx* C) override {
    const Geo& g = C->geo;
    {
      ProfScope ps_(C, "k_cmax_only");
      launch<CmaxOnly<D, P>>(C, "k_cmax_only", k_cmax_only<D, P>, blocks_for(g.Nq, BS), BS, 0, g, C->W_cv,
                             C->counts + 2, C->flags + 1);
    }
    CKL();
    {
      ProfScope ps_(C, "k_dt_final");
      launch<DtFinal>(C, "k_dt_final", k_dt_final, 1, 1, 0, C->h_dt, C->cfg.cfl_coeff, C->counts + 2, C->flags + 1,
                      C->dt, C->dt_visc);
    }
    CKL();
    return 0;
  }

  // affected faces of all directions per substep in a record slot or tape
  static size_t hist_aff_stride(const spd_ctx* C) {
    size_t per = 0;
    for (int d = 0; d < D; ++d) per += (size_t)n_faces(C->geo, d);
    return per;
  }
  static double* tape_aff(spd_ctx* C, int i) {
    return C->tape_aff + ((size_t)C->tape_step * C->T + i) * hist_aff_stride(C);
  }

  // units of a key's upper word that lie within the relative tolerance (Nad)
  static int nad_slack(const spd_config& cf) {
    if (cf.NAD_delta || !(cf.tolerance * 0x1p20 > 2.0)) return -1;
    return (int)std::ceil(std::min(cf.tolerance * 0x1p20, 1024.0)) - 2;
  }

  int fv_update(spd_ctx* C) {
    const Geo& g = C->geo;
    const spd_config& cf = C->cfg;
    // switch_to_finite_volume (src/sdader_simulator.py:288-298)
    if (int r = sp_to_cv(C)) return r;
    {
      ProfScope ps_(C, "k_integrate_faces");
      const FaceArrays fa{{C->Ffp[0], C->Ffp[1], C->Ffp[2]}, {C->F_HO[0], C->F_HO[1], C->F_HO[2]}};
      launch<IntegrateFaces<D, P>>(C, "k_integrate_faces", k_integrate_faces<D, P>,
                                   blocks_for(D * g.Nc * g.T * k::nf, 128), 128, 0, C->ops, g, fa);
    }
    CKL();
    long long nface[3] = {1, 1, 1};
    for (int d = 0; d < D; ++d) nface[d] = n_faces(g, d);
    const BcBufs bc{{C->bcbuf[0], C->bcbuf[1], C->bcbuf[2]}};
    const Counters counters{C->flags, C->counts};
    const unsigned nb_q = blocks_for(g.Nq, BS), nb_ghost = blocks_for(n_ghosts<D>(g), BS);
    for (int i = 0; i < C->T; ++i) {
      const double w_i = C->ops.w_tp[i];
      if (C->recording)
        CK(cudaMemcpyAsync(C->hist_ucv + (size_t)i * k::V * g.Nq, C->U_cv, sizeof(double) * k::V * g.Nq,
                           cudaMemcpyDeviceToDevice, C->stream));
      const double* FH[3] = {nullptr, nullptr, nullptr};
      for (int d = 0; d < D; ++d) FH[d] = C->F_HO[d] + (long long)i * k::V * nface[d];
      {
        ProfScope ps_(C, "k_fv_candidate");
        launch<FvCandidate<D>>(C, "k_fv_candidate", k_fv_candidate<D>, blocks_for(g.Nq, BS), BS, 0, g, C->fvg, C->dt,
                               w_i, FH[0], FH[1], FH[2], C->U_cv, C->U_new, C->ext_old, C->ext_new,
                               cf.FB ? (i == 0 ? 1 : 2) : 0, counters, i == C->T - 1 ? C->W_cv : nullptr,
                               (const double*)C->gphi_fv, (const double*)C->Ueq_cv,
                               (const double*)C->Weq_cv);
      }
      CKL();
      if (cf.FB && C->tape_mode == 2) {
        // the affected faces of the taped step instead of trouble detection
        size_t off = 0;
        for (int d = 0; d < D; ++d) {
          CK(cudaMemcpyAsync(C->aff[d], tape_aff(C, i) + off, sizeof(double) * nface[d], cudaMemcpyDeviceToDevice,
                             C->stream));
          off += (size_t)nface[d];
        }
        // no detection, only the ghosts
        launch<Nad<D>>(C, "k_nad", k_nad<D>, nb_ghost, BS, 0, g, 0u, bc, cf.tolerance, -1, cf.NAD_delta, 1, C->ext_old,
                       C->ext_new, C->mask, C->flags, (long long*)nullptr, C->counts + 3);
        CKL();
      } else if (cf.FB) {
        // detect_troubles (src/trouble_detection.py:5-87)
        const int sed = (P > 1 && cf.SED) ? 1 : 0;
        {
          ProfScope ps_(C, "k_nad");
          long long* sed_list = sed ? C->list_sed : nullptr;
          launch<Nad<D>>(C, "k_nad", k_nad<D>, nb_q + nb_ghost, BS, 0, g, nb_q, bc, cf.tolerance, nad_slack(cf),
                         cf.NAD_delta, P > 0 ? 1 : 0, C->ext_old, C->ext_new, C->mask, C->flags, sed_list,
                         C->counts + 3);
        }
        CKL();
        if (sed) {
          ProfScope ps_(C, "k_sed");
          const unsigned nb = (unsigned)std::min<long long>(PERSIST_BLOCKS, blocks_for(2 * g.Nq, BS));
          launch<Sed<D>>(C, "k_sed", k_sed<D>, nb, BS, 0, g, C->fvg, C->list_sed, C->counts + 3, C->ext_new,
                         C->mask);
          CKL();
        }
        {
          ProfScope ps_(C, "k_troubles");
          launch<Troubles<D>>(C, "k_troubles", k_troubles<D>, nb_q + nb_ghost, BS, 0, g, nb_q, cf.PAD,
                              cf.min_rho, cf.max_rho, cf.min_P, C->mask, (const int*)C->flags, sed, (const double*)C->ext_old,
                              C->ext_new, bc, C->theta_src, C->troubles, (const double*)C->Weq_cv);
        }
        CKL();
        double* th = C->theta_src;
        if (cf.blending) {
          {
            ProfScope ps_(C, "k_blend_neighbours");
            launch<BlendNeighbours<D>>(C, "k_blend_neighbours", k_blend_neighbours<D>, blocks_for(g.Nqe, BS), BS, 0, g,
                                       C->theta_src, C->theta_a);
          }
          CKL();
          {
            ProfScope ps_(C, "k_blend_last");
            launch<BlendLast<D>>(C, "k_blend_last", k_blend_last<D>, blocks_for(g.Nqe, BS), BS, 0, g, C->theta_a,
                                 C->theta_b);
          }
          CKL();
          th = C->theta_b;
        }
        C->theta_final = th;
      }
      if (cf.FB) {
        // affected faces, marks and the fallback fluxes (src/sdader_simulator.py:343-346)
        {
          ProfScope ps_(C, "k_affected_all");
          const double* th = C->tape_mode == 2 ? nullptr : C->theta_final;
          const AffectedOut out{{C->aff[0], C->aff[1], C->aff[2]},
                                {C->list_face[0], C->list_face[1], C->list_face[2]},
                                C->list_cell,
                                C->list_q,
                                C->counts};
          launch<AffectedAll<D>>(C, "k_affected_all", k_affected_all<D>, blocks_for(g.Nqe, BS), BS, 0, g, cf.godunov,
                                 th, out);
        }
        CKL();
        if (C->tape_mode == 1) {
          size_t off = 0;
          for (int d = 0; d < D; ++d) {
            CK(cudaMemcpyAsync(tape_aff(C, i) + off, C->aff[d], sizeof(double) * nface[d], cudaMemcpyDeviceToDevice,
                               C->stream));
            off += (size_t)nface[d];
          }
        }
        k_muscl_cells_grid(C, w_i, i);
        CKL();
        if (C->recording) {
          const size_t nq = (size_t)k::V * g.Nqe;
          double* dst = C->hist_mpred + (size_t)i * (1 + D) * nq;
          CK(cudaMemcpyAsync(dst, C->Mpred, sizeof(double) * nq, cudaMemcpyDeviceToDevice, C->stream));
          CK(cudaMemcpyAsync(dst + nq, C->S, sizeof(double) * D * nq, cudaMemcpyDeviceToDevice, C->stream));
        }
        long long nface_all = 0;
        for (int d = 0; d < D; ++d) nface_all += nface[d];
        if (C->tape_mode == 0) {
          ProfScope ps_(C, "k_muscl_faces");
          const unsigned nb = (unsigned)std::min<long long>(PERSIST_BLOCKS, blocks_for(nface_all, 128));
          if (C->brec && !C->brec->one_fv) muscl_faces<-1>(C, nb);
          else if (cf.riemann_solver_fv == RS_LLF) muscl_faces<RS_LLF>(C, nb);
          else muscl_faces<RS_HLLC>(C, nb);
          CKL();
        }
        for (int d = 0; d < D && C->tape_mode != 0; ++d) {
          ProfScope ps_(C, "k_muscl_faces");
          const unsigned nb = (unsigned)std::min<long long>(PERSIST_BLOCKS, blocks_for(nface[d], BS));
          const unsigned long long* fcount = C->counts + 4 + d;
          unsigned* tp = C->tape_fb[d] + ((size_t)C->tape_step * C->T + i) * nface[d];
          if (C->tape_mode == 1)
            k_muscl_faces<D, 1><<<nb, BS, 0, C->stream>>>(g, d, cf.riemann_solver_fv, C->list_face[d], fcount,
                                                         C->Mpred, C->S, C->F_FB[d], tp, nullptr, nullptr);
          else
            k_muscl_faces<D, 2><<<nb, BS, 0, C->stream>>>(g, d, cf.riemann_solver_fv, C->list_face[d], fcount,
                                                         C->Mpred, C->S, C->F_FB[d], tp, nullptr, nullptr);
          CKL();
        }
        k_fv_correct_grid(C, w_i, FH, i == C->T - 1 ? C->W_cv : nullptr);
        CKL();
        C->fb_ran = true;
        if (C->recording) {
          size_t off = 0;
          const size_t per = hist_aff_stride(C);
          for (int d = 0; d < D; ++d) {
            CK(cudaMemcpyAsync(C->hist_aff + (size_t)i * per + off, C->aff[d], sizeof(double) * nface[d],
                               cudaMemcpyDeviceToDevice, C->stream));
            off += (size_t)nface[d];
          }
        }
      }
      std::swap(C->U_cv, C->U_new);
    }
    // switch_to_high_order (src/sdader_simulator.py:300-307)
    {
      ProfScope ps_(C, "k_cv_to_sp");
      launch<CvToSp<D, P>>(C, "k_cv_to_sp", k_cv_to_sp<D, P>,
                           blocks_for(g.Nc * (k::V * Full<D, P>::tiles), 128), 128, 0, g,
                           (const Coef*)C->Kt_cv_to_sp, C->K_soft, C->U_cv, C->U_sp);
    }
    CKL();
    return 0;
  }

  template <int SV>
  void muscl_faces(spd_ctx* C, unsigned nb) {
    const FaceLists fl{{C->list_face[0], C->list_face[1], C->list_face[2]},
                       C->counts + 4,
                       {C->F_FB[0], C->F_FB[1], C->F_FB[2]},
                       {C->Meq_faces[0], C->Meq_faces[1], C->Meq_faces[2]},
                       {C->Feq_faces[0], C->Feq_faces[1], C->Feq_faces[2]}};
    launch<MusclFacesAll<D, SV>>(C, "k_muscl_faces", k_muscl_faces_all<D, SV>, nb, 128, 0, C->geo,
                                 C->cfg.riemann_solver_fv, fl, C->Mpred, C->S);
  }

  void k_muscl_cells_grid(spd_ctx* C, double w_i, int i) {
    const Geo& g = C->geo;
    const long long nb = std::min<long long>(2 * PERSIST_BLOCKS, blocks_for(g.Nqe, LIST_CELLS));
    const dim3 block(LIST_CELLS, k::V);
    ProfScope ps_(C, "k_muscl_cells");
    if (C->tape_mode == 0) {
      unsigned char* no_tape = nullptr;
      launch<MusclCells<D>>(C, "k_muscl_cells", k_muscl_cells<D>, (unsigned)nb, block, 0, g, C->fvg,
                            C->cfg.slope_limiter, C->dt, w_i, C->list_cell, C->counts, C->ext_old, C->Mpred, C->S,
                            no_tape, (const double*)C->Meq_fv, (const double*)C->gphi_fv);
      return;
    }
    unsigned char* lt = C->tape_lim + ((size_t)C->tape_step * C->T + i) * D * k::V * g.Nqe;
    if (C->tape_mode == 1)
      k_muscl_cells<D, 1><<<(unsigned)nb, block, 0, C->stream>>>(g, C->fvg, C->cfg.slope_limiter, C->dt, w_i,
                                                               C->list_cell, C->counts, C->ext_old, C->Mpred, C->S, lt,
                                                               nullptr, nullptr);
    else
      k_muscl_cells<D, 2><<<(unsigned)nb, block, 0, C->stream>>>(g, C->fvg, C->cfg.slope_limiter, C->dt, w_i,
                                                               C->list_cell, C->counts, C->ext_old, C->Mpred, C->S, lt,
                                                               nullptr, nullptr);
  }

  void k_fv_correct_grid(spd_ctx* C, double w_i, const double* const* FH, double* W_cv) {
    const Geo& g = C->geo;
    const long long nb = std::min<long long>(2 * PERSIST_BLOCKS, blocks_for(g.Nq, LIST_CELLS));
    const dim3 block(LIST_CELLS, k::V);
    {
      ProfScope ps_(C, "k_fv_correct");
      launch<FvCorrect<D>>(C, "k_fv_correct", k_fv_correct<D>, (unsigned)nb, block, 0, g, C->fvg, C->dt, w_i,
                           C->cfg.godunov, C->list_q, C->counts + 1, FH[0], FH[1], FH[2], C->F_FB[0], C->F_FB[1],
                           C->F_FB[2], C->aff[0], C->aff[1], C->aff[2], C->U_cv, C->U_new, C->ext_new, W_cv,
                           (const double*)C->gphi_fv, (const double*)C->Ueq_cv, (const double*)C->Weq_cv);
    }
  }

  // adjoint of the recorded step (spd_adjoint_exec.cuh, compiled in its own
  // translation units)
  int vjp(spd_ctx* C) override { return adjoint_vjp<D, P>(C); }

  // well-balanced mode: U_sp -/+ U_eq_sp around the step
  int wb_shift(spd_ctx* C, double sign) {
    const Geo& g = C->geo;
    const long long n = (long long)k::V * k::NS * g.Nc;
    {
      ProfScope ps_(C, "k_wb_shift");
      launch<WbShift>(C, "k_wb_shift", k_wb_shift, blocks_for(n, BS), BS, 0, n, sign, C->U_sp,
                      (const double*)C->Ueq_sp);
    }
    CKL();
    return 0;
  }

  int eq_prims(spd_ctx* C) override {
    const Geo& g = C->geo;
    {
      ProfScope ps_(C, "k_prim_only");
      launch<PrimOnly<D>>(C, "k_prim_only", k_prim_only<D>, blocks_for(g.Nq, BS), BS, 0, g, C->Ueq_cv, C->Weq_cv);
    }
    CKL();
    return 0;
  }

  int update(spd_ctx* C) override {
    const int final_mode = (C->cfg.update == SPD_UPDATE_SD) ? 1 : 2;
    if (C->Ueq_sp) {
      // src/sdader_simulator.py:363-365, 372-376: the step advances the
      // perturbation; afterwards U_sp += U_eq_sp, U_cv += U_eq_cv (with the
      // SD update U_cv is the previous step's) and W_cv = prim(U_cv)
      if (int r = wb_shift(C, -1.0)) return r;
      if (int r = predictor(C, final_mode)) return r;
      if (C->cfg.update == SPD_UPDATE_FV)
        if (int r = fv_update(C)) return r;
      if (int r = wb_shift(C, 1.0)) return r;
      const Geo& g = C->geo;
      {
        ProfScope ps_(C, "k_wb_end");
        launch<WbEnd<D>>(C, "k_wb_end", k_wb_end<D>, blocks_for(g.Nq, BS), BS, 0, g, C->U_cv,
                         (const double*)C->Ueq_cv, C->W_cv);
      }
      CKL();
      return 0;
    }
    if (int r = predictor(C, final_mode)) return r;
    if (C->cfg.update == SPD_UPDATE_FV) {
      if (int r = fv_update(C)) return r;
      // W_cv = prim(U_cv) (src/sdader_simulator.py:376): written by the last
      // substep's candidate and corrected updates
      if (C->cfg.FB) return 0;
    }
    // W_cv = prim(U_cv) (src/sdader_simulator.py:376)
    return wcv(C);
  }
};

template <int D, int P>
StepperBase* make_stepper_of() {
  return new Stepper<D, P>();
}

}  // namespace spd_host
