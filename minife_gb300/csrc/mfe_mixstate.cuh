// State of the mixed-precision CG on the device (mfe_mixed.cu, mfe_mixed_loop.cu).
#pragma once

namespace mfe {

struct MixState {
  double rr;            // r.r of the current recursive residual (FP64 accumulated)
  double rr_new;        // r.r after this iteration's update
  double pAp;           // written by the FP32 SpMV's epilogue
  double beta;
  double rr_true;       // ||b - A x||^2 from the gated FP64 residual SpMV
  double rr_at_update;  // rr right after the last reliable update
  double normr0, tol_abs, normr_true;
  double delta2;        // update when rr_new < delta2 * rr_at_update
  double alpha_prev;    // alpha of the last update, whose x32 += alpha p is still pending
  int k;                // inner iterations done
  int max_iter;
  int since;            // iterations since the last reliable update
  int refine_k;         // update at least every refine_k iterations
  int max_refine;       // stop after this many updates (0: no cap)
  int gate;             // 1: a reliable update runs in this iteration
  int cont;             // loop condition
  int run;              // 0: the rest of the loop body's iterations do nothing
  int first;            // next p update is p = r
  int updates;          // reliable updates done
  int status;           // 0 ok, MFE_BREAKDOWN
  int record;
  unsigned err;
  int x_pending;        // 1: x32 += alpha_prev p is due (done by the next p update or
                        // the gated x update, whichever comes first)
  double* history;      // recursive normr per iteration (record)
};

}  // namespace mfe
