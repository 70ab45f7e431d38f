// One Newton iteration's assembly as one call: the pair kernels, the beam, the contact tangent and the residual
// on the caller's stream and three side streams, joined before it returns to the caller's.
//
// Each part goes through its own entry point; what this call saves is host time.  Nine entry points, each with its
// arguments and streams marshalled, and some ten stream waits took the caller's interpreter longer than the
// kernels of an ordinary strand take the GPU.
// Measured eagerly at the 37-wire strand in double: 125 -> 75 us (the segments' records of pair.cu included).
#include "context.cuh"

xk_status xk_pair_step_seg(const xk_mesh* m, xk_pairs* p, const xk_contact_pattern* pat, const double* u,
                           const double* u_ref, const xk_contact_params* cp, int stages, int precision, int out_mode,
                           const double* seg64, void* rec, xk_stream s);
xk_status xk_contact_gather_force_norm(const xk_contact_pattern* pat, const void* rec, int precision,
                                       const double* base, double scale, const double* f_ext, const uint8_t* fixed,
                                       double* out, double* norm2, xk_stream s);

namespace {

constexpr int STAGES = XK_STAGE_NARROW | XK_STAGE_NORMAL | XK_STAGE_FRICTION | XK_STAGE_TANGENT;

// The events of the forks and joins, per thread and context.  A wait takes what its event holds when it is issued,
// so they serve one call after the other; threads have their own.
enum { EV_START, EV_NODES, EV_BEAM, EV_OTHERS, EV_MEMBERS, EV_SUMS, EV_TANGENT, EV_N };
struct Events {
  cudaEvent_t e[EV_N] = {};
  void drop() {
    for (cudaEvent_t x : e)
      if (x) cudaEventDestroy(x);
  }
};
xk_status events_here(Events** out) {
  thread_local PerContext<Events> sets;
  XK_TRY(sets.here(out));
  for (cudaEvent_t& x : (*out)->e)
    if (!x) {
      RelaxedCapture relaxed;
      XK_CUDA(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
    }
  return XK_OK;
}

xk_status mark(cudaEvent_t e, cudaStream_t on) {
  XK_CUDA(cudaEventRecord(e, on));
  return XK_OK;
}
xk_status wait(cudaStream_t s, cudaEvent_t e) {
  XK_CUDA(cudaStreamWaitEvent(s, e, 0));
  return XK_OK;
}

}  // namespace

extern "C" xk_status xk_assemble(const xk_assembly* a, const double* u, const double* u_ref, const double* f_ext,
                                 const uint8_t* fixed, xk_stream s) {
  if (!a || !a->mesh || !a->section || !a->plan || !a->pat || !a->cp || !u)
    return xk_set_error(XK_ERR_ARG, "xk_assemble: null argument");
  if (a->precision != XK_FP64 && a->precision != XK_MIXED)
    return xk_set_error(XK_ERR_ARG, "xk_assemble: precision");
  const bool mixed = a->precision == XK_MIXED;
  if (mixed ? !a->pairs32 || !a->node32 : !a->pairs || !a->elem_ref)
    return xk_set_error(XK_ERR_ARG, "xk_assemble: null argument");
  Events* ev;
  XK_TRY(events_here(&ev));
  cudaStream_t st = (cudaStream_t)s, so = (cudaStream_t)a->side[0], sb = (cudaStream_t)a->side[1],
               sg = (cudaStream_t)a->side[2];
  const xk_contact_pattern* pat = a->pat;
  const int n_o = mixed ? a->pairs32->n - a->pairs32->n_members : pat->n_others;
  void* const K_beam = a->tangent ? a->K_beam : nullptr;
  // the beam and the other pairs' narrowphase each on a stream of their own
  if (mixed) {
    XK_TRY(xk_nodes_prepare(a->mesh, u, u_ref, a->node32, s));
    XK_TRY(mark(ev->e[EV_NODES], st));
    if (n_o > 0) {
      XK_TRY(wait(so, ev->e[EV_NODES]));
      XK_TRY(xk_pair_step32(a->pairs32, a->node32, a->cp, (float*)a->rec, XK_PAIRS_OTHERS, so));
    }
    XK_TRY(wait(sb, ev->e[EV_NODES]));
    XK_TRY(xk_beam_assemble32(a->mesh, a->section, a->elem32, a->plan, a->node32, a->f_int, (float*)K_beam, sb));
    XK_TRY(xk_pair_step32(a->pairs32, a->node32, a->cp, (float*)a->rec, XK_PAIRS_MEMBERS, s));
  } else {
    XK_TRY(mark(ev->e[EV_START], st));
    XK_TRY(wait(sb, ev->e[EV_START]));
    XK_TRY(xk_beam_assemble(a->mesh, a->section, a->elem_ref, a->plan, u, a->precision, a->f_int, K_beam, sb));
    if (a->seg64 && a->pairs->n > 0) XK_TRY(xk_segments64(a->mesh, u, u_ref, a->seg64, s));
    if (n_o > 0) {
      XK_TRY(mark(ev->e[EV_NODES], st));
      XK_TRY(wait(so, ev->e[EV_NODES]));
      XK_TRY(xk_pair_step_seg(a->mesh, a->pairs, pat, u, u_ref, a->cp, XK_STAGE_NARROW | XK_STAGE_NO_MEMBERS,
                              a->precision, XK_OUT_COMBINED, a->seg64, a->rec, so));
    }
    XK_TRY(xk_pair_step_seg(a->mesh, a->pairs, pat, u, u_ref, a->cp, STAGES | XK_STAGE_NO_OTHERS, a->precision,
                            XK_OUT_COMBINED, a->seg64, a->rec, s));
  }
  // the contact tangent from the members' records; its element-side schedule leaves the sums for the residual
  const bool gather = a->tangent && pat->nnzb > 0, elem_force = gather && a->gather_variant == XK_GATHER_SIDES;
  if (gather) {
    XK_TRY(mark(ev->e[EV_MEMBERS], st));
    XK_TRY(wait(sg, ev->e[EV_MEMBERS]));
    if (elem_force) {
      XK_TRY(xk_contact_gather_tangent(pat, a->rec, a->precision, XK_OUT_COMBINED, XK_WHICH_COMBINED,
                                       XK_GATHER_SIDES_SUMS, a->K_c, sg));
      XK_TRY(mark(ev->e[EV_SUMS], sg));
      XK_TRY(xk_contact_gather_tangent(pat, a->rec, a->precision, XK_OUT_COMBINED, XK_WHICH_COMBINED,
                                       XK_GATHER_SIDES_BLOCKS, a->K_c, sg));
    } else {
      XK_TRY(xk_contact_gather_tangent(pat, a->rec, a->precision, XK_OUT_COMBINED, XK_WHICH_COMBINED,
                                       a->gather_variant, a->K_c, sg));
    }
  }
  XK_TRY(mark(ev->e[EV_BEAM], sb));
  XK_TRY(wait(st, ev->e[EV_BEAM]));
  if (elem_force) {
    XK_TRY(wait(st, ev->e[EV_SUMS]));
    XK_TRY(xk_contact_gather_force_elem(pat, a->precision, a->f_int, -1.0, f_ext, fixed, a->R, a->norm2, s));
  } else {
    XK_TRY(xk_contact_gather_force_norm(pat, a->rec, a->precision, a->f_int, -1.0, f_ext, fixed, a->R, a->norm2, s));
  }
  if (n_o > 0) {
    XK_TRY(mark(ev->e[EV_OTHERS], so));
    XK_TRY(wait(st, ev->e[EV_OTHERS]));
  }
  if (gather) {
    XK_TRY(mark(ev->e[EV_TANGENT], sg));
    XK_TRY(wait(st, ev->e[EV_TANGENT]));
  }
  return XK_OK;
}
