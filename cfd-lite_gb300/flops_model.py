"""FP64 thread-instructions per launch of the kernels that do FP64 arithmetic.

GB300 issues about two FP64 thread-instructions per SM per clock (the
cfdl_probe_fp64 DFMA probe measures 0.63 T instructions/s, 1.25 TFLOP/s), so
the assembly kernels of the outer iteration are bound by the FP64 pipe before
they are bound by HBM.  The figures are the FP64 instructions the kernels
execute (DADD, DMUL, DFMA and the rest of the double-precision class, each one
pipe slot), as ncu counted them (sm__sass_thread_inst_executed_op_fp64_pred_on),
per cell unless said otherwise.

form "flow": FP64 flow without the energy equation, the default benchmark
(profiles/fp64_instructions_forms.md, 48^3 and 128^3 hex cavities):

  k_coef_uvw_face  36 per interior face
  k_calc_mip       23 per interior face (9 without the Rhie-Chow term)
  k_coef_uvw_init  99.8, and 164 per wall face, fitted to both sizes: a warp with a wall cell among
                   its 32 goes through the boundary terms with all its lanes,
                   half of the warps at 128^3
  k_mom_*          BiCGStab with three active right-hand sides, with the
                   reductions of tiles of 1024 cells and more
  k_v_*, k_apc_q   the pressure solve's mesh-level rows: 8 the sweeps, 7 the
                   residual

form "ordered": FP64 with the energy equation, whose kernels keep one order of
sums (the same file).

form "separate": the capture of profiles/fp64_instructions_cavity48.md, of the
single routines' kernels and the forms before those two.  Its k_calc_mip is
the mean over two launches with the Rhie-Chow term (26 per face) and one
without (11).

W = faces per cell; the W-slot rows are scaled from the hex counts by W / 6.
"""


def _separate(ne, nf, nbf, W):
    nfi, w = nf - nbf, W / 6.0
    return {
        "k_coef_uvw_face": 40 * nfi,
        "k_calc_mip": 21 * nfi,
        "k_coef_uvw_cell": 70 * ne + 50 * nbf,
        "k_grad3": 12 * W * ne,
        "k_grad1": 4 * W * ne,
        "k_mom_init": 42.7 * w * ne,
        "k_mom_v": 26.5 * w * ne,
        "k_mom_t": 31.3 * w * ne,
        "k_mom_x": 17.3 * ne,
        "k_mom_s": 8.8 * ne,
        "k_v_jac_f": 9.0 * w * ne,
        "k_v_resid_f": 8.0 * w * ne,
        "k_apc_q": 9.3 * w * ne,
    }


def _flow(ne, nf, nbf, W):
    nfi, w = nf - nbf, W / 6.0
    return {
        "k_coef_uvw_face": 36 * nfi,
        "k_calc_mip": 23 * nfi,
        "k_coef_uvw_init": (30 + 69.8 * w) * ne + 164 * nbf,
        "k_grad3": 12 * W * ne,
        "k_grad1": 4 * W * ne,
        "k_mom_p": 9.0 * ne,
        "k_mom_v": 24.3 * w * ne,
        "k_mom_s": 9.3 * ne,
        "k_mom_t": 27.6 * w * ne,
        "k_mom_x": 18.6 * ne,
        "k_v_jac_f": 8.0 * w * ne,
        "k_v_resid_f": 7.0 * w * ne,
        "k_apc_q": 8.1 * w * ne,
    }


def _ordered(ne, nf, nbf, W):
    t, w = _flow(ne, nf, nbf, W), W / 6.0
    t.update({
        "k_coef_uvw_face": 40 * (nf - nbf),
        "k_calc_mip": 26 * (nf - nbf),
        "k_coef_uvw_init": (30 + 72 * w) * ne + 29 * nbf,
        "k_v_jac_f": (2 * 10.0 + 9.0) / 3 * w * ne,      # of three sweeps, two from t and one from z
        "k_v_resid_f": 13.0 * w * ne,
    })
    return t


_FORMS = {"separate": _separate, "flow": _flow, "ordered": _ordered}


def fp64_inst(name, ne, nf, nbf, W, form="separate"):
    v = _FORMS[form](ne, nf, nbf, W).get(name)
    return int(round(v)) if v is not None else None
