"""The FP64 instruction model of the forms that run, against the counts committed
in profiles/fp64_instructions_forms.md: within 2% at both sizes.  CPU only."""
import os
import re
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cfd-lite_gb300"))

from flops_model import fp64_inst  # noqa: E402

# model name -> the kernel whose count it stands for, per section of the file
FLOW = {"k_coef_uvw_face": "k_coef_uvw_face<1>", "k_calc_mip": "k_calc_mip<1>", "k_coef_uvw_init": "k_coef_uvw_init<0>",
        "k_grad3": "k_grad<3>", "k_grad1": "k_grad<1>"}
FLOW48 = dict(FLOW, k_v_jac_f="k_v_jac_mesh<0>", k_v_resid_f="k_v_resid_mesh", k_apc_q="k_apc_q<0>",
              k_mom_p="k_mom_p<double, 3>", k_mom_v="k_mom_v<double, 3, 0, 0>", k_mom_s="k_mom_s<double, 3, 0>",
              k_mom_t="k_mom_t<double, 3, 0, 0>", k_mom_x="k_mom_x<double, 3, 0>")
FLOW128 = dict(FLOW, k_v_jac_f="k_v_jac_pair64<0>", k_v_resid_f="k_v_resid_pair64", k_apc_q="k_apc_q<0>")
ORDERED = {"k_coef_uvw_face": "k_coef_uvw_face<0>", "k_calc_mip": "k_calc_mip<0>", "k_coef_uvw_init": "k_coef_uvw_init<1>"}


def counts():
    out, key = {}, None
    for line in open(os.path.join(ROOT, "profiles", "fp64_instructions_forms.md")):
        if line.startswith("## "):
            key = ("flow" if line.startswith("## FP64 flow") else "ordered", int(re.search(r"(\d+)\^3", line).group(1)))
        m = re.match(r"\| `([^`]+)` \| \d+ \| (\d+) \|", line)
        if m and key:
            out[key + (m.group(1),)] = int(m.group(2))
    return out


@pytest.mark.parametrize("form,n,names", [("flow", 48, FLOW48), ("flow", 128, FLOW128), ("ordered", 48, ORDERED),
                                          ("ordered", 128, ORDERED)])
def test_counts(form, n, names):
    got = counts()
    ne, nbf = n ** 3, 6 * n * n
    nf = 3 * n * n * (n - 1) + nbf
    for model, kernel in names.items():
        c = got[form, n, kernel]
        m = fp64_inst(model, ne, nf, nbf, 6, form)
        assert abs(m - c) <= 0.02 * c, (model, m, c)


def test_sweep_means_of_the_ordered_form():
    got = counts()
    ne = 48 ** 3
    mean = (2 * got["ordered", 48, "k_v_jac<double, 0>"] + got["ordered", 48, "k_v_jac<double, 1>"]) / 3
    assert abs(fp64_inst("k_v_jac_f", ne, 0, 0, 6, "ordered") - mean) <= 0.02 * mean
    assert fp64_inst("k_v_resid_f", ne, 0, 0, 6, "ordered") == got["ordered", 48, "k_v_resid_order"]
