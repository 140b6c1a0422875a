"""The packed conversion of a PlannerConfig to the C struct, against one ctypes
assignment a field: the same bytes for what it takes, the same conversions and
refusals for what it leaves to them."""
import ctypes as C

import numpy as np
import pytest

from kgmt_gb300._abi import KgmtConfig, to_c
from kgmt_gb300.config import double_integrator_single, dubins_airplane, quadrotor_large, unicycle


def by_field(cfg):
    k = KgmtConfig()
    for name, _ in KgmtConfig._fields_:
        v = getattr(cfg, name)
        setattr(k, name, (C.c_float * 4)(*[float(x) for x in v]) if name in ("u_min", "u_max") else v)
    return k


BASE = double_integrator_single(3)
FORMS = {
    "di": BASE, "quad": quadrotor_large(2 ** 64 - 1), "dubins": dubins_airplane(0), "unicycle": unicycle(7),
    "ints for floats": BASE.replace(epsilon=1, u_min=(-1, -1, -1, 0)), "numpy floats": BASE.replace(step_size=np.float32(0.07)),
    "numpy bounds": BASE.replace(u_max=np.float32([1, 2, 3, 4])), "list": BASE.replace(u_min=[-1.0, -2.0, -3.0, 0.5]),
    "short bounds": BASE.replace(u_min=(-1.0, -1.0)), "text bounds": BASE.replace(u_min=("-1", "-1", "-1", "0")),
    "wraps": BASE.replace(tree_capacity=-1, model=2 ** 31), "negative seed": BASE.replace(seed=-5), "bool": BASE.replace(di_rule=True),
    "infinite": BASE.replace(v_max=float("inf"), ws_min=float("nan")), "numpy int": BASE.replace(tree_capacity=np.int64(5)), "past float": BASE.replace(v_max=1e300),
}
REFUSED = {"float for int": BASE.replace(max_steps=2.0), "none": BASE.replace(epsilon=None),
           "long bounds": BASE.replace(u_min=(0.0,) * 5), "text": BASE.replace(epsilon="1")}


@pytest.mark.parametrize("form", FORMS)
def test_same_struct(form):
    assert bytes(to_c(FORMS[form])) == bytes(by_field(FORMS[form]))


@pytest.mark.parametrize("form", REFUSED)
def test_same_refusal(form):
    with pytest.raises(Exception) as want:
        by_field(REFUSED[form])
    with pytest.raises(want.type):
        to_c(REFUSED[form])
