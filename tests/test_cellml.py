"""CellML parser / code generator."""
import glob
import os
import re
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

import helpers as H
from opendihu_b200 import cellml
from oracle import oracle as O

ROOT = H.ROOT
#: the reference checkout, where a run names one ($OPENDIHU_REFERENCE); the tests that read it skip otherwise
REF = os.environ.get("OPENDIHU_REFERENCE", "")
REF_INPUT = os.path.join(REF, "testing/unit_testing/input") if REF else ""


def test_expression_precedence():
    e = cellml.parse_expression("a0 - 1 > 0 && 2 < 3 ? 1 : 0".replace("a0", "STATES[0]"))
    assert e[0] == "tern" and e[1][0] == "bin" and e[1][1] == "&&"
    assert cellml.eval_expr(cellml.parse_expression("2 - 3 - 4"), {}) == -5
    assert cellml.eval_expr(cellml.parse_expression("2 / 4 * 8"), {}) == 4
    assert cellml.eval_expr(cellml.parse_expression("- 2 * 3 + 1"), {}) == -5
    assert cellml.eval_expr(cellml.parse_expression("1 + - 2"), {}) == -1
    env = {"T": 0.25, "S": [], "C": [], "A": [], "R": []}
    e = cellml.parse_expression("VOI>=0.00000&&VOI<0.500000 ? 150.000 : 0.00000")
    assert cellml.eval_expr(e, env) == 150.0


def test_integer_exponent_detection():
    # reference rule (03_generator_vc.cpp:68-117): digits/sign/dot only and atoi != 0
    f = lambda t: cellml._int_exponent(cellml.parse_expression(t))
    assert f("3.00000") == 3
    assert f("- 1.00000") == -1
    assert f("0.500000") is None
    assert f("CONSTANTS[1]") is None


def test_integer_power_helpers_multiplication_order():
    x = 1.1
    assert cellml._int_pow_value(x, 2) == x * x
    assert cellml._int_pow_value(x, 3) == x * (x * x)
    assert cellml._int_pow_value(x, 4) == (x * x) * (x * x)
    assert cellml._int_pow_value(x, -1) == 1.0 / x


def test_parameter_substitution():
    model = cellml.Model(name="t", source="t.c", n_states=1, n_algebraics=2, n_constants=2, states_initial=[0.0],
                         constants=[1.0, 2.0], constant_lines=[],
                         lines=[("A", 0, cellml.parse_expression("CONSTANTS[1]*STATES[0]")),
                                ("A", 1, cellml.parse_expression("ALGEBRAIC[0]+CONSTANTS[0]")),
                                ("R", 0, cellml.parse_expression("ALGEBRAIC[1]"))])
    lines = cellml.substitute_parameters(model, [0], [1])
    assert len(lines) == 2  # the line assigning ALGEBRAIC[0] is dropped
    assert lines[0][2][2] == ("var", "P", 0)  # ALGEBRAIC[0] -> PARAMS[0]
    lines = cellml.substitute_parameters(model, [], [1])
    assert lines[0][2][2] == ("var", "P", 0)  # CONSTANTS[1] -> PARAMS[0]


@pytest.mark.skipif(not os.path.isdir(REF_INPUT), reason="reference checkout not present")
def test_generated_sources_are_current(tmp_path):
    cuda_dir = tmp_path / "cuda"
    c_dir = tmp_path / "c"
    cuda_dir.mkdir()
    c_dir.mkdir()
    cellml.generate_all(REF_INPUT, str(cuda_dir), str(c_dir))
    for d, committed in ((cuda_dir, os.path.join(ROOT, "opendihu_b200/csrc/generated")),
                         (c_dir, os.path.join(ROOT, "oracle/generated"))):
        for f in os.listdir(d):
            assert open(os.path.join(d, f)).read() == open(os.path.join(committed, f)).read(), f


def _ref_lib(name):
    p = os.path.join(ROOT, "oracle", "_ref", f"libref_{name}.so")
    if not os.path.exists(p):
        pytest.skip("oracle/_ref not built (make -C oracle ref needs the reference checkout)")
    L = C.CDLL(p)
    L.computeRates.argtypes = [C.c_double] + [C.POINTER(C.c_double)] * 4
    L.initConsts.argtypes = [C.POINTER(C.c_double)] * 3
    return L


@pytest.mark.parametrize("model,params_alg,params_const,n_const", [
    (H.HH, [], [2, 3, 4], 9), (H.SHORTEN, [32], [65], 105)])
def test_generated_rhs_matches_reference_model_file(model, params_alg, params_const, n_const):
    """generated C right-hand side == the reference's own computeRates (compiled in oracle/_ref)."""
    L = _ref_lib(model)
    ns, na, npar, init = O.model_info(model)
    consts = np.zeros(n_const)
    rates0 = np.zeros(ns)
    states0 = np.zeros(ns)
    L.initConsts(consts.ctypes.data_as(C.POINTER(C.c_double)), rates0.ctypes.data_as(C.POINTER(C.c_double)),
                 states0.ctypes.data_as(C.POINTER(C.c_double)))
    np.testing.assert_array_equal(states0, init)
    rng = np.random.default_rng(0)
    for trial in range(20):
        st = init * (1 + 0.05 * rng.standard_normal(ns))
        st[0] = init[0] + 30 * rng.standard_normal()
        t = 0.3 if trial % 2 else 60.2
        # parameters: constant parameters at random values, algebraic parameters at a fixed value
        p_const = [consts[c] * (1 + 0.1 * rng.standard_normal()) for c in params_const]
        p_alg = [12.5 for _ in params_alg]
        c2 = consts.copy()
        for c, v in zip(params_const, p_const):
            c2[c] = v
        r_ref = np.zeros(ns)
        a_ref = np.zeros(max(na, 1))
        L.computeRates(t, c2.ctypes.data_as(C.POINTER(C.c_double)), r_ref.ctypes.data_as(C.POINTER(C.c_double)),
                       st.ctypes.data_as(C.POINTER(C.c_double)), a_ref.ctypes.data_as(C.POINTER(C.c_double)))
        r, a = O.rates(model, st, np.array(p_alg + p_const), t=t)
        if params_alg:
            # the reference computes the algebraic parameter from VOI; the generated code reads the
            # parameter instead, so compare against the reference evaluated with that value forced in:
            # only the lines not depending on it are expected to agree exactly
            dep = np.abs(r - r_ref) > 1e-12 * (1 + np.abs(r_ref))
            assert dep.sum() <= 2, np.nonzero(dep)
        else:
            np.testing.assert_allclose(r, r_ref, rtol=1e-14, atol=1e-300)


def test_mappings_of_the_example_settings():
    # the "mappings" the fibers_emg example builds for its models (examples/electrophysiology/fibers/fibers_emg/
    # helper.py:112-132) resolve to the parameter variants built into the library
    from opendihu_b200 import cellml as CM
    hh = CM.model_variable_names("hodgkin_huxley_1952")
    m = CM.parse_mappings({("parameter", 0): ("constant", "membrane/i_Stim"),
                           ("connectorSlot", 0): ("state", "membrane/V")}, hh)
    assert m["parametersUsedAsConstant"] == [2] and m["parametersUsedAsAlgebraic"] == []
    assert m["statesForTransfer"] == [0] and m["algebraicsForTransfer"] == []
    sh = CM.model_variable_names("shorten_ocallaghan_davidson_soboleva_2007")
    m = CM.parse_mappings({("parameter", 0): ("algebraic", "wal_environment/I_HH"),
                           ("parameter", 1): ("constant", "razumova/L_x"),
                           ("connectorSlot", 0): ("state", "wal_environment/vS")}, sh)
    assert (m["parametersUsedAsAlgebraic"], m["parametersUsedAsConstant"], m["statesForTransfer"]) == ([32], [65], [0])


def test_mappings_forms():
    # 00_cellml_adapter_base.tpp:160-607: bare names are looked up among algebraics, states, constants; numbers
    # may replace names; slots given by name are numbered on; parameters sort before connector slots; a
    # constant that is a parameter can be a slot (as that parameter)
    from opendihu_b200 import cellml as CM
    names = {"state": ["c/V", "c/m"], "algebraic": ["c/i_Na", "c/i_K"], "constant": ["c/g", "c/E", "c/I"]}
    m = CM.parse_mappings({("connectorSlot", "vm"): "c/V", ("connectorSlot", "ik"): "c/i_K",
                           ("parameter", 1): ("constant", "c/I"), ("parameter", 0): ("algebraic", 0),
                           ("connectorSlot", 5): ("constant", "2"), 2: ("constant", "c/g")}, names)
    assert m["parametersUsedAsAlgebraic"] == [0] and m["parametersUsedAsConstant"] == [2, 0]
    assert m["statesForTransfer"] == [0] and m["algebraicsForTransfer"] == [1]
    assert m["parametersForTransfer"] == [1] and m["slotNames"] == ["vm", "ik", ""]
    with pytest.raises(ValueError):
        CM.parse_mappings({("parameter", 0): ("state", "c/V")}, names)
    with pytest.raises(ValueError):
        CM.parse_mappings({("parameter", 0): "c/unknown"}, names)
    with pytest.raises(ValueError):
        CM.parse_mappings({("connectorSlot", 0): ("constant", "c/E")}, names)


def test_settings_with_mappings():
    from test_only_if_stimulated import reference_settings
    from opendihu_b200 import solver as S
    cfg = reference_settings(n_fibers=2)
    for inst in cfg["RepeatedCall"]["MultipleInstances"]["instances"][0]["StrangSplitting"]["Term1"][
            "MultipleInstances"]["instances"]:
        c = inst["Heun"]["CellML"]
        del c["parametersUsedAsAlgebraic"], c["parametersUsedAsConstant"]
        c["mappings"] = {("parameter", 0): ("constant", "membrane/i_Stim"),
                         ("parameter", 1): ("constant", "sodium_channel/g_Na"),
                         ("connectorSlot", 0): ("state", "membrane/V"),
                         ("connectorSlot", 1): ("algebraic", "potassium_channel/i_K")}
        c["parametersInitialValues"] = [0.0, 100.0]
    s = S.parse_settings(cfg)
    assert list(s.states_for_transfer) == [0]
    assert list(s.algebraics_for_transfer) == [4]
    # slots of the built variant: i_Stim, g_Na, g_K (g_K keeps its model value 36)
    np.testing.assert_allclose(s.parameters[:, 0], [0.0, 100.0, 36.0])


def test_fp64_form_exponentials():
    # Hodgkin-Huxley in FP64: the three exponentials of slope 1/10 are in divisors and come from one reduction, at
    # offsets 0 (alpha_m), -1.5 (alpha_n) and 0.5 (beta_h); exp(u) - 1 has a function of its own; the other three
    # exponentials stand alone
    text = cellml.emit_cuda_model(cellml.builtin_model(H.HH), (), (2, 3, 4))
    f64 = text[text.index("static void rates_f64("):text.index("// FP32 form")]
    body = "\n".join(x for x in f64.split("\n") if not x.startswith("#"))
    names = ("M::exp_group", "FDM_EXPM1_OF(", "FDM_EXP_OF(", "FDM_EXP(", "FDM_DIV(", "FDM_DIV0(")
    assert [body.count(f) for f in names] == [1, 2, 1, 3, 1, 2]
    for b in (Fraction(-3, 2), Fraction(1, 2)):
        e, lo = (float.fromhex(x) for x in re.search(r"\{(.*), (.*)\}", cellml._exp_offset_text(b)).groups())
        assert e == np.exp(float(b)) and cellml._exp_offset_text(b) in f64
        assert abs(np.longdouble(e) + np.longdouble(lo) - np.exp(np.longdouble(float(b)))) <= 1.1e-19 * e


def test_exponentials_far_apart_share_nothing():
    # offsets above 2 and exponentials outside divisors stand alone
    lines = [("R", 0, cellml.parse_expression("1.0/(1.0+exp(STATES[0]))+1.0/(1.0+exp(STATES[0]+2.5))+exp(STATES[0]+1.0)")),
             ("R", 1, cellml.parse_expression("1.0/(1.0+exp(2.0*STATES[0]))+1.0/(2.0+exp(2.0*STATES[0]-1.0))"))]
    em = cellml._Fast64Emitter("R", [], lines)
    assert em.bases == [lines[1][2][2][3][3][2][0]]
    assert sorted(b for _, b in em.members.values()) == [-1, 0]


def test_divisions_that_need_no_special_values():
    # FDM_DIV only where the divisor is known to be finite and away from 0 and the quotient finite; FDM_DIV0 only where
    # dividend and divisor vanish together
    model = lambda *texts: [("R", k, cellml.parse_expression(t)) for k, t in enumerate(texts)]
    lean = ("1.0/(1.0+exp(STATES[0]/10.0))", "STATES[1]/(2.0+exp(STATES[0]))",
            "3.0/(0.2+5.65*pow((STATES[0]+90.0)/100.0, 2.0))", "2.0/(-1.0-exp(STATES[0]))")
    # (1/exp(u) is not exp(-u) where the exponential is approximated)
    general = ("1.0/STATES[0]", "1.0/exp(STATES[0])", "1.0/(1.0+0.5/STATES[1])", "exp(STATES[0])/(1.0+exp(STATES[1]))",
             "STATES[0]/(STATES[1]+1.0)", "1.0/(exp(STATES[0])-1.0)", "STATES[0]/(1.0-exp(STATES[0]/25.0))",
             "(STATES[0]+50.0)/(exp((STATES[0]+51.0)/10.0)-1.0)", "1.0/(1.0+log(STATES[0]))",
             "exp(STATES[1])*(STATES[0]+50.0)/(exp((STATES[0]+50.0)/10.0)-1.0)", "1.0/(1e-305+exp(STATES[0]))")
    together = ("0.1*(STATES[0]+50.0)/(1.0-exp(-(STATES[0]+50.0)/10.0))", "STATES[1]*(STATES[0]-40.0)/(exp((STATES[0]-40.0)*0.2)-1.0)")
    for texts, name in ((lean, "FDM_DIV("), (together, "FDM_DIV0("), (general, "FDM_DIV_ANY(")):
        for text in texts:
            lines = model(text)
            out = cellml._Fast64Emitter("R", [], lines).expr(lines[0][2])
            assert {x for x in ("FDM_DIV(", "FDM_DIV0(", "FDM_DIV_ANY(", " / ") if x in out} == {name}, (text, out)
    # no division: by constants, by powers of them
    for text in ("STATES[0]/3.0", "STATES[0]/pow(0.2, 3.0)"):
        lines = model(text)
        assert "DIV" not in cellml._Fast64Emitter("R", [], lines).expr(lines[0][2])
    # a range known from an algebraic variable
    lines = [("A", 0, cellml.parse_expression("1.0/(1.0+exp(STATES[0]))")), ("R", 0, cellml.parse_expression("1.0/(0.5+ALGEBRAIC[0])"))]
    assert "FDM_DIV(" in cellml._Fast64Emitter("R", [], lines).expr(lines[1][2])


def test_squared_exponentials_stay_in_the_range_of_fp32():
    # the paired FP32 form takes exp(x + b_k) from the square of an exponential of half the slope only where neither the
    # square nor the factor comes near the ends of FP32: at V = 0 the model below is 1/(1 + e^-5) and so on, with
    # exp((V - 900)/20)^2 it would be 0 times infinity
    def squares(shift, factor="1.0"):
        lines = [("R", 0, cellml.parse_expression(
            f"1.0/(1.0+exp((STATES[0]-50.0)/10.0))+1.0/(1.0+exp((STATES[0]-20.0)/10.0))"
            f"+{factor}*exp((STATES[0]-{shift})/20.0)"))]
        repl, groups = cellml._exp_groups(lines, [])
        return cellml._squared_groups(lines, [], repl, groups)
    assert list(squares("75.0")) == [0] and list(squares("75.0", "0.07")) == [0]
    assert squares("900.0") == {} and squares("-900.0") == {} and squares("75.0", "1e9") == {}
