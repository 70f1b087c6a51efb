"""CUDA path against the CPU oracle on the same meshes, initial conditions and step counts.

Tolerances (written per test):
  FP64, no wet/dry: per variable max |q_gpu - q_oracle| <= 1e-12 * max |q_oracle| (relative to the
  variable's scale), L2 errors equal to 1e-12 relative.
  FP32 bulk: the L2 error against the analytic solution within 1.05x of the FP64 oracle's.
  Wet/dry + limiter (threshold branches can flip on last-bit differences): wet-cell counts within
  0.5 %, state within 1e-9 of the variable scale after a short run.
"""
import numpy as np
import pytest

from dgswemv2_b200 import Problem, configs, meshgen
from dgswemv2_b200.types import FUNCTION, LAND

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    """max over variables of max|a-b| / max|b| (per-variable scale)."""
    out = 0.0
    for v in range(3):
        scale = max(np.max(np.abs(b[:, v, :])), 1e-300)
        out = max(out, np.max(np.abs(a[:, v, :] - b[:, v, :])) / scale)
    return out


def run_pair(oracle, mesh, cfg, nsteps, **kw):
    P = Problem(cfg, mesh, **kw)
    O = oracle.problem(cfg, mesh, n_threads=8)
    q0g, q0o = P.get_state(), O.get_state()
    assert rel_err(q0g, q0o) <= 1e-13, "initial projection"
    P.step_serial(nsteps)
    O.step(nsteps)
    return P, O


def test_config1_manufactured_p1_1000_steps(oracle):
    """Config 1: 800 triangles, p=1, SSP-RK2, dt=1 s, 1000 steps, FP64."""
    mesh, cfg = configs.config1()
    P, O = run_pair(oracle, mesh, cfg, 1000)
    e = rel_err(P.get_state(), O.get_state())
    assert e <= 1e-12, e
    lg, lo = P.compute_residual_L2(), O.l2_error()
    assert abs(lg - lo) <= 1e-12 * lo, (lg, lo)
    assert P.time()[0] == O.time() == 1000.0


@pytest.mark.parametrize("tile", [128, 256])
def test_p2_rk3_jittered(oracle, tile):
    """p=2, SSP-RK3, jittered mesh (config-2 discretisation on a small mesh), 100 steps, FP64."""
    mesh, cfg = configs.manufactured(24, p=2, rk=(3, 3), dt=2.0, jitter=0.2, seed=2)
    P, O = run_pair(oracle, mesh, cfg, 100, tile=tile)
    e = rel_err(P.get_state(), O.get_state())
    assert e <= 1e-12, e
    assert abs(P.compute_residual_L2() - O.l2_error()) <= 1e-12 * O.l2_error()


def test_stage_by_stage_and_graphs_agree(oracle):
    """stage_serial calls, graph-captured steps and plain launches give the same bits."""
    mesh, cfg = configs.manufactured(10, p=1, rk=(3, 3), dt=5.0)
    A = Problem(cfg, mesh, use_graphs=True)
    B = Problem(cfg, mesh, use_graphs=False)
    C = Problem(cfg, mesh)
    A.step_serial(7)
    B.step_serial(7)
    for _ in range(21):
        C.stage_serial()
    assert np.array_equal(A.get_state(), B.get_state())
    assert np.array_equal(A.get_state(), C.get_state())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_multi_step_graphs_agree_with_plain_launches(precision):
    """Batches of 8 steps replay one captured 8-step graph; the remainder replays one-step graphs. 21 steps
    (two 8-step graphs and five one-step graphs, across both swap parities) give the same bits as plain
    launches, on the p = 2 manufactured case (stage increments in FP32) and on the wet/dry + limiter bowl,
    also when a batch starts in the middle of a step."""
    cases = [configs.manufactured(12, p=2, rk=(3, 3), dt=2.0, jitter=0.2, precision=precision),
             configs.config3(nq=32, dt=1.0, precision=precision)]
    for mesh, cfg in cases:
        A = Problem(cfg, mesh, use_graphs=True)
        B = Problem(cfg, mesh, use_graphs=False)
        A.step_serial(21)
        B.step_serial(21)
        assert np.array_equal(A.get_state(), B.get_state())
        assert np.array_equal(A.get_wet(), B.get_wet())
        A.stage_serial()
        B.stage_serial()
        A.step_serial(17)
        B.step_serial(17)
        assert np.array_equal(A.get_state(), B.get_state())
        assert A.time() == B.time()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_register_budget_and_tile_order_do_not_change_results(precision):
    """The autotuner's knobs change speed only. The tile order gives the same bits (tiles are independent
    and each is computed in a fixed order), on a p = 2 manufactured run and on the wet/dry + limiter bowl.
    The alternative register budget is a separate compilation of the same kernel: it gives the same bits
    except in FP64 with the analytic source, where the compiler fuses a multiply-add of the source terms
    differently in the two builds (measured 5e-17 of the state's scale; allowed 1e-15)."""
    cases = [("mms", configs.manufactured(16, p=2, rk=(3, 3), dt=2.0, jitter=0.2, precision=precision)),
             ("bowl", configs.config3(nq=48, dt=1.0, precision=precision))]
    for name, (mesh, cfg) in cases:
        runs = {}
        for occ, order in ((0, 0), (1, 0), (0, 1), (1, 1)):
            P = Problem(cfg, mesh, occupancy=occ, tile_order=order)
            assert (P.info.occupancy, P.info.tile_order) == (occ, order)
            P.step_serial(15)
            runs[occ, order] = P.get_state()
        for occ in (0, 1):
            assert np.array_equal(runs[occ, 1], runs[occ, 0])  # tile order: bit for bit
        exact = not (precision == "fp64" and name == "mms")
        q0, q1 = runs[0, 0], runs[1, 0]
        if exact:
            assert np.array_equal(q1, q0)
        else:
            assert np.abs(q1 - q0).max() <= 1e-15 * np.abs(q0).max()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_autotuned_shared_memory_choice_does_not_change_results(precision):
    """The autotuner also chooses between the stage kernel with compile-time shared-memory capacities and the
    one sized to the mesh's largest tile (dgsw_info.smem_capped). Both do the same arithmetic in the same
    order: an autotuned handle gives the same bits as a handle built with its tile, budget and order, which
    takes the capped kernel wherever the mesh fits the caps."""
    mesh, cfg = configs.manufactured(128, p=2, rk=(3, 3), dt=1.0, jitter=0.2, precision=precision)
    A = Problem(cfg, mesh, tile=-1)
    B = Problem(cfg, mesh, tile=A.info.tile, occupancy=A.info.occupancy, tile_order=A.info.tile_order)
    A.step_serial(12)
    B.step_serial(12)
    assert np.array_equal(A.get_state(), B.get_state())


def test_renumbering_does_not_change_results(oracle):
    mesh, cfg = configs.manufactured(12, p=2, rk=(2, 2), dt=5.0, jitter=0.15)
    A = Problem(cfg, mesh, renumber=True)
    B = Problem(cfg, mesh, renumber=False)
    A.step_serial(20)
    B.step_serial(20)
    assert np.array_equal(A.get_state(), B.get_state())


def test_fp32_bulk_l2_within_5_percent(oracle):
    """FP32 bulk path: L2 error vs the analytic solution within 1.05x of the FP64 oracle's."""
    mesh, cfg = configs.manufactured(20, p=2, rk=(3, 3), dt=2.0, jitter=0.2, precision="fp32")
    P = Problem(cfg, mesh)
    cfg64 = configs.manufactured(20, p=2, rk=(3, 3), dt=2.0, jitter=0.2)[1]
    O = oracle.problem(cfg64, mesh, n_threads=8)
    P.step_serial(200)
    O.step(200)
    lg, lo = P.compute_residual_L2(), O.l2_error()
    assert lg <= 1.05 * lo, (lg, lo)
    assert rel_err(P.get_state(), O.get_state()) < 1e-4


def test_fp32_l2_stays_within_5_percent_over_2000_steps():
    """Config-2 discretisation (p = 2, SSP-RK3, jittered) at 64 x 64 quads for 2,000 steps of dt = 2 s: the
    FP32 path's L2 error against the analytic solution within 1.05x of the FP64 path's."""
    l2 = {}
    for prec in ("fp32", "fp64"):
        mesh, cfg = configs.manufactured(64, p=2, rk=(3, 3), dt=2.0, jitter=0.2, precision=prec)
        P = Problem(cfg, mesh)
        P.step_serial(2000)
        l2[prec] = P.compute_residual_L2()
    assert l2["fp32"] <= 1.05 * l2["fp64"], l2


@pytest.mark.parametrize("p,rk,tile", [(2, (3, 3), 256), (1, (3, 3), 128), (2, (5, 4), 128)])
def test_fp32_stage_increments(p, rk, tile):
    """FP32 arithmetic keeps the intermediate stage states as FP32 increments from the carried state (kept
    as two FP32 parts) wherever only the stage kernel reads them: no wetting/drying, limiter or levees, and
    three or more stages (a two-stage scheme keeps FP64 stage states). Against the same FP32 path with FP64
    stage states (fp64_stages), on the config-2 discretisation at 24 x 24 quads for 300 steps: each variable within 1e-5 of its scale and the L2 errors within 0.1 %. Graph-replayed steps,
    plain launches and stage-by-stage calls give the same bits, and a state read and written back through
    the host API in the middle of a step (Q_s = q_0 + d_s formed in FP64, then split again) continues
    within 1e-6 of the undisturbed run. SSP(5,4) covers combinations with several increment terms and a
    stored stage solution."""
    mesh, cfg = configs.manufactured(24, p=p, rk=rk, dt=2.0, jitter=0.2, precision="fp32")
    ns = rk[0]
    A = Problem(cfg, mesh, tile=tile)
    B = Problem(cfg, mesh, tile=tile, fp64_stages=True)
    assert A.info.stage_increments == 1 and B.info.stage_increments == 0
    m2, c2 = configs.manufactured(8, p=p, rk=(2, 2), dt=2.0, precision="fp32")
    assert Problem(c2, m2).info.stage_increments == 0
    A.step_serial(300)
    B.step_serial(300)
    assert rel_err(A.get_state(), B.get_state()) <= 1e-5
    la, lb = A.compute_residual_L2(), B.compute_residual_L2()
    assert abs(la - lb) <= 1e-3 * lb, (la, lb)
    G = Problem(cfg, mesh, tile=tile, use_graphs=False)
    S = Problem(cfg, mesh, tile=tile)
    R = Problem(cfg, mesh, tile=tile)
    G.step_serial(300)
    for _ in range(3 * ns):
        S.stage_serial()
    S.step_serial(297)
    assert np.array_equal(G.get_state(), A.get_state())
    assert np.array_equal(S.get_state(), A.get_state())
    # through the host API in the middle of a step: read the stage state, write it back, finish the run
    R.step_serial(299)
    R.stage_serial()
    mid = R.get_state()
    assert R.time()[2] == 1
    R.set_state(mid)
    assert rel_err(R.get_state(), mid) <= 1e-7
    R.step_serial(1)
    assert rel_err(R.get_state(), A.get_state()) <= 1e-6


def test_fp32_stage_increments_behind_the_host_api():
    """Every host-API read of a state in the middle of a step forms it from the stage increments, and every
    write splits it again: after one stage of step 41 the handle with stage increments and the one with
    FP64 stage states agree on the mass (the current stage's state), the L2 error (the carried state), the
    writers' values and the state copied device to device, within the FP32 path's rounding; a state
    written device to device mid-step reads back unchanged up to the increment's FP32 rounding."""
    import torch

    mesh, cfg = configs.manufactured(16, p=2, rk=(3, 3), dt=2.0, jitter=0.2, precision="fp32")
    A = Problem(cfg, mesh)
    B = Problem(cfg, mesh, fp64_stages=True)
    assert A.info.stage_increments == 1 and B.info.stage_increments == 0
    for P in (A, B):
        P.step_serial(40)
        P.stage_serial()
    assert A.time() == B.time() and A.time()[2] == 1
    assert abs(A.mass() - B.mass()) <= 1e-7 * abs(B.mass())
    la, lb = A.compute_residual_L2(), B.compute_residual_L2()
    assert abs(la - lb) <= 1e-4 * lb, (la, lb)
    pa, ca, _, _ = A.postprocess()
    pb, cb, _, _ = B.postprocess()
    assert np.abs(pa - pb).max() <= 1e-5 * np.abs(pb).max()
    assert np.abs(ca - cb).max() <= 1e-5 * np.abs(cb).max()
    d = torch.empty((A.ne, 3, A.nd), dtype=torch.float64, device="cuda")
    A.get_state_device(d.data_ptr())
    torch.cuda.synchronize()
    qa = d.cpu().numpy()
    assert rel_err(qa, A.get_state()) == 0.0
    assert rel_err(qa, B.get_state()) <= 1e-5
    A.set_state_device(d.data_ptr())
    torch.cuda.synchronize()
    assert rel_err(A.get_state(), qa) <= 1e-7
    A.step_serial(5)
    B.step_serial(5)
    assert rel_err(A.get_state(), B.get_state()) <= 1e-5


def test_fp32_l2_on_a_limited_p2_run():
    """FP32 at equal L2 on a limited p = 2 run: the config-2 discretisation (manufactured solution, p = 2,
    SSP-RK3, jittered) at 32 x 32 quads with the Cockburn-Shu limiter (M = 1e-8), 500 steps of dt = 2 s. The
    limiter acts on about 7 % of the elements per stage and a flipped write-back decision zeroes an
    element's p = 2 modes; the FP32 path's L2 error against the analytic solution stays within 1.05x of the
    FP64 path's. (Thacker's bowl at p = 2 with wetting/drying and the limiter is no test case: the FP64
    oracle itself produces a NaN there after 120-150 s of simulated time, at every time step tried.)"""
    l2 = {}
    for prec in ("fp32", "fp64"):
        mesh, cfg = configs.manufactured(32, p=2, rk=(3, 3), dt=2.0, jitter=0.2, precision=prec)
        cfg.slope_limiting = True
        P = Problem(cfg, mesh)
        P.step_serial(500)
        l2[prec] = P.compute_residual_L2()
        assert 0.02 <= float(np.mean(P.get_limited())) <= 0.2, np.mean(P.get_limited())
    assert l2["fp32"] <= 1.05 * l2["fp64"], l2


def test_fp32_limiter_against_the_fp64_limiter():
    """The FP32 path limits in FP32 arithmetic on FP64 differences (limiter_kernel.cuh). On the config-3 bowl
    (wetting/drying, limiter, p = 1) at 128 x 128 quads for 400 steps, against the same FP32 path with the
    FP64 limiter: limiter decisions agree on >= 99.5 % of the cells, wet counts within 0.5 %, states
    within 1e-3 of each variable's scale, mass to 1e-7 relative (the FP32 bulk arithmetic's bound; the
    limiter keeps each element's FP64 mean), and the L2 error against Thacker's solution within 1.05x of
    the FP64 path's."""
    mesh, cfg = configs.config3(nq=128, dt=0.5, precision="fp32")
    A = Problem(cfg, mesh)
    B = Problem(cfg, mesh, fp64_limiter=True)
    m64, c64 = configs.config3(nq=128, dt=0.5)
    C = Problem(c64, m64)
    m0 = A.mass()
    for P in (A, B, C):
        P.step_serial(400)
    assert np.mean(A.get_limited() != B.get_limited()) <= 0.005
    assert A.get_limited().sum() > 100  # the limiter acts
    assert abs(int(A.get_wet().sum()) - int(B.get_wet().sum())) <= 0.005 * mesh.n_elems
    assert rel_err(A.get_state(), B.get_state()) <= 1e-3
    assert abs(A.mass() / m0 - 1) <= 1e-7
    assert A.compute_residual_L2() <= 1.05 * C.compute_residual_L2()


def test_land_boundaries_conserve_mass(oracle):
    """Closed basin with land boundaries: FP64 mass is conserved to rounding."""
    mesh = meshgen.quad_mesh(16, 16, corners=((0, 0), (1000, 0), (1000, 1000), (0, 1000)), bc=(LAND,) * 4,
                             jitter=0.2, seed=5, bathymetry=meshgen.bath_flat(5.0))
    cfg = configs.ProblemConfig(p=2, rk_nstages=3, rk_order=3, dt=0.5, ic_type=1,
                                function_set=configs.FN_GAUSSIAN_HUMPS,
                                fn_params=configs.humps_params([(0.3, 500.0, 400.0, 120.0)]))
    P, O = run_pair(oracle, mesh, cfg, 200)
    assert rel_err(P.get_state(), O.get_state()) <= 1e-12
    m0 = O.mass()
    assert abs(P.mass() - m0) <= 1e-12 * m0


def test_wet_dry_and_limiter_bowl(oracle):
    """Thacker bowl with wetting/drying and the Cockburn-Shu limiter (config-3 physics, 48x48 quads)."""
    mesh, cfg = configs.config3(nq=48, dt=1.0)
    P, O = run_pair(oracle, mesh, cfg, 50)
    wg, wo = P.get_wet(), O.get_wet()
    assert abs(int(wg.sum()) - int(wo.sum())) <= max(2, 0.005 * mesh.n_elems)
    assert rel_err(P.get_state(), O.get_state()) <= 1e-9
    lim_g, lim_o = P.get_limited(), O.limited_flags()
    assert np.mean(lim_g != lim_o) <= 0.005


def test_nan_is_reported_not_aborted(oracle):
    """A NaN injected into the host state comes back as DGSW_ERR_NAN with the element ID."""
    from dgswemv2_b200._lib import DgswError

    mesh, cfg = configs.manufactured(6, p=1)
    P = Problem(cfg, mesh)
    q = P.get_state()
    q[5, 1, 0] = np.nan
    P.set_state(q)
    with pytest.raises(DgswError) as ei:
        P.step_serial(1)
    assert ei.value.status == 4
    assert "element" in str(ei.value)


def test_nan_mid_batch_reports_the_first_stage_and_element(oracle):
    """A NaN that enters in the middle of a batch of steps is reported as the reference's per-stage
    scrutiny reports it (rkdg_swe_proc_serial_step.hpp:59-65): at the first stage whose new state holds a
    NaN, the smallest element ID there - not the smallest ID carrying a NaN when the batch ends, by which
    time the NaN has spread. The NaN goes into one element's stage-1 state; the oracle, stepped stage by
    stage, gives the expected stage and element."""
    from dgswemv2_b200._lib import DgswError

    mesh, cfg = configs.manufactured(10, p=1, rk=(3, 3), dt=5.0)
    P = Problem(cfg, mesh)
    O = oracle.problem(cfg, mesh)
    P.stage_serial()
    O.stage()
    q = P.get_state()
    bad = 117
    q[bad, 2, 1] = np.nan
    P.set_state(q)
    O.set_state(q)
    expected = None
    for k in range(1, 9):  # stages 1, 2 of step 0, then step 1, ...
        try:
            O.stage()
        except RuntimeError as e:  # the oracle's scrutiny stops at the first stage with a NaN
            rows = np.nonzero(np.isnan(O.get_state()).any(axis=(1, 2)))[0]
            expected = (k // 3, k % 3, int(rows.min()))
            assert "NaN found at element %d" % expected[2] in str(e)
            break
    assert expected is not None and expected[:2] == (0, 1)
    assert expected[2] < bad  # a neighbour with a smaller ID is hit at the same stage
    with pytest.raises(DgswError) as ei:
        P.step_serial(4)
    assert ei.value.status == 4
    assert "NaN found at element %d (step %d, stage %d)" % (expected[2], expected[0], expected[1]) in str(ei.value)


def test_fp32_bowl_keeps_the_fp64_wet_set():
    """Bowl with Gaussian humps at 131,072 triangles, FP32 bulk arithmetic: a flattened dry cell sits at
    depth h_o, which the FP64 threshold 1e6 h_o eps separates from wet only if the stage states carry
    FP64 (an FP32-stored surface elevation is off by about 1e-6 m). The FP32 run keeps exactly the FP64
    run's wet set for 200 steps, stays finite, and conserves mass to 1e-7 (FP64: 1e-12)."""
    P = {}
    for prec in ("fp32", "fp64"):
        mesh, cfg = configs.bowl_humps(nq=256, seed=0, dt=0.25, precision=prec)
        P[prec] = Problem(cfg, mesh)
    m0 = {k: v.mass() for k, v in P.items()}
    for _ in range(2):
        for k in P:
            P[k].step_serial(100)
        assert np.array_equal(P["fp32"].get_wet(), P["fp64"].get_wet())
    assert np.isfinite(P["fp32"].get_state()).all()
    assert abs(P["fp32"].mass() / m0["fp32"] - 1) <= 1e-7
    assert abs(P["fp64"].mass() / m0["fp64"] - 1) <= 1e-12


@pytest.mark.parametrize("p", [1, 2])
def test_trouble_indicator_matches_oracle(oracle, p):
    """check_trouble (swe_trouble_check.hpp:6-116), which the reference computes in every limiter pass
    without using it: indicator values within 1e-9 relative (1e-12 absolute) and troubled flags equal to
    the oracle's after the same steps (flags may differ only where I is within 1e-9 of the threshold 1)."""
    # the indicator divides by r^((p+1)/2) in mesh units, so it trips on a unit-size basin (metre-size
    # meshes never reach I > 1): a Gaussian hump on 1 m of still water in a 1 m x 1 m box
    from dgswemv2_b200.types import ProblemConfig

    mesh = meshgen.quad_mesh(12, 12, bc=(LAND,) * 4, jitter=0.15, seed=2, bathymetry=meshgen.bath_flat(1.0))
    cfg = ProblemConfig(p=p, rk_nstages=2, rk_order=2, dt=5e-4, g=9.81, wetting_drying=True, h_o=0.01,
                        slope_limiting=True, sl_M=1.0e-8, sl_nu=1.5, ic_type=1,
                        function_set=configs.FN_GAUSSIAN_HUMPS,
                        fn_params=configs.humps_params([(0.9, 0.5, 0.5, 0.05)]), precision="fp64")
    P = Problem(cfg, mesh)
    P.set_trouble(True)
    O = oracle.problem(cfg, mesh, n_threads=8)
    seen = 0
    for _ in range(3):
        P.step_serial(5)
        O.step(5)
        Ig, tg = P.get_trouble()
        Io, to = O.trouble()
        assert np.allclose(Ig, Io, rtol=1e-9, atol=1e-12), np.max(np.abs(Ig - Io))
        near = np.abs(Io - 1.0) < 1e-9
        assert np.array_equal(tg[~near] != 0, to[~near] != 0)
        seen += int(to.sum())
    assert seen > 0


TIDE_CASES = [
    # p, rk, dt, friction, lower bound cf, ramp (days), river flow
    (1, (2, 2), 2.0, "chezy", 0.0025, 0.01, True),
    (2, (3, 3), 1.0, "manning", 0.0005, 0.01, True),
    (1, (3, 3), 2.0, None, 0.0, 0.0, False),
    (2, (2, 2), 1.0, "chezy", 0.004, 0.0, True),
]


@pytest.mark.parametrize("case", TIDE_CASES, ids=lambda c: "p%d-%s-ramp%g" % (c[0], c[3], c[5]))
def test_tidal_channel_matches_oracle(oracle, case):
    """Tide and flow boundaries (M2 + K1 tide with amplitude/phase varying along the open end, steady +
    periodic river flow), the forcing ramp and Chezy / Manning friction, FP64: per-variable state within
    1e-12 of the oracle's scale after 300 steps."""
    p, rk, dt, fr, cf, ramp, flow = case
    mesh, cfg = configs.tidal_channel(p=p, rk=rk, dt=dt, friction=fr, cf=cf, ramp_days=ramp, flow=flow)
    P, O = run_pair(oracle, mesh, cfg, 300)
    q = O.get_state()
    assert np.abs(q[:, 0, 0]).max() > 0.05  # the tide has entered the channel
    e = rel_err(P.get_state(), q)
    assert e <= 1e-12, e
    assert P.time()[0] == O.time()


def test_tidal_channel_fp32_bulk(oracle):
    """FP32 bulk arithmetic with FP64 forcing evaluation and states: within 1e-4 of the FP64 oracle's
    per-variable scale after 300 steps."""
    mesh, cfg = configs.tidal_channel(p=2, rk=(3, 3), dt=1.0, friction="manning", cf=0.0005, precision="fp32")
    P = Problem(cfg, mesh)
    cfg64 = configs.tidal_channel(p=2, rk=(3, 3), dt=1.0, friction="manning", cf=0.0005)[1]
    O = oracle.problem(cfg64, mesh, n_threads=8)
    P.step_serial(300)
    O.step(300)
    e = rel_err(P.get_state(), O.get_state())
    assert e < 1e-4, e


def test_tidal_channel_ensemble_matches_single_runs(oracle):
    """Members with their own tide / flow data and Manning n in one ensemble handle give each member's
    single-handle result."""
    from dgswemv2_b200 import ensemble

    cases = [configs.tidal_channel(nx=12, ny=4, friction="manning", cf=0.0005, seed=s, jitter=0.1 * s)
             for s in (1, 2, 3)]
    meshes = [m for m, _ in cases]
    cfg = cases[0][1]
    E = ensemble(cfg, meshes, tile=0)
    E.step_serial(100)
    q = E.get_state()
    for k, m in enumerate(meshes):
        first, n = E.member_range(k)
        P = Problem(cfg, m)
        P.step_serial(100)
        assert rel_err(q[first:first + n], P.get_state()) <= 1e-12, k


def test_tide_face_without_data_is_a_mesh_error():
    from dgswemv2_b200._lib import DgswError

    mesh, cfg = configs.tidal_channel(nx=6, ny=3, flow=False)
    mesh.forcing = []
    with pytest.raises(DgswError, match="unable to find tide data") as ei:
        Problem(cfg, mesh)
    assert ei.value.status == 2


@pytest.mark.parametrize("p, rk, dt, steps", [(1, (2, 2), 2.0, 600), (2, (3, 3), 1.0, 1000)])
def test_levee_channel_matches_oracle(oracle, p, rk, dt, steps):
    """Levee interfaces (ISP::Levee): the tide overtops a barrier across the channel (reflective,
    subcritical and supercritical weir branches); FP64 state within 1e-12 of the oracle's scale."""
    mesh, cfg = configs.levee_channel(p=p, rk=rk, dt=dt)
    P, O = run_pair(oracle, mesh, cfg, steps)
    q = O.get_state()
    xc = mesh.node_xyz[mesh.elem_nodes, 0].mean(1)
    assert q[xc > 5000, 0, 0].mean() > 0.05  # water has come over the levee
    e = rel_err(P.get_state(), q)
    assert e <= 1e-12, e


def test_levee_floods_dry_land(oracle):
    """Overtopping onto dry land (wetting/drying, gravity dropped on the dry receiving side): wet-cell
    counts within 0.5 %, state within 1e-9 of the variable scale."""
    mesh, cfg = configs.levee_channel(p=1, dt=2.0, dry_right=True)
    P, O = run_pair(oracle, mesh, cfg, 600)
    wg, wo = P.get_wet(), O.get_wet()
    assert int(wo.sum()) > mesh.n_elems // 2 + 10  # the dry half has started to flood
    assert abs(int(wg.sum()) - int(wo.sum())) <= max(2, 0.005 * mesh.n_elems)
    assert rel_err(P.get_state(), O.get_state()) <= 1e-9


def test_levee_channel_fp32_bulk(oracle):
    mesh, cfg = configs.levee_channel(p=2, rk=(3, 3), dt=1.0, precision="fp32")
    P = Problem(cfg, mesh)
    O = oracle.problem(configs.levee_channel(p=2, rk=(3, 3), dt=1.0)[1], mesh, n_threads=8)
    P.step_serial(1000)
    O.step(1000)
    e = rel_err(P.get_state(), O.get_state())
    assert e < 1e-3, e


def test_levee_ensemble_matches_single_runs(oracle):
    """Members with their own barriers, levee data and tide blocks in one ensemble handle give each
    member's single-handle result (levee interfaces indexed across members)."""
    from dgswemv2_b200 import ensemble

    cases = [configs.levee_channel(nx=12 + 2 * s, ny=4, seed=s, crest=0.1 + 0.02 * s) for s in (1, 2, 3)]
    meshes = [m for m, _ in cases]
    cfg = cases[0][1]
    E = ensemble(cfg, meshes, tile=0)
    E.step_serial(700)
    q = E.get_state()
    for k, m in enumerate(meshes):
        first, n = E.member_range(k)
        P = Problem(cfg, m)
        P.step_serial(700)
        assert rel_err(q[first:first + n], P.get_state()) <= 1e-12, k


def test_levee_with_limiter_and_flooding(oracle):
    """The slope limiter across levee interfaces (the element over the barrier is a neighbour) while the
    tide floods dry land behind the levee: wet counts within 0.5 %, state within 1e-9, limiter decisions
    within 0.5 %."""
    mesh, cfg = configs.levee_channel(p=1, dt=2.0, dry_right=True, limiter=True)
    P, O = run_pair(oracle, mesh, cfg, 600)
    wg, wo = P.get_wet(), O.get_wet()
    assert int(wo.sum()) > mesh.n_elems // 2 + 10
    assert abs(int(wg.sum()) - int(wo.sum())) <= max(2, 0.005 * mesh.n_elems)
    assert rel_err(P.get_state(), O.get_state()) <= 1e-9
    assert np.mean(P.get_limited() != O.limited_flags()) <= 0.005


@pytest.mark.parametrize("which", ["tidal", "levee"])
def test_spherical_correction_with_forcing_and_levees(oracle, which):
    """The spherical correction factor (spherical_projection) on the tide / flow ghost fluxes and on both
    sides of levee interfaces: FP64 within 1e-12 of the oracle after 300 steps."""
    if which == "tidal":
        mesh, cfg = configs.tidal_channel(p=2, rk=(3, 3), dt=1.0, friction="manning", cf=0.0005)
    else:
        mesh, cfg = configs.levee_channel(p=1, dt=2.0)
    mesh.node_xyz = mesh.node_xyz.copy()
    mesh.node_xyz[:, 1] += 3.3e6  # about 30 degrees north on the projection cylinder
    cfg.spherical = True
    cfg.sp_lat0_deg = 30.0
    P, O = run_pair(oracle, mesh, cfg, 300)
    e = rel_err(P.get_state(), O.get_state())
    assert e <= 1e-12, e


def _north(mesh, cfg):
    """The problem moved to about 30 degrees north on the projection cylinder."""
    mesh.node_xyz = mesh.node_xyz.copy()
    mesh.node_xyz[:, 1] += 3.3e6
    cfg.spherical = True
    cfg.sp_lat0_deg = 30.0
    return mesh, cfg


@pytest.mark.parametrize("precision,bar", [("fp64", 1e-9), ("fp32", 1e-4)])
@pytest.mark.parametrize("p,tile", [(1, 128), (1, 256), (2, 128)])
def test_spherical_correction_at_a_shoreline(oracle, p, tile, precision, bar):
    """The spherical correction together with wetting/drying: a bowl with a hump that floods and drains its shore, with
    wet in sides against dry ex sides and the other way round. FP64 as for the other wet/dry runs; FP32: the
    pressure and bathymetry terms, g h^2 / 2 with h up to 10 m, cancel to a surface slope's worth, which leaves
    2^-24 x 10 x (10 / 0.5 m) of the momentum's scale, 1e-5, per unit of condition; the bar is ten times that."""
    mesh, cfg = configs.bowl_humps(nq=40, dt=1.0, limiter=False, precision=precision)
    mesh, cfg = _north(mesh, cfg)
    cfg.p, cfg.rk_nstages, cfg.rk_order = p, p + 1, p + 1
    cfg.fn_params = configs.humps_params([(3.0, 500.0, 3.3e6 + 2300.0, 600.0)])
    P = Problem(cfg, mesh, tile=tile)
    O = oracle.problem(cfg, mesh, n_threads=8)
    intf = P.topology()[2]
    before = P.get_wet().astype(bool)
    in_wet, ex_wet = before[intf[:, 0]], before[intf[:, 1]]
    assert (in_wet & ~ex_wet).sum() > 20 and (~in_wet & ex_wet).sum() > 20
    P.step_serial(160)
    O.step(160)
    wg, wo = P.get_wet(), O.get_wet()
    assert (wo.astype(bool) != before).sum() > 20  # the shoreline has moved
    assert np.count_nonzero(wg != wo) <= (0 if precision == "fp64" else 2)
    e = rel_err(P.get_state(), O.get_state())
    assert e <= bar, e


def test_spherical_correction_fp32(oracle):
    """FP32 arithmetic with the spherical correction on the forced channel, without and with stage increments: the
    bar of the FP32 channel without it."""
    mesh, cfg64 = _north(*configs.tidal_channel(p=2, rk=(3, 3), dt=1.0))
    cfg = _north(*configs.tidal_channel(p=2, rk=(3, 3), dt=1.0, precision="fp32"))[1]
    O = oracle.problem(cfg64, mesh, n_threads=8)
    O.step(300)
    for fp64_stages in (False, True):
        P = Problem(cfg, mesh, fp64_stages=fp64_stages)
        P.step_serial(300)
        e = rel_err(P.get_state(), O.get_state())
        assert e < 1e-4, e


def test_manning_friction_in_drying_cells(oracle):
    """Manning friction while the levee floods dry land (depths near h_o make g n^2 / h^(1/3) large):
    wet counts within 0.5 %, state within 1e-9."""
    mesh, cfg = configs.levee_channel(p=1, dt=2.0, dry_right=True, friction="manning", cf=0.0005)
    P, O = run_pair(oracle, mesh, cfg, 600)
    wg, wo = P.get_wet(), O.get_wet()
    assert int(wo.sum()) > mesh.n_elems // 2 + 10
    assert abs(int(wg.sum()) - int(wo.sum())) <= max(2, 0.005 * mesh.n_elems)
    assert rel_err(P.get_state(), O.get_state()) <= 1e-9


def test_forcing_block_with_a_repeated_node_is_rejected():
    """A node listed twice in one block would shift its constituents in the reference's per-node lists;
    the library rejects it with DGSW_ERR_MESH instead."""
    from dgswemv2_b200._lib import DgswError

    mesh, cfg = configs.tidal_channel(nx=6, ny=3, flow=False)
    b = mesh.forcing[0]
    b.nodes = np.concatenate([b.nodes, b.nodes[:1]])
    b.amplitude = np.concatenate([b.amplitude, b.amplitude[:, :1]], 1)
    b.phase = np.concatenate([b.phase, b.phase[:, :1]], 1)
    with pytest.raises(DgswError, match="twice") as ei:
        Problem(cfg, mesh)
    assert ei.value.status == 2
    mesh2, cfg2 = configs.levee_channel(nx=6, ny=3)
    mesh2.levee_pairs = mesh2.levee_pairs[1:]
    mesh2.levee_data = mesh2.levee_data[1:]
    with pytest.raises(DgswError, match="unable to find levee data") as ei:
        Problem(cfg2, mesh2)
    assert ei.value.status == 2


def test_p2_limiter_matches_where_decisions_are_clear(oracle):
    """p = 2 with the Cockburn-Shu limiter on a steep hump (many elements limited from the first stage,
    far from the 1e-12 write-back threshold): state within 1e-12 and identical limiter decisions over
    the first step. Over long runs with small states the 1e-12 relative-change test can flip on
    last-bit differences, and a flip zeroes that element's p = 2 modes, so long p = 2 limiter runs agree
    only statistically (the reference itself would differ between compilers the same way)."""
    mesh = meshgen.quad_mesh(16, 16, corners=((0, 0), (1000, 0), (1000, 1000), (0, 1000)), bc=(LAND,) * 4,
                             jitter=0.15, seed=6, bathymetry=meshgen.bath_flat(5.0))
    cfg = configs.ProblemConfig(p=2, rk_nstages=3, rk_order=3, dt=0.5, ic_type=1,
                                function_set=configs.FN_GAUSSIAN_HUMPS, slope_limiting=True, sl_M=1e-8, sl_nu=1.5,
                                fn_params=configs.humps_params([(1.0, 500.0, 500.0, 60.0)]))
    P = Problem(cfg, mesh, use_graphs=False)
    O = oracle.problem(cfg, mesh, n_threads=8)
    for _ in range(3):
        P.stage_serial()
        O.stage()
        lg, lo = P.get_limited(), O.limited_flags()
        assert np.array_equal(lg, lo)
        assert rel_err(P.get_state(), O.get_state()) <= 1e-12
    assert lo.sum() > 10


@pytest.mark.parametrize("nx,ny", [(1, 1), (9, 7), (8, 8), (13, 5), (64, 2)])
@pytest.mark.parametrize("p,tile", [(1, 128), (1, 256), (2, 128), (2, 256)])
def test_tile_edges_and_remainders(oracle, nx, ny, p, tile):
    """Meshes of 2, 126, 128, 130 and 256 triangles (less than a tile, one exactly, a remainder of two, a strip
    whose tiles are mostly halo and boundary faces) with tide, river and land faces, and stage and step calls mixed:
    the last element's face slots, the ghost slots behind the halo slots and the forcing values of the second
    copy of the step's time. Bar: 1e-12 of each variable's scale, as for the other FP64 runs here."""
    mesh, cfg = configs.tidal_channel(nx, ny, p=p, rk=(2, 2) if p == 1 else (3, 3), dt=0.5, jitter=0.1 if nx > 1 else 0.0)
    P = Problem(cfg, mesh, tile=tile)
    O = oracle.problem(cfg, mesh)
    q = np.random.default_rng(5).uniform(-0.02, 0.02, (P.ne, 3, P.nd))  # every variable well above rounding
    q[:, 1:] *= 10.0
    P.set_state(q)
    O.set_state(q)
    P.step_serial(3)
    for _ in range(cfg.rk_nstages):
        P.stage_serial()
    P.step_serial(9)
    O.step(13)
    assert rel_err(P.get_state(), O.get_state()) <= 1e-12


@pytest.mark.parametrize("nx,ny", [(1, 1), (9, 7), (8, 8), (13, 5), (64, 2)])
@pytest.mark.parametrize("p,tile", [(1, 128), (1, 256), (2, 128), (2, 256)])
def test_tile_edges_and_remainders_fp32(oracle, nx, ny, p, tile):
    """The same meshes in FP32, at p = 2 with stage increments (its own kernel) and with FP64 stage states: ghost slots
    behind the halo slots, halo copies by threads past the last element, the p = 2 faces' run-time table. A step changes a
    mode by dt / dx (at most 0.5 / 150) times flux and volume terms of up to g ze h = 2, some ten of them, each within a
    few 2^-24: 13 steps leave up to 13 x 10 x 0.0033 x 2 x 2^-23 = 1e-7, 5e-6 of the smallest scale (ze, 0.02) if all
    add up, a tenth of it as they come. Bar: 2e-6 (measured 2e-7). A wrong slot moves a flux by a part of itself, 1e-3 of
    the scale in one stage."""
    rk, jitter = ((2, 2) if p == 1 else (3, 3)), (0.1 if nx > 1 else 0.0)
    mesh, cfg64 = configs.tidal_channel(nx, ny, p=p, rk=rk, dt=0.5, jitter=jitter)
    cfg = configs.tidal_channel(nx, ny, p=p, rk=rk, dt=0.5, jitter=jitter, precision="fp32")[1]
    O = oracle.problem(cfg64, mesh)
    q = np.random.default_rng(5).uniform(-0.02, 0.02, (mesh.n_elems, 3, (p + 1) * (p + 2) // 2))
    q[:, 1:] *= 10.0
    O.set_state(q)
    O.step(13)
    for fp64_stages in (False, True) if p == 2 else (True,):
        P = Problem(cfg, mesh, tile=tile, fp64_stages=fp64_stages)
        assert bool(P.info.stage_increments) != fp64_stages
        P.set_state(q)
        P.step_serial(3)
        for _ in range(cfg.rk_nstages):
            P.stage_serial()
        P.step_serial(9)
        e = rel_err(P.get_state(), O.get_state())
        assert e <= 2e-6, (fp64_stages, e)


@pytest.mark.parametrize("p,rk", [(1, (2, 2)), (2, (3, 3))])
def test_fp32_closed_basin_mass(p, rk):
    """Both elements of an interface evaluate its flux, each with its own scaled normal, so that their mass fluxes cancel
    to the rounding of the element geometry (2e-7 of the flux in FP32). 4,000 steps of a sloshing hump in a closed basin
    over uneven bottom, jittered mesh: the mass drifts by 6e-11 of itself (1e-9 with one rounded flux per edge and two
    rounded weights). Bar: 1e-9."""
    bath = meshgen.bath_gaussians(3, ((0, 1e4), (0, 1e4)))
    mesh = meshgen.quad_mesh(48, 48, corners=((0, 0), (1e4, 0), (1e4, 1e4), (0, 1e4)), bc=(LAND,) * 4, jitter=0.2, seed=5,
                             bathymetry=bath)
    cfg = configs.ensemble_member(8, 1, precision="fp32")[1]
    cfg.p, cfg.rk_nstages, cfg.rk_order, cfg.wetting_drying = p, rk[0], rk[1], False
    P = Problem(cfg, mesh)
    m0, q0 = P.mass(), P.get_state()
    P.step_serial(4000)
    assert np.abs(P.get_state()[:, 1:]).max() > 0.1 and np.abs(P.get_state() - q0).max() > 0.1  # it sloshes
    assert abs(P.mass() / m0 - 1) <= 1e-9, P.mass() / m0 - 1
