"""Failure paths on the GPU: every failure is reported as a status, the GPU is never
trapped, and the context stays usable.  Failures are provoked from the host
(tolerance 0, a restart cap of 1, NaN in the initial data, misuse of the API)."""
from __future__ import annotations

import numpy as np
import pytest

import imex_b200 as ix
from imex_b200.problems import vortex

pytestmark = pytest.mark.gpu


def test_gmres_restart_cap_is_reported_and_context_survives():
    prob = vortex(32)
    sv = ix.Solver.for_problem(prob, 2, dict(recon="VanLeer", magfield="StaggerCT", GMREStol=0.0,
                                             gmres_max_restarts=1, gmres_restart=5))
    with pytest.raises(ix.ImexError) as err:
        sv.step()
    assert err.value.status in (ix.ImexError(4, "").status, 5)
    # the context is still usable after the error
    d = sv.divergence()
    assert np.isfinite(d["face_l2"])
    sv.close()


def test_nonfinite_input_is_reported():
    prob = vortex(32)
    prob.prim[0, 5, 7] = np.nan
    sv = ix.Solver.for_problem(prob, 2, dict(recon="VanLeer", magfield="StaggerCT"))
    with pytest.raises(ix.ImexError) as err:
        sv.step()
    assert err.value.status == 6
    sv.close()


def test_ct_variant_must_match_magfield():
    prob = vortex(16)
    sv = ix.Solver.for_problem(prob, 2, dict(recon="VanLeer", magfield="PotentialA"))
    with pytest.raises(ix.ImexError) as err:
        sv.Staggered_CT_Consistent(0.01, 0)
    assert err.value.status == 1
    sv.close()


def test_bad_buffer_and_stage_indices():
    sv = ix.Solver.for_problem(vortex(16), 2, dict(recon="VanLeer", magfield="StaggerCT"))
    with pytest.raises(ix.ImexError):
        sv.get_buffer("Hs", index=2)
    with pytest.raises(ix.ImexError):
        sv.stage(5)
    sv.close()


def test_barrier_wait_times_out_and_reports_sync_error():
    """A device-wide barrier that waits for CTAs that never launch must give up after its
    bound (0.2 s here), return IMEX_ERR_SYNC, and leave the context usable."""
    sv = ix.Solver.for_problem(vortex(64), 2, dict(recon="VanLeer", magfield="StaggerCT"))
    us = sv.selftest_barrier(200)           # healthy barriers complete
    assert 0.0 < us < 1000.0
    with pytest.raises(ix.ImexError) as err:
        sv.selftest_barrier(5, phantom_blocks=1, timeout_s=0.2)
    assert err.value.status == 8
    dt = sv.step()                          # the solver still works afterwards
    assert dt > 0 and sv.divergence()["face_l2"] < 1e-12
    sv.close()


def test_strong_field_redlich_kwong_is_reported_like_the_reference_fails():
    """At beta = 1e-4 the reference scheme itself goes non-finite within two steps on the
    Redlich-Kwong random field; the GPU path must report that as a status, not carry on."""
    from imex_b200.problems import random_field
    prob = random_field(32, beta=1e-4)
    settings = dict(recon="Minmod", magfield="StaggerCT", eos_type="REDLICH_KWONG", m_alfa=0.4275, m_b=0.0866)
    sv = ix.Solver.for_problem(prob, 2, settings)
    with pytest.raises(ix.ImexError) as err:
        for _ in range(2):
            sv.step()
    assert err.value.status in (5, 6, 7, 9)  # Newton cap, non-finite, positivity or EOS iteration cap
    sv.scalars()  # the context still answers after the error
    sv.close()


@pytest.mark.parametrize("iterations", [1, 2, 7])
def test_pass_end_is_given_up_by_every_block_or_by_none(iterations):
    """The pass end of the row-marching solves, whose last arrival is the first block's, 0.2 s after the
    others' bound of 0.02 s ran out: that block finds the arrivals complete, and yet the launch counts as
    given up in every block.  With a bound that is long enough, or without delay, in none."""
    sv = ix.Solver.for_problem(vortex(64), 2, dict(recon="VanLeer", magfield="StaggerCT"))
    r = sv.selftest_pass_end(iterations, late_s=0.2, timeout_s=2.0)
    assert r["status"] == 0 and r["gave_up"] == 0 and r["blocks"] > 1
    r = sv.selftest_pass_end(iterations, late_s=0.2, timeout_s=0.02)
    assert r["status"] == 8 and r["gave_up"] == r["blocks"], r
    r = sv.selftest_pass_end(iterations, phantom_blocks=1, timeout_s=0.02)
    assert r["status"] == 8 and r["gave_up"] == r["blocks"], r
    r = sv.selftest_pass_end(200)
    assert r["status"] == 0 and r["gave_up"] == 0 and 0.0 < r["us"] < 1000.0, r
    assert sv.step() > 0 and sv.divergence()["face_l2"] < 1e-12
    sv.close()


VORTEX = dict(recon="VanLeer", magfield="StaggerCT", GMREStol=1e-12)
AT_ONCE = 1e-9  # a bound of two clock cycles: a block gives up if the others are not there while it looks again


def _give_up(sv):
    """Stages until one of their waits has run out (each has some fifty); its status is not read yet."""
    sv.set_barrier_timeout(AT_ONCE)
    sv.begin_step()
    for _ in range(50):
        sv.stage(0)
        if sv.stats()["status"] == 8:
            sv.set_barrier_timeout(2.0)
            return
    pytest.fail("no wait ran out")


def _fresh_run(steps):
    sv = ix.Solver.for_problem(vortex(64), 2, VORTEX)
    for _ in range(steps):
        sv.step()
    c = sv.cons()
    sv.close()
    return c


def test_solves_wait_again_after_a_reset_of_the_statistics():
    """A stage whose solves gave up, and whose status is cleared by imex_reset_stats before a call
    reads it: the next steps are a fresh context's, bit for bit."""
    sv = ix.Solver.for_problem(vortex(64), 2, VORTEX)
    _give_up(sv)
    sv.reset_stats()
    sv.load(vortex(64))
    sv.step()
    sv.step()
    np.testing.assert_array_equal(sv.cons(), _fresh_run(2))
    sv.close()


@pytest.mark.parametrize("streams,graph", [(0, True), (0, False), (2, False)])
def test_ensemble_waits_again_after_a_wait_ran_out(streams, graph):
    """The step of an ensemble whose waits run out reports IMEX_ERR_SYNC; with a bound as usual the
    members' next steps are a fresh ensemble's, bit for bit."""
    probs = [vortex(64), vortex(48, 96), vortex(80)]
    batch = ix.Batch(probs, 2, VORTEX, streams=streams, graph=graph)
    for sv in batch.members:
        sv.set_barrier_timeout(AT_ONCE)
    for _ in range(2):
        with pytest.raises(ix.ImexError) as err:
            batch.step(50)
        assert err.value.status == 8
    for sv in batch.members:
        sv.set_barrier_timeout(2.0)
    assert batch.lib.imex_batch_configure(batch.b, streams, 1 if graph else 0) == 0
    fresh = ix.Batch(probs, 2, VORTEX, streams=streams, graph=graph)
    for sv, p in zip(batch.members, probs):
        sv.load(p)
    batch.step(2)
    fresh.step(2)
    for a, b in zip(batch.members, fresh.members):
        np.testing.assert_array_equal(a.cons(), b.cons())
    batch.close()
    fresh.close()


def test_solves_wait_again_when_an_eos_flag_hides_the_timed_out_wait():
    """A status of IMEX_ERR_EOS stands for a timed-out wait too.  The flag is raised by another context's
    upload (the flags belong to the device): with attraction 1e-300 and pressure 0 the inversion of the
    Redlich-Kwong EOS starts at T = 1e-300 and triples it each iteration towards 1e-200, past its cap of 200."""
    rk = ix.Solver.for_problem(vortex(64), 2, dict(VORTEX, eos_type="REDLICH_KWONG", m_alfa=1e-300, m_b=0.1))
    empty = vortex(64)
    empty.prim[0], empty.prim[1:8] = 1.0, 0.0
    sv = ix.Solver.for_problem(vortex(64), 2, VORTEX)
    _give_up(sv)
    rk.load(empty)
    rk.scalars()  # the upload is done
    with pytest.raises(ix.ImexError) as err:
        sv.end_step()
    assert err.value.status == 9
    rk.close()
    sv.load(vortex(64))
    sv.step()
    sv.step()
    np.testing.assert_array_equal(sv.cons(), _fresh_run(2))
    sv.close()
