"""bench.py's own chi-squared (the parity block of the bench line) against the
oracle's batched chi-squared, on seeded synthetic batch means (no GPU)."""

from __future__ import annotations

import numpy as np

import bench
from oracle import stats


def test_bench_chi2_matches_the_oracle():
    rng = np.random.default_rng(11)
    a = rng.uniform(1.0, 2.0, 500)
    b = a + rng.normal(0.0, 0.02, 500)
    sa, sb = rng.uniform(0.01, 0.03, 500), rng.uniform(0.01, 0.03, 500)
    chi2, mean, p = bench.batched_chi2(a, sa, 10, b, sb, 20)
    r = stats.chi2_batched(a, sa, 10, b, sb, 20)
    assert np.isclose(chi2, r["chi2"]) and np.isclose(mean, r["null_mean"])
    assert np.isclose(p, r["p_value"], rtol=1e-9, atol=1e-12)


def test_the_printed_line_is_short_and_keeps_what_is_asked_of_it():
    errors = {k: dict(sigma_eq=0.019590735169996577, bias_mean=-0.00065361722, bias_integral=1.5) for k in ("0.5", "0.1", "0.01")}
    rung = dict(histories_per_beamlet=30870, fraction_of_plain=0.125, denoised=errors, plain_same_histories=errors,
                history_gain=1.2912290098248949)
    region = dict(history_scale=0.5, s_per_dij_at_2pct=0.023551328659057617, speedup_vs_plain=8.803050133674429,
                  denoised=errors, plain_same_histories=errors)
    record = dict(case="ct_beamlets column 0 (40000 histories, >= 0.1 of max)", chi2_per_dof=1.1255566081561454,
                  null_mean_per_dof=1.1819831974492563, p=0.25, n_voxels=345, passed=True)
    full = dict(metric=bench.METRIC, value=1045333799.5122386, unit="histories/s", n_gpus=1, steps=3, warmup=3,
                ms_per_step=22.185344060262043, denoiser=dict(ladder=[rung] * 24, regions={"0.5": region, "0.1": region}),
                plan=dict(plain=dict(s=1.08), denoiser=dict(ladder=[rung] * 5)),
                parity=dict(reference="fixtures", records=[record] * 8),
                e2e=dict(value=828000000.1234567, h2d_bytes_per_step=34698272, d2h_bytes_per_step=193177648),
                clocks=dict(sm_mhz=1965.0, reasons=[]), cpu_baseline=None)
    line = bench.short_line(full)
    text = bench.json.dumps(line)
    assert len(text) < 2048 and bench.json.loads(text) == line
    assert line["value"] == full["value"] and line["ms_per_step"] == full["ms_per_step"]
    assert line["e2e"] == dict(value=828000000.0, h2d_bytes_per_step=34698272, d2h_bytes_per_step=193177648)
    assert line["parity"] == dict(reference="fixtures", min_p=0.25)
    assert line["plan"]["denoiser"]["ladder"] == [[0.125, 0.01959074]] * 5
    assert line["denoiser"]["regions"]["0.1"] == dict(history_scale=0.5, s_per_dij_at_2pct=0.02355133,
                                                      speedup_vs_plain=8.80305, sigma_eq=0.01959074, bias_integral=1.5)
    assert "ladder" in full["denoiser"] and "records" in full["parity"]  # the full record keeps them
    empty = dict(full, denoiser=None, plan=None, parity=None)
    assert bench.short_line(empty)["denoiser"] is None
