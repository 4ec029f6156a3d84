"""CPU check of two quotients by a tabled or kept reciprocal against IEEE division:
the level-0 half-sweeps' by the count of fluid neighbours (all 2^32 dividends were
run once with stride 1; this test takes a strided subset and the signed zeros,
subnormal and threshold values) and the ray marcher's by the sides of the box."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_tabled_quotients_match_ieee(tmp_path):
    exe = tmp_path / "quotient_check"
    env = dict(os.environ)
    env.pop("CC", None)
    subprocess.run(["gcc", "-O2", "-fopenmp", "-ffp-contract=off", "-march=x86-64-v3",
                    os.path.join(HERE, "quotient_check.c"), "-o", str(exe), "-lm"], check=True, env=env)
    r = subprocess.run([str(exe), "4093"], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
    assert " 0 bit mismatches" in r.stdout
