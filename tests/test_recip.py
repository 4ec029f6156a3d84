"""CPU check of the coarse levels' division by a correctly rounded reciprocal
(div_recip in smokesim_b200/csrc/k_coarse.cu): the same bits as IEEE division
for the counts 1..6 and for sums of fluid fractions."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_division_by_reciprocal_matches_ieee(tmp_path):
    exe = tmp_path / "recip_check"
    env = dict(os.environ)
    env.pop("CC", None)
    subprocess.run(["gcc", "-O2", "-fopenmp", "-ffp-contract=off", "-march=x86-64-v3",
                    os.path.join(HERE, "recip_check.c"), "-o", str(exe), "-lm"], check=True, env=env)
    r = subprocess.run([str(exe), "512"], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
    assert " 0 bit mismatches" in r.stdout
