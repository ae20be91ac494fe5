"""The pinned words of a call whose wait failed are not handed out again."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_words_given_up(tmp_path):
    exe = tmp_path / "starts_abandon_test"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-O1", "-pthread", "-I",
                    str(ROOT / "gpumultisplit_gb300" / "csrc"), str(ROOT / "tests" / "cpp" / "starts_abandon_test.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
