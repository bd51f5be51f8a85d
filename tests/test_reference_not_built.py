"""Where the reference's solver is not built, a test ends as skipped at its comparison with it, and every other failure stays
one: also what the same test asserts before."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))

BODY = '''
import oracle, pytest
oracle._LIBS["reference"] = ("/nowhere/oracle/_ref/libpsref.so", "ref_")

def reference():
    return oracle.OracleModel("reference", (1, 1, 1), [1.0], 0.3, [0] * 24)

def test_asserts_first():
    assert 1 == 2
    reference()

def test_compares():
    assert 1 == 1
    reference()

@pytest.fixture
def refs():
    assert oracle.available("reference"), "oracle/_ref (the reference's solver) is not built"

def test_fixture(refs):
    pass

def test_other_file_missing():
    open("/nowhere/at/all")
'''


def test_only_the_missing_reference_skips(tmp_path):
    (tmp_path / "test_body.py").write_text(BODY)
    (tmp_path / "conftest.py").write_text(open(os.path.join(HERE, "conftest.py")).read())
    env = dict(os.environ, PYTHONPATH=os.path.dirname(HERE))
    p = subprocess.run([sys.executable, "-m", "pytest", "-q", "-rA", "-p", "no:cacheprovider", str(tmp_path)], env=env, cwd=tmp_path, capture_output=True,
                       text=True, timeout=120)
    assert "2 failed, 2 skipped" in p.stdout, p.stdout
    for name in ("test_asserts_first", "test_other_file_missing"):
        assert f"FAILED test_body.py::{name}" in p.stdout, p.stdout
