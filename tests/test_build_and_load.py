"""What a build needs of the machine and what the package needs of a build: the library stands alone, the CPython extension is
one way to it among two."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT


def child(code, **env):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, **env), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout
    return r.stdout


def test_build_without_the_interpreters_headers(built, tmp_path, monkeypatch, capfd):
    """No Python.h: the extension is left out with one line, and an outdated one goes."""
    import sysconfig

    from graphtok_b200 import build
    paths = dict(sysconfig.get_paths(), include=str(tmp_path), platinclude=str(tmp_path))
    monkeypatch.setattr(sysconfig, "get_paths", lambda *a, **k: paths)
    monkeypatch.setattr(build, "HOST", str(tmp_path / "_host.so"))
    (tmp_path / "_host.so").write_bytes(b"outdated")
    os.utime(str(tmp_path / "_host.so"), (1, 1))
    assert build.build_host() is None
    out = capfd.readouterr().out
    assert out.count("\n") == 1 and "Python.h" in out
    assert not os.path.exists(build.HOST)


def test_build_with_headers_that_do_not_compile(built, tmp_path, monkeypatch, capfd):
    from graphtok_b200 import build
    (tmp_path / "Python.h").write_text("#error not this one\n")
    monkeypatch.setattr(build, "HOST", str(tmp_path / "_host.so"))
    monkeypatch.setattr(build, "_host_includes", lambda: [str(tmp_path)])
    assert build.build_host() is None
    out = capfd.readouterr().out
    assert out.count("\n") == 1 and "not this one" in out


def test_package_without_the_extension(built):
    out = child("import sys; sys.modules['graphtok_b200._host'] = None\n"
                "import graphtok_b200 as g, numpy as np\n"
                "print(g.plan_documents(np.array([0, 10, 20, 30, 40]), 2).tolist(), type(g.load_lib().host).__name__)\n"
                "from graphtok_b200.gpu_bpe_tokenizer import Tokenizer, Dispatcher\n")
    assert out.strip() == "[0, 2, 4] CtypesHost"


def test_one_copy_of_the_library_whatever_the_library_path(built, tmp_path):
    """Another libgtok.so first on the library path: neither loaded nor asked for its calls."""
    from graphtok_b200 import build, load_lib
    (tmp_path / "other.cc").write_text('extern "C" int gtok_create() { return 7; }\n')
    subprocess.run(["g++", "-fPIC", "-shared", "-o", str(tmp_path / "libgtok.so"), str(tmp_path / "other.cc")], check=True)
    out = child("import graphtok_b200 as g\n"
                "kind = type(g.load_lib().host).__name__\n"
                "paths = {line.split()[-1] for line in open('/proc/self/maps') if 'libgtok.so' in line}\n"
                "print(kind, *paths)\n", LD_LIBRARY_PATH="%s:%s" % (tmp_path, os.environ.get("LD_LIBRARY_PATH", "")))
    assert out.split() == [type(load_lib().host).__name__, build.LIB]


def test_no_figure_for_the_reference_without_its_encoder():
    """The reference arm of the benchmark times the reference's own encoder or nothing."""
    import json

    import oracle_lib
    if os.path.exists(oracle_lib.REF_SO):
        pytest.skip("the reference's encoder is built here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"], cwd=ROOT, stdout=subprocess.PIPE, text=True)
    line = json.loads(r.stdout)
    assert r.returncode == 0 and line["impl"] == "reference" and line["unavailable"] and "value" not in line
