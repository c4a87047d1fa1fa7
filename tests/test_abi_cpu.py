"""CPU-side checks of the boundary: the library loads without a GPU, exports every symbol the
header declares, and refuses to open a device that is not there (no CPU fallback)."""
import ctypes as C
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    from vectorstorekit_b200 import build, _lib
    build.build_library()
    return _lib.load()


def _declared():
    text = open(os.path.join(ROOT, "include", "vsk_cuda.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(vsk_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported_and_bound(lib):
    from vectorstorekit_b200 import _lib
    names = _declared()
    assert len(names) >= 15
    for n in names:
        assert hasattr(lib, n), f"{n} declared in vsk_cuda.h but not exported"
    assert set(names) == set(_lib.SIGNATURES), set(names) ^ set(_lib.SIGNATURES)


def test_header_compiles_as_c():
    import subprocess, tempfile
    with tempfile.TemporaryDirectory() as t:
        src = os.path.join(t, "t.c")
        open(src, "w").write('#include "vsk_cuda.h"\nint main(void){return VSK_OK;}\n')
        subprocess.run(["gcc", "-std=c99", "-Wall", "-Werror", "-I", os.path.join(ROOT, "include"), "-c", src,
                        "-o", os.path.join(t, "t.o")], check=True)


def test_status_strings(lib):
    assert lib.vsk_status_string(0) == b"ok"
    assert lib.vsk_status_string(9) == b"empty input"


def test_no_cpu_fallback(lib):
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    h = C.c_void_p()
    assert lib.vsk_open(0, C.byref(h)) == 1  # VSK_ERR_DEVICE_NOT_AVAILABLE
    import vectorstorekit_b200 as vsk
    with pytest.raises(vsk.DeviceNotAvailable):
        vsk.CUDAAcceleratorStrategy().initialize()


def test_product_never_reaches_the_cpu_checkers():
    """Nothing under the package may import, load or execute the checkers under oracle/: every line of the
    package's sources that mentions the word at all fails the test unless it is in the short list of known
    comments (where the word names the numeric type, not the folder)."""
    pkg = os.path.join(ROOT, "vectorstorekit_b200")
    hits = []
    for dirpath, dirs, files in os.walk(pkg):
        dirs[:] = [d for d in dirs if d not in ("_build", "__pycache__")]
        for f in files:
            if not f.endswith((".py", ".cu", ".cuh", ".hpp", ".h", ".cpp", ".c")):
                continue
            for no, line in enumerate(open(os.path.join(dirpath, f), errors="replace"), 1):
                low = line.lower()
                if "oracle" in low or "cpu_ref" in low or "vskref" in low or "metalref" in low:
                    hits.append(f"{os.path.relpath(os.path.join(dirpath, f), ROOT)}:{no}: {line.strip()}")
    # a comment may say that a kernel is bit-identical to the CPU checker; code may not name it
    allowed = [h for h in hits if re.search(r"^\S+:\d+: (//|#|\*|/\*)", h) and
               not re.search(r"import|cdll|dlopen|subprocess|popen|system\(|exec", h.lower())]
    assert hits == allowed, "\n".join(h for h in hits if h not in allowed)
    # and no dynamic loading of anything outside the package's own library
    for dirpath, dirs, files in os.walk(pkg):
        dirs[:] = [d for d in dirs if d not in ("_build", "__pycache__")]
        for f in files:
            if f.endswith(".py"):
                text = open(os.path.join(dirpath, f)).read()
                for m in re.finditer(r"CDLL\(([^)]*)\)", text):
                    assert m.group(1).strip() == "LIB_PATH", f"{f}: loads {m.group(1)}"
                assert "importlib" not in text and "__import__" not in text, f


def test_sharded_slice_covers_every_query_once(lib):
    import numpy as np
    from vectorstorekit_b200.engine import sharded_slice
    for nq in (1, 7, 64, 1000, 10_000):
        for g in (1, 2, 3, 8):
            seen = np.zeros(nq, np.int32)
            for r in range(g):
                f, c = C.c_int64(), C.c_int64()
                lib.vsk_sharded_slice(nq, g, r, C.byref(f), C.byref(c))
                assert (f.value, c.value) == sharded_slice(nq, g, r)
                seen[f.value:f.value + c.value] += 1
            assert np.all(seen == 1)


def test_search_schedule_always_advances(lib):
    """Every chunk of the search schedule has at least one row, for every list size a search may keep and any number
    of rows seen: a schedule that returned 0 would never finish."""
    for keep in (1, 2, 10, 100, 112, 1000, 2047, 2048):
        for level in (0, 1, 2):
            for seen in (0, 1, 255, 1024, 4096, 10 ** 6, 2 ** 31 - 1):
                assert lib.vsk_schedule_chunk(seen, keep, level) >= 1, (seen, keep, level)
    assert lib.vsk_schedule_chunk(1024, 2049, 0) == -1 and lib.vsk_schedule_chunk(1024, 0, 0) == -1


def test_nccl_entry_points_fail_cleanly_without_a_device(lib):
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    assert lib.vsk_comm_init(None, 2, 0, None) == 7      # VSK_ERR_INVALID_INPUT: no context
    n, r = C.c_int32(5), C.c_int32(5)
    assert lib.vsk_comm_info(None, C.byref(n), C.byref(r)) == 7


def test_unsupported_metric_raises():
    import vectorstorekit_b200 as vsk
    from vectorstorekit_b200.engine import _metric_id
    with pytest.raises(vsk.UnsupportedOperation):
        _metric_id(vsk.DistanceMetric.hamming)
    assert _metric_id("cosine") == 1


def _build_host_mirror(tmp):
    import subprocess
    exe = os.path.join(tmp, "host_mirror_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", os.path.join(ROOT, "tests", "host_mirror_test.cpp"), "-o", exe,
                    "-L", os.path.join(ROOT, "vectorstorekit_b200"), "-lvsk_cuda",
                    "-Wl,-rpath," + os.path.join(ROOT, "vectorstorekit_b200")], check=True)
    return exe


def test_cpp_host_mirror_compiles_and_refuses_without_gpu(lib, tmp_path):
    import subprocess
    import torch
    exe = _build_host_mirror(str(tmp_path))
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out
    assert out.stdout.strip() == ("ok" if torch.cuda.is_available() else "no-device")


def test_launch_attributes_are_not_kept_per_process():
    """A kernel's attributes belong to one device: a flag that lives as long as the process would leave a second device opened
    in it without them (no second device is at hand to launch on)."""
    import glob
    for path in glob.glob(os.path.join(ROOT, "vectorstorekit_b200", "csrc", "*.cu*")):
        for line in open(path):
            assert not re.search(r"static bool \w*(attr|carveout)", line), f"{os.path.basename(path)}: {line.strip()}"
