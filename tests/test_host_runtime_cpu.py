"""The library's host code where the CUDA runtime fails or is used from several
threads and devices, without a GPU: host_runtime_driver.cu links the library's
own objects against a runtime that keeps device memory on the host and makes
chosen calls fail."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "cpu-vh_b200")
OBJ = [f"_build/{n}.o" for n in ("vh_kt", "vh_fo", "vh_capi", "vh_noalloc", "vh_batch", "vh_mixed", "vh_ic", "vh_host",
                                 "vh_powf_table", "vh_server")]


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    missing = [o for o in OBJ if not os.path.exists(os.path.join(PKG, o))]
    if missing:
        subprocess.run(["make", "-s", "-j4", "-C", PKG] + missing, check=True)
    exe = str(tmp_path_factory.mktemp("driver") / "host_runtime_driver")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-O1", "-std=c++17", "-cudart", "none",
                    "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(PKG, "..", "include"),
                    "-I", os.path.join(PKG, "host"), "-I", os.path.join(PKG, "csrc"), "-Xcompiler", "-pthread",
                    os.path.join(HERE, "host_runtime_driver.cu")] + [os.path.join(PKG, o) for o in OBJ] + ["-o", exe], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["error_cleared", "regrow_failure", "setup_rollback", "chain_failure", "opt_in_devices", "opt_in_threads", "opt_in_batches"])
def test_scenario(driver, scenario):
    env = {k: v for k, v in os.environ.items() if not k.startswith("VH_")}
    r = subprocess.run([driver, scenario], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
