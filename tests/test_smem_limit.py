"""Dynamic shared-memory limits of kernels that several host threads launch
with different amounts: the policy on the CPU (smem_limit.h built with g++ and
a fake setter), and two threads whose products launch the same replayed kernel
with different shared memory on the GPU."""
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

import sp3mm4amg_b200 as S

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sp3mm4amg_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not found")
def test_limits_never_shrink(tmp_path):
    exe = str(tmp_path / "smem_limit_test")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", CSRC,
                    os.path.join(HERE, "smem_limit_test.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.startswith("ok"), out.stdout


def _rows(rng, M, N, n):
    cols = np.sort(np.argsort(rng.random((64, N)), axis=1)[:, :n], axis=1)
    return S.CSR(np.arange(M + 1, dtype=np.int64) * n, cols[np.arange(M) % 64].ravel(),
                 rng.uniform(-1, 1, M * n), (M, N))


@pytest.mark.gpu
def test_two_threads_launch_different_sizes():
    # 22 and 30 left steps of 16 products: the replayed kernel's CTAs take
    # different amounts of shared memory, both above 48 KB.
    rng = np.random.default_rng(1)
    A, P = _rows(rng, 200, 300, 16), _rows(rng, 300, 200, 3)
    Rs = [_rows(rng, 16384, 200, n) for n in (22, 30)]
    failed = []

    def work(R):
        try:
            with S.Context() as ctx:
                d = [ctx.upload(m) for m in (R, A, P)]
                for _ in range(400):
                    ctx.rap(*d, S.DIRECT, S.UB).free()
        except S.Sp3mmError as e:
            failed.append(str(e))

    threads = [threading.Thread(target=work, args=(R,)) for R in Rs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
