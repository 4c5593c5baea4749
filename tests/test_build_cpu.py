"""A failed build ends every compiler that it started before it reports the
failure and removes their output directory."""

import os
import signal
import stat
import subprocess
import time

import pytest

from ddhdg_b200 import build

# stands in for nvcc, which runs other programs: the first unit fails, the
# others would run for a minute
FAKE = """#!/bin/sh
case "$*" in
  *{failing}*) exit 3 ;;
esac
sleep 60 &
echo $! >> {pids}
wait
"""


def _running(pid):
    try:
        with open(f"/proc/{pid}/stat") as f:
            return f.read().rsplit(")", 1)[1].split()[0] != "Z"
    except OSError:
        return False


def test_a_failing_unit_leaves_no_compiler_behind(tmp_path, monkeypatch):
    fake, pids = tmp_path / "nvcc", tmp_path / "pids"
    fake.write_text(FAKE.format(failing=build.UNITS[0][0], pids=pids))
    fake.chmod(fake.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setattr(build, "nvcc", lambda: str(fake))
    monkeypatch.setattr(build, "LIB", str(tmp_path / "lib.so"))
    real = subprocess.Popen
    started = []

    def popen(*args, **kw):
        job = real(*args, **kw)
        started.append(job)
        if len(started) == len(build.UNITS):  # all of them run before the first is waited for
            end = time.time() + 30
            while time.time() < end and (not pids.exists() or
                                         len(pids.read_text().split()) < len(build.UNITS) - 1):
                time.sleep(0.01)
        return job

    monkeypatch.setattr(subprocess, "Popen", popen)
    try:
        with pytest.raises(subprocess.CalledProcessError) as e:
            build.build(force=True)
        assert e.value.returncode == 3
        assert len(started) == len(build.UNITS)
        assert all(job.poll() is not None for job in started)
        end = time.time() + 10
        while time.time() < end and any(_running(p) for p in pids.read_text().split()):
            time.sleep(0.01)
        assert not any(_running(p) for p in pids.read_text().split())
    finally:
        for job in started:
            if job.poll() is None:
                job.kill()
                job.wait()
        for p in pids.read_text().split():
            if _running(p):
                os.kill(int(p), signal.SIGKILL)
    assert not os.path.exists(build.LIB)
