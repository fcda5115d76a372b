"""What a test starts ends with it (conftest.no_process_left)."""
import signal
import subprocess
import sys

left = []


def test_leaves_processes():
    for code in ("import time; time.sleep(300)",
                 "import signal, time; signal.signal(signal.SIGTERM, signal.SIG_IGN); print('on', flush=True); time.sleep(300)"):
        left.append(subprocess.Popen([sys.executable, "-c", code], stdout=subprocess.PIPE))
    assert left[1].stdout.readline() == b"on\n"
    assert all(p.poll() is None for p in left)


def test_that_have_ended():
    assert [p.poll() for p in left] == [-signal.SIGTERM, -signal.SIGKILL]


def test_run_is_as_ever():
    assert subprocess.run([sys.executable, "-c", "print(7)"], capture_output=True, text=True).stdout == "7\n"
