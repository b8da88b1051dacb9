"""The build compiles a file again when the command that compiles it has
changed, not only when its text has (a stand-in for the compiler, no GPU)."""
import os
import stat

from nexusmd_gb300 import build as b


def _fake_nvcc(path, log, version="13.0"):
    path.write_text("#!/bin/sh\nif [ \"$1\" = --version ]; then echo release %s; exit 0; fi\necho \"$@\" >> %s\n"
                    "while [ $# -gt 0 ]; do if [ \"$1\" = -o ]; then echo object > \"$2\"; fi; shift; done\n"
                    % (version, log))
    path.chmod(path.stat().st_mode | stat.S_IXUSR)


def test_changed_flags_compile_again(tmp_path, monkeypatch):
    log = tmp_path / "log"
    log.write_text("")
    _fake_nvcc(tmp_path / "nvcc", log)
    monkeypatch.setenv("NVCC", str(tmp_path / "nvcc"))
    monkeypatch.setattr(b, "BUILD", str(tmp_path / "_build"))
    monkeypatch.setattr(b, "LIB", str(tmp_path / "lib.so"))
    monkeypatch.setattr(b, "PROBE_LIB", str(tmp_path / "probe.so"))
    os.makedirs(b.BUILD)

    def compiled():
        log.write_text("")
        b.build()
        lines = log.read_text().splitlines()
        return sum(" -c " in " " + line for line in lines), sum(b.PROBE_SRC in line for line in lines)

    files = len(b.CUDA_SOURCES) + len(b.HOST_SOURCES)
    assert compiled() == (files, 1)
    assert compiled() == (0, 0)
    monkeypatch.setattr(b, "ARCH", b.ARCH + ["-DNXM_OTHER"])
    assert compiled() == (files, 1)
    assert compiled() == (0, 0)
    _fake_nvcc(tmp_path / "nvcc", log, "13.1")
    assert compiled() == (files, 1)
