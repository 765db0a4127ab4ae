"""The build of _plain.so: CUDA's headers, and what makes it out of date."""
import shutil

from flash_attn_with_score_b200 import build


def test_plain_is_built_with_an_nvcc_of_any_name(tmp_path, monkeypatch):
    """CUDA's headers are where nvcc says, not beside the program that was called: a wrapper elsewhere builds as well."""
    wrapper = tmp_path / "tools" / "nvcc"
    wrapper.parent.mkdir()
    wrapper.write_text(f'#!/bin/sh\nexec "{shutil.which(build._nvcc())}" "$@"\n')
    wrapper.chmod(0o755)
    source = tmp_path / "small.cpp"
    source.write_text("#include <cuda_runtime_api.h>\nextern \"C\" int version() { return CUDART_VERSION; }\n")
    monkeypatch.setenv("NVCC", str(wrapper))
    for name, path in (("PLAIN_SOURCE", source), ("PLAIN", tmp_path / "_plain.so"), ("OBJDIR", tmp_path)):
        monkeypatch.setattr(build, name, str(path))
    build._build_plain(False)
    assert (tmp_path / "_plain.so").exists() and (tmp_path / "plain.digest").read_text() == build._plain_digest()


def test_another_compiler_call_makes_plain_out_of_date(monkeypatch):
    before = build._plain_digest()
    monkeypatch.setenv("NVCC", shutil.which("true"))
    assert build._plain_digest() != before
