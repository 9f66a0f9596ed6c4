"""autotune.choices() names the variant that an index of the library stands for."""
import ctypes
import re
from pathlib import Path

import tnpy_gb300.autotune as autotune

SOURCE = Path(__file__).resolve().parents[1] / "tnpy_gb300" / "csrc" / "matvec_bf16x3.cu"


def _split_gemm_variants():
    """Output tiles of split_gemm's variants in the order of its switch."""
    body = SOURCE.read_text().split("int split_gemm(", 1)[1].split("\n}\n", 1)[0]
    single, pair = r"launch_gemm<(?P<s>\d+)>", r"launch_pair<(?P<p>\d+),"
    return [f"128x{m['s']}" if m["s"] else f"256x{m['p']}" for m in re.finditer(f"{single}|{pair}", body)]


def test_a_name_for_every_split_gemm_variant():
    tiles = _split_gemm_variants()
    assert len(tiles) == int(re.search(r"SPLIT_VARIANTS = (\d+)", SOURCE.read_text())[1])
    assert [name.split("/")[0] for name in autotune.VARIANTS[3]] == tiles


def test_choices_gives_names(monkeypatch):
    lines = "\n".join(f"3 2048 1024 5120 8 0 -> {i} 0.1 0.2 0.3 0.4" for i in range(4)).encode() + b"\n\0"

    class Library:
        @staticmethod
        def tnx_autotune_report(buf, n):
            if buf is not None:
                ctypes.memmove(buf, lines, len(lines))
            return len(lines)

    monkeypatch.setattr(autotune, "lib", Library)
    got = autotune.choices()
    assert [c["choice"].split("/")[0] for c in got] == _split_gemm_variants()
    assert all(c["kind"] == "bf16x3_gemm_tile" and c["ms"] == [0.1, 0.2, 0.3, 0.4] for c in got)
