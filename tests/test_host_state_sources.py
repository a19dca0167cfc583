"""Host state that outlives a call is shared by threads: a static variable inside a function of the
CUDA sources is constant (initialised once, under the language's own lock), atomic, a lock, or in a
function that takes a lock before it is used."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "lbm3d_bb_b200" / "csrc"
SAFE = re.compile(r"static\s+(const\b|constexpr\b|thread_local\b|std::atomic\b|std::mutex\b)")


def _unsafe(text):
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    for m in re.finditer(r"^[ \t]+static\s[^();]*?[=;{]", text, flags=re.M):
        if re.match(r"\s*static\s+(__device__|inline|__host__)", m.group(0)) or SAFE.match(m.group(0).strip()):
            continue
        end = text.find("\n}\n", m.start())
        if "std::lock_guard" not in text[m.start():end]:
            yield " ".join(m.group(0).split())


def test_statics_inside_functions_are_safe_for_threads():
    found = {p.name: list(_unsafe(p.read_text())) for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh")}
    assert not any(found.values()), found
