"""The registry of parts in a program that brings its own."""

import subprocess
import sys

import pytest

PROGRAMS = {
    "derives from a part before anything is built": """
from atomserve_b200.parts.norms import RMSNorm
from atomserve_b200.parts import PartSpec, build_part, register_part
class Own(RMSNorm):
    pass
register_part("norm", "own", Own)
assert type(build_part("norm", PartSpec("own", dict(eps=1e-6)), 8)) is Own
assert type(build_part("embedding", PartSpec("token_embedding", dict(vocab_size=4)), 8)).__name__ == "TokenEmbedding"
""",
    "takes a kind for itself before anything is built": """
from atomserve_b200.parts import Norm, PartSpec, build_part, register_part
class Own(Norm):
    def __init__(self, hidden_size, prefix):
        pass
register_part("norm", "rms_norm", Own)
assert type(build_part("norm", PartSpec("rms_norm"), 8)) is Own
assert type(build_part("embedding", PartSpec("token_embedding", dict(vocab_size=4)), 8)).__name__ == "TokenEmbedding"
assert type(build_part("norm", PartSpec("rms_norm"), 8)) is Own
""",
}


@pytest.mark.parametrize("program", PROGRAMS.values(), ids=PROGRAMS)
def test_builtin_parts_are_there(program):
    subprocess.run([sys.executable, "-c", program], check=True, timeout=300)
