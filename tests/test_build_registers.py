"""A build whose dim_head-64 score kernel does not start with the registers that it shares out anew fails, and leaves the library as it was."""
import sys

import pytest

from lookahead_keys_attention_b200 import _lib

LOG = """ptxas info    : Compiling entry function '_ZN6castle17castle_bwd_kernelI6__halfLi64EEEvNS_9BwdParamsE' for 'sm_100a'
ptxas info    : Function properties for _ZN6castle17castle_bwd_kernelI6__halfLi64EEEvNS_9BwdParamsE
    0 bytes stack frame, 0 bytes spill stores, 0 bytes spill loads
ptxas info    : Used {} registers, used 16 barriers, 1024 bytes smem
ptxas info    : Compiling entry function '_ZN6castle22castle_bwd_delta_kernelI6__halfEEvNS_9BwdParamsE' for 'sm_100a'
ptxas info    : Used 23 registers, used 0 barriers
ptxas info    : Compiling entry function '_ZN6castle17castle_bwd_kernelI13__nv_bfloat16Li64EEEvNS_9BwdParamsE' for 'sm_100a'
ptxas info    : Used {} registers, used 16 barriers
ptxas info    : Compiling entry function '_ZN6castle23castle_bwd128_kv_kernelI6__halfLb1EEEvNS_9BwdParamsE' for 'sm_100a'
ptxas info    : Used 80 registers, used 16 barriers
"""


@pytest.mark.parametrize("used,wrong", [((96, 96), 0), ((95, 96), 1), ((96, 128), 1), ((64, 64), 2)])
def test_build_with_other_registers_fails(tmp_path, used, wrong):
    assert len(_lib.wrong_registers(LOG.format(*used))) == wrong
    target, stamp = tmp_path / "lib.so", tmp_path / "lib.so.stamp"
    target.write_text("old")

    def compiler(out):
        return [sys.executable, "-c", "import pathlib, sys; pathlib.Path(sys.argv[1]).write_text('new'); print(sys.argv[2])", str(out), LOG.format(*used)]

    if wrong:
        with pytest.raises(RuntimeError, match="registers a thread instead of 96"):
            _lib._compile([(target, stamp, "digest", compiler)])
        assert target.read_text() == "old" and not stamp.exists()
    else:
        _lib._compile([(target, stamp, "digest", compiler)])
        assert target.read_text() == "new" and stamp.read_text() == "digest\n"
    assert [p.name for p in tmp_path.iterdir() if ".tmp." in p.name] == []
