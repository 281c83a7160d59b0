"""The first device call of a process from several host threads at once: what the call wrappers keep of
torch becomes visible in an order in which no thread can see a part of it. Another thread may run
between any two bytecodes, so the name the others look at has to be stored last."""
import dis

import ddc_b200.splines as S


def test_first_call_is_never_half_done():
    stored = [i.argval for i in dis.get_instructions(S._torch_ops) if i.opname == "STORE_GLOBAL"]
    assert sorted(stored) == ["_Tensor", "_f64", "_torch"]
    assert stored[-1] == "_torch"
