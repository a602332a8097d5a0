"""CPU: what the gates' gradients refuse before anything is launched."""
import ctypes



def test_query_key_gradient_wants_pairs():
    from fairseq_apollo_b200 import _lib
    lib = _lib.lib()
    at = lambda v: ctypes.c_void_p(v)
    good = dict(z=4096, ld_z=64, rot=None, dq=8192, ld_dq=64, dk=16384, ld_dk=64, dz=32768, ld_dz=64)

    def call(dtype, **kw):
        a = dict(good, **kw)
        return lib.mega_gate_qk_bwd(at(a["z"]), a["ld_z"], at(4096), a["rot"] and at(a["rot"]), 8, 8, 0, at(a["dq"]), a["ld_dq"],
                                    at(a["dk"]), a["ld_dk"], at(a["dz"]), a["ld_dz"], at(4096), at(4096), None, dtype, 8, 64, 1e-5, None)

    for name in ("ld_z", "ld_dq", "ld_dk", "ld_dz"):
        assert call(1, **{name: 65}) == 5 and call(0, **{name: 67}) == 5
        assert call(1, **{name: 62}) == 4
    for name in ("z", "dq", "dk", "dz"):
        assert call(1, **{name: good[name] + 2}) == 5      # bf16: an element on, half a pair
        assert call(0, **{name: good[name] + 4}) == 5
    assert call(1, rot=4100) == 5
