"""BselMarg.eval packs a sample's record as one struct: the same bytes as the
C structure's fields."""
import ctypes as C

from y3_cluster_cpp_b200 import _capi as A
from y3_cluster_cpp_b200.engine import BselMarg


def test_record_matches_the_c_structure():
    head, size = C.sizeof(A.Cosmo), C.sizeof(A.BselSample)
    assert BselMarg._RECORD.size + head == size
    v = [3 * i + 1 for i in range(22)] + [0.5 * i for i in range(6)]
    s = A.BselSample()
    buf = (C.c_ubyte * size).from_buffer(s)
    BselMarg._RECORD.pack_into(buf, head, *v)

    def address(p):
        return C.cast(p, C.c_void_p).value

    t = s.t
    got = [t.n_hm, address(t.hmf_m_h), t.n_hz, address(t.hmf_z), address(t.dndlnmh), t.n_dist,
           address(t.dist_z), address(t.dist_da), t.n_sci, address(t.sci_z), address(t.sci_val),
           address(s.dist_dc), s.n_hl, s.n_hz, address(s.halo_lnM), address(s.halo_z),
           address(s.bias), s.n_xr, s.n_xz, address(s.xi_r), address(s.xi_z), address(s.xi_nl)]
    assert got == v[:22]
    assert list(s.hod) == v[-6:]
