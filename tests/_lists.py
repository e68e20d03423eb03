"""nbl_list_info of a plan or a batch."""
import ctypes


class ListInfo(ctypes.Structure):
    _fields_ = [("workspace_bytes", ctypes.c_int64), ("list_bytes", ctypes.c_int64)] + [
        (n, ctypes.c_int) for n in ("lists", "by_atoms", "two_words", "short_of_room")]


def list_info(plan=None, batch=None):
    from matscipy_neighbours import _matscipy_neighbours as ext
    info = ListInfo()
    fn = ext.lib.nbl_debug_lists
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    ext.check(fn(plan, batch, ctypes.byref(info)))
    return info
