"""Thread-local storage of the library.  The block is allocated as a whole when a thread first touches any of it, so what a
caller that must not allocate (pb_conv2d_umma_noalloc) runs through may not keep state there, and the rest stays small: an error
message and a few pointers."""
import ctypes as C
import os
import struct
import threading

from paella_b200 import capi


def test_the_block_of_a_thread_is_small():
    path = os.path.join(os.path.dirname(capi.__file__), "libpaella_b200.so")
    with open(path, "rb") as f:
        head = f.read(64)
        assert head[:4] == b"\x7fELF" and head[4] == 2
        phoff, phentsize, phnum = struct.unpack_from("<Q", head, 32)[0], *struct.unpack_from("<HH", head, 54)
        sizes = []
        for i in range(phnum):
            f.seek(phoff + i * phentsize)
            kind, _, _, _, _, _, memsz, _ = struct.unpack("<IIQQQQQQ", f.read(56))
            if kind == 7:             # PT_TLS
                sizes.append(memsz)
    assert sum(sizes) <= 1024, sizes


def test_tilings_asked_for_by_many_threads_agree():
    """The shapes hit the same slots of the kept tilings from eight threads at once."""
    L = capi.load()

    def infos():
        out = []
        for i in range(400):
            p = capi.OpParams()
            p.dtype, p.C, p.Cs, p.K, p.Ks = 1, 64 + 8 * (i % 7), 64 + 8 * (i % 7), 16 + 8 * (i % 61), 16 + 8 * (i % 61)
            p.H = p.W = p.P = p.Q = 7 + i % 13
            p.R, p.S, p.stride_h, p.stride_w, p.pad_h, p.pad_w, p.groups, p.batch = 3, 3, 1, 1, 1, 1, 1, 1 + i % 3
            li = capi.LaunchInfo()
            assert L.pb_op_info(capi.STAGE_CONV_UMMA, C.byref(p), C.byref(li)) == 0
            out.append(bytes(li))
        return out

    want, got = infos(), [None] * 8

    def work(k):
        got[k] = infos()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(g == want for g in got)
