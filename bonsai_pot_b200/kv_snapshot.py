"""`KvSnapshot`: the host-resident "BONSAIKV" v1 blob of the cache rows
[0, pos) (reference: src/kv_snapshot.rs). The bytes are produced and consumed
by the C ABI (`bp_snapshot_capture` / `bp_snapshot_apply`); this class is the
reference's value type around them."""
from __future__ import annotations

import ctypes as C
import mmap
import struct

from . import _lib
from .errors import ConfigError

MAGIC = b"BONSAIKV"
VERSION = 1
HEADER_BYTES = 32


def payload_bytes(n_layer, kv_dim, pos):
    """src/kv_snapshot.rs:150-154."""
    return int(_lib.load().bp_snapshot_payload_bytes(n_layer, kv_dim, pos))


def payload_offset(n_layer, kv_dim, pos, kind, il, sect):
    """src/kv_snapshot.rs:158-169; kind 0 = K, 1 = V; sect 0 = d, 1 = qs."""
    return int(_lib.load().bp_snapshot_payload_offset(n_layer, kv_dim, pos, kind, il, sect))


# Prototypes of this module's own: the attributes of `ctypes.pythonapi` are shared with everything else in the process.
_bytes_new = C.PYFUNCTYPE(C.py_object, C.c_char_p, C.c_ssize_t)(("PyBytes_FromStringAndSize", C.pythonapi))
_bytes_address = C.PYFUNCTYPE(C.c_void_p, C.py_object)(("PyBytes_AsString", C.pythonapi))
_madvise = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_size_t, C.c_int)(("madvise", C.CDLL(None)))
_HUGE_PAGE = 2 << 20


def new_blob(size):
    """An uninitialised `bytes` object and the address of its bytes, for a call that fills it: a capture then
    touches every page of the blob once (zeroing a buffer and copying it out took longer than the transfer). Its whole
    huge pages come in one fault each if the system grants the wish (a capture of 42 MB 5800 -> 2575 us); asked for here
    because this memory is the blob's own, where a buffer handed to the C entry is its caller's."""
    blob = _bytes_new(None, size)
    address = _bytes_address(blob)
    first, last = -(-address // _HUGE_PAGE) * _HUGE_PAGE, (address + size) // _HUGE_PAGE * _HUGE_PAGE
    if first < last:
        _madvise(first, last - first, mmap.MADV_HUGEPAGE)
    return blob, address


class KvSnapshot:
    """Holds the whole blob (header and payload): `to_bytes` and a restore hand it on without a copy."""

    def __init__(self, n_layer, kv_dim, max_seq, pos, payload: bytes):
        self._n_layer, self._kv_dim, self._max_seq, self._pos = n_layer, kv_dim, max_seq, pos
        self.payload = payload

    pos = property(lambda self: self._pos)
    n_layer = property(lambda self: self._n_layer)
    kv_dim = property(lambda self: self._kv_dim)
    max_seq = property(lambda self: self._max_seq)

    @property
    def payload(self) -> bytes:
        if self._payload is None:  # cut out of the blob at the first read and kept: it may be tens of megabytes
            self._payload = self._blob[HEADER_BYTES:]
        return self._payload

    @payload.setter
    def payload(self, payload):
        self._payload = bytes(payload)
        self._blob = MAGIC + struct.pack("<6I", VERSION, self._n_layer, self._kv_dim, self._max_seq, self._pos, 0) + self._payload

    def to_bytes(self) -> bytes:
        """src/kv_snapshot.rs:69-80."""
        return self._blob

    @classmethod
    def from_bytes(cls, blob: bytes) -> "KvSnapshot":
        """src/kv_snapshot.rs:104-140."""
        if len(blob) < HEADER_BYTES:
            raise ConfigError("invalid config: KvSnapshot blob too short: missing header")
        if blob[:8] != MAGIC:
            raise ConfigError("invalid config: KvSnapshot blob has wrong magic")
        version, n_layer, kv_dim, max_seq, pos, reserved = struct.unpack("<6I", blob[8:32])
        if version != VERSION:
            raise ConfigError("invalid config: KvSnapshot blob has unsupported version")
        if reserved != 0:
            raise ConfigError("invalid config: KvSnapshot blob has non-zero reserved field")
        if len(blob) - HEADER_BYTES != payload_bytes(n_layer, kv_dim, pos):
            raise ConfigError("invalid config: KvSnapshot blob payload length does not match header")
        snap = cls.__new__(cls)
        snap._n_layer, snap._kv_dim, snap._max_seq, snap._pos = n_layer, kv_dim, max_seq, pos
        snap._blob, snap._payload = bytes(blob), None  # (a `bytes` is kept as it is)
        return snap

    def clone(self) -> "KvSnapshot":
        snap = KvSnapshot.__new__(KvSnapshot)
        snap.__dict__.update(self.__dict__)
        return snap

    # -- device side ---------------------------------------------------------
    @classmethod
    def capture(cls, ctxs, pos) -> "KvSnapshot":
        """`Session::snapshot`: read rows [0, pos) of every layer. `ctxs` is one
        AttnContext, or the list of all KV-head shards (each fills its columns)."""
        ctxs = list(ctxs) if isinstance(ctxs, (list, tuple)) else [ctxs]
        lib = _lib.load()
        size = int(lib.bp_snapshot_size(ctxs[0]._h, pos))
        blob, address = new_blob(size)
        if ctxs[0].cfg.n_shards != 1:
            C.memset(address, 0, size)  # a shard that is not in the list leaves its columns zero
        for ctx in ctxs:
            ctx._check(lib.bp_snapshot_capture(ctx._h, pos, address, size))
        return cls.from_bytes(blob)

    def apply(self, ctxs) -> int:
        """`Session::restore`: validate against the context(s) and write the rows back. Returns pos."""
        ctxs = list(ctxs) if isinstance(ctxs, (list, tuple)) else [ctxs]
        lib = _lib.load()
        blob = self.to_bytes()
        pos = C.c_uint32(0)
        for ctx in ctxs:
            ctx._check(lib.bp_snapshot_apply(ctx._h, blob, len(blob), C.byref(pos)))
        return pos.value
