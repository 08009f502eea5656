"""The packed room table and point arrays of a batch against each room's own arguments."""
import numpy as np
import pytest

from gpurir_gb300 import batch, polar_patterns


def _rooms():
    rng = np.random.default_rng(0)
    f = lambda *n: rng.uniform(0.2, 2.0, n)
    return [
        dict(room_sz=[3, 4.1, 2], beta=f(6), pos_src=f(2, 3), pos_rcv=f(5, 3).astype(np.float32), nb_img=[3, 4, 5], Tmax=0.3),
        dict(room_sz=f(3, 1), beta=list(f(6)), pos_src=list(f(3)), pos_rcv=f(3, 2).T[:, [0, 1, 1]].tolist(),
             nb_img=np.array([6.0, 7.9, 8.0]), Tmax=np.float32(0.2), Tdiff=0.1, mic_pattern="card", orV_rcv=f(6)),
        dict(room_sz=f(1, 3).astype(np.float32), beta=f(2, 3), pos_src=f(12)[::2], pos_rcv=f(1, 1, 3),
             nb_img=np.array([[9], [10], [11]]), Tmax=1, Tdiff=None, spkr_pattern="bidir", orV_src=f(2, 3)[::-1],
             mic_pattern=None, orV_rcv=None),
    ]


def test_pack_every_form():
    rooms = _rooms()
    table, ps, pr, os_, or_ = batch.pack(rooms)
    f32 = lambda v, *s: np.asarray(v, dtype=np.float32).reshape(*s)
    i = j = 0
    for g, r in zip(table, rooms):
        n, m = g.n_src, g.n_rcv
        assert (n, m) == (f32(r["pos_src"], -1, 3).shape[0], f32(r["pos_rcv"], -1, 3).shape[0])
        assert np.array_equal(g.room_sz[:], f32(r["room_sz"], 3)) and np.array_equal(g.beta[:], f32(r["beta"], 6))
        assert g.nb_img[:] == [int(x) for x in np.asarray(r["nb_img"]).reshape(3)]
        assert g.Tmax == np.float32(r["Tmax"]) and g.Tdiff == np.float32(r.get("Tdiff") or r["Tmax"])
        assert g.spkr_pattern == polar_patterns[r.get("spkr_pattern") or "omni"]
        assert g.mic_pattern == polar_patterns[r.get("mic_pattern") or "omni"]
        for got, want in ((ps[i:i + n], r["pos_src"]), (pr[j:j + m], r["pos_rcv"]),
                          (os_[i:i + n], r.get("orV_src")), (or_[j:j + m], r.get("orV_rcv"))):
            assert got.dtype == np.float32
            assert np.array_equal(got, np.zeros(got.shape) if want is None else f32(want, -1, 3))
        i, j = i + n, j + m
    assert (len(ps), len(pr), len(os_), len(or_)) == (i, j, i, j)


@pytest.mark.parametrize("key,value", [("room_sz", [1, 2]), ("beta", np.zeros(5)), ("nb_img", [1, 2]),
                                       ("pos_src", np.zeros(4)), ("orV_src", np.zeros((3, 3))), ("mic_pattern", "x")])
def test_pack_refuses(key, value):
    rooms = _rooms()
    rooms[0][key] = value
    with pytest.raises((ValueError, KeyError)):
        batch.pack(rooms)
