"""Test support: the node path for calls with so few stars that the sizes choose the general
path, and workspaces of a given size."""


def force_nodes(monkeypatch, size=None):
    """rubix_cube_fwd and rubix_cube_fwd_dust through rubix_cube_fwd_nodes, with the workspace it
    asks for; ``size(name, sizes)``: another size for a workspace query."""
    from rubix_gb300 import _lib

    query, call = _lib.query, _lib.call

    def q(name, *args):
        if name == "rubix_cube_workspace_size":
            name = "rubix_cube_nodes_workspace_size"
        if size is not None and name in ("rubix_cube_nodes_workspace_size",
                                         "rubix_cube_bwd_workspace_size"):
            return size(name, args)
        return query(name, *args)

    def c(name, *args):
        if name == "rubix_cube_fwd":
            return call("rubix_cube_fwd_nodes", *args[:15], None, None, *args[15:])
        if name == "rubix_cube_fwd_dust":
            return call("rubix_cube_fwd_nodes", *args)
        return call(name, *args)

    monkeypatch.setattr(_lib, "query", q)
    monkeypatch.setattr(_lib, "call", c)


def least_workspace(name, sizes):
    """The smallest workspace (to 256 bytes) that still holds the node path of these sizes."""
    from rubix_gb300 import _lib

    lib = _lib.lib()
    back = name == "rubix_cube_bwd_workspace_size"
    full = int(getattr(lib, name)(*sizes))

    def launches(b):
        return (lib.rubix_cube_bwd_launches(*sizes, 0, b) if back
                else lib.rubix_cube_fwd_launches(*sizes, 2, b))

    general = int(lib.rubix_cube_general_workspace_size(*sizes))
    least = launches(full)
    lo, hi = general // 256, -(-full // 256)  # hi holds it
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if launches(mid * 256) >= least:  # the general path has fewer launches
            hi = mid
        else:
            lo = mid
    return max(hi * 256, general)
