// Which caller arrays kernels may use where they are (usable_in_place in
// hussar_gb300/csrc/hsr_internal.h), on made-up addresses that nothing dereferences.
// Arguments: inputs and outputs in turn as "i:address:bytes:align" / "o:...". Prints 1 or 0.
#include "hsr_internal.h"

#include <cstdio>
#include <cstdlib>

using namespace hsr;

int main(int argc, char **argv) {
    CallerArray in[3] = {}, out[3] = {};
    int ni = 0, no = 0;
    for (int k = 1; k < argc; ++k) {
        char kind;
        unsigned long long at, bytes, align;
        if (std::sscanf(argv[k], "%c:%llu:%llu:%llu", &kind, &at, &bytes, &align) != 4) return 1;
        if (kind == 'i' ? ni == 3 : no == 3) return 1;
        (kind == 'i' ? in[ni++] : out[no++]) =
            CallerArray{reinterpret_cast<const void *>(uintptr_t(at)), size_t(bytes), size_t(align)};
    }
    // what was not given is null, as an output the caller does not want is
    for (int k = 0; k < 3; ++k) {
        if (k >= ni) in[k].align = 1;
        if (k >= no) out[k].align = 1;
    }
    std::printf("%d\n", int(usable_in_place({in[0], in[1], in[2]}, {out[0], out[1], out[2]})));
    return 0;
}
