// A Python list of whole numbers as 32-bit integers, on the host.  A prompt's token ids come as such a list; numpy takes
// 40 ns a number for the conversion and checks the range in two more passes (3,359 tokens: 160 us, more than the launch of
// the whole captured step), this 6 ns with the check.  The interpreter's functions are looked up when the first list
// comes, so the library itself does not depend on one; the caller holds its lock (ctypes.PyDLL).
#include <dlfcn.h>

#include "common.cuh"

namespace {

struct Interpreter {
    long (*list_size)(void*);
    void* (*list_item)(void*, long);                // a borrowed reference
    long (*as_long)(void*, int*);                   // value, and whether it overflows
    void* (*error)();
    void (*clear)();
    bool found;
};

Interpreter interpreter() {
    Interpreter p;
    p.list_size = reinterpret_cast<long (*)(void*)>(dlsym(RTLD_DEFAULT, "PyList_Size"));
    p.list_item = reinterpret_cast<void* (*)(void*, long)>(dlsym(RTLD_DEFAULT, "PyList_GetItem"));
    p.as_long = reinterpret_cast<long (*)(void*, int*)>(dlsym(RTLD_DEFAULT, "PyLong_AsLongAndOverflow"));
    p.error = reinterpret_cast<void* (*)()>(dlsym(RTLD_DEFAULT, "PyErr_Occurred"));
    p.clear = reinterpret_cast<void (*)()>(dlsym(RTLD_DEFAULT, "PyErr_Clear"));
    p.found = p.list_size && p.list_item && p.as_long && p.error && p.clear;
    return p;
}

}  // namespace

// out[i] = list[i] for the `count` numbers of the list.  0: all of them are whole numbers from 0 to below `limit`; else
// `out` says nothing and the caller looks at the list itself.
NNIS_API int nnis_list_to_ints(void* list, long count, long limit, int* out) {
    static const Interpreter py = interpreter();
    if (!py.found || !list || !out || limit > 0x7fffffffL || py.list_size(list) != count) {
        if (py.found && py.error()) py.clear();
        return NNIS_ERR_UNSUPPORTED;
    }
    for (long i = 0; i < count; ++i) {
        // (a number's own conversion may run code that changes the list: the item is looked up again each time)
        void* item = i < py.list_size(list) ? py.list_item(list, i) : nullptr;
        int overflow = 0;
        const long v = item ? py.as_long(item, &overflow) : -1;
        if (v < 0 || v >= limit || overflow) {
            if (py.error()) py.clear();
            return NNIS_ERR_ARGUMENT;
        }
        out[i] = (int)v;
    }
    return NNIS_OK;
}
