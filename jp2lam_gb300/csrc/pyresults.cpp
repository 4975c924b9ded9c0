// Codestreams' memory from Python bytes objects (jp2g_py_result_alloc), by way
// of the interpreter's functions as the caller passes them: this library is
// not linked to one.
#include "jp2g.h"

extern "C" uint8_t* jp2g_py_result_alloc(void* user, uint32_t index, size_t bytes) {
  jp2g_py_results* r = static_cast<jp2g_py_results*>(user);
  if (!r || index >= r->n || bytes > (size_t)PTRDIFF_MAX) return nullptr;
  const int gil = r->gil_ensure();
  if (r->objects[index]) r->decref(r->objects[index]);
  r->objects[index] = r->new_bytes(nullptr, (ptrdiff_t)bytes);
  uint8_t* at = nullptr;
  if (r->objects[index]) at = reinterpret_cast<uint8_t*>(r->bytes_at(r->objects[index]));
  else r->clear_error();  // out of memory: reported by the encode call
  r->gil_release(gil);
  return at;
}
